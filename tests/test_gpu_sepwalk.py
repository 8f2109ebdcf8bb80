"""The block walk of the separable storage moves against the one-lane walk (the whole-class launch
walks every move so): the same points, sums and draws, so the states and counts are equal bit for bit."""
import numpy as np
import pytest

from esmgb.device import DeviceChain
from esmgb.model import initial_state, make_model

pytestmark = pytest.mark.gpu


def _state(m, R, seed, edge):
    st = initial_state(m, R, seed=seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    st.g = st.g + 0.02 * rng.standard_normal(st.g.shape)
    st.theta = 5.0 * rng.standard_normal(st.theta.shape)
    st.e = rng.uniform(-0.02, 1.02, st.e.shape)         # some states beyond the box: walks of ray steps
    if edge:                                            # many clamps at one time, and states at a bound
        st.e = np.round(4.0 * st.e) / 4.0
    return st


# (nodes, steps, replicas, options): one task per block up to full batches; lists sorted by one lane, in
# registers (one to eight entries a lane) and in memory; the point cap; windows of one clamp and of many
CASES = [
    (5, 24, 1, {}),
    (12, 73, 3, {}),
    (40, 24, 33, {}),
    (40, 219, 16, {}),
    (40, 24, 8, {"max_points": 8}),
    (40, 24, 8, {"max_points": 600, "maxnats": 4000.0}),
    (12, 120, 8, {"maxnats": 4000.0}),
    (12, 120, 8, {"maxnats": 0.5}),
    (96, 24, 4, {}),
]


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("edge", [False, True])
@pytest.mark.parametrize("N,T,R,kw", CASES)
def test_block_walk_equals_one_lane_walk(N, T, R, kw, edge, precision):
    if edge and kw.get("max_points") == 8:
        pytest.skip("the cap falls inside a group of events of one time, whose order is free")
    m = make_model(N, (3 * N) // 2, T, seed=3)
    st = _state(m, R, 7, edge)
    out = []
    for schedule in ("move", "class"):
        d = DeviceChain(m, R, precision=precision, seed=9, **kw)
        d.upload(st)
        d.set_move_schedule(schedule)
        counts = d.sweeps(1, 0)
        out.append((counts, d.download()))
        d.close()
    (ca, a), (cb, b) = out
    assert np.array_equal(ca, cb)
    for k in ("theta", "g", "e"):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("units", [1, 3, 13, 41])
def test_block_walk_from_units(units):
    """Moves below the set number of units take the one-lane walk: the same state."""
    m = make_model(40, 60, 24, seed=3)
    st = _state(m, 16, 7, False)
    out = []
    for u in (0, units):
        d = DeviceChain(m, 16, precision=32, seed=9)
        d.upload(st)
        d.set_sep_walk(u)
        d.sweeps(1, 0, stats=False)
        out.append(d.download())
        d.close()
    for k in ("theta", "g", "e"):
        assert np.array_equal(out[0][k], out[1][k]), k
