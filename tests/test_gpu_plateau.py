"""The storage sweeps' routes. A pass of the multiscale sweep takes a thread or a warp per task by the
number of its tasks (and a warp for long blocks); both sum a move in the same order, so a replica's state
does not depend on how many others run beside it, bit for bit. The long-range sweep takes a warp per task
for a year of at most 256 steps and a block beyond, whose terms go to global memory where a year of them
does not fit on chip: each against the oracle."""
import copy

import numpy as np
import pytest

from esmgb.device import DeviceChain
from esmgb.model import initial_state, make_model
from flipdiag import classify, first_diffs, summary
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _state(m, R, edge=False):
    st = initial_state(m, R, seed=3)
    rng = np.random.Generator(np.random.PCG64(17))
    st.g = st.g + 0.05 * rng.standard_normal(st.g.shape)
    st.e = rng.uniform(-0.02, 1.02, st.e.shape) if edge else rng.uniform(0.05, 0.95, st.e.shape)
    st.theta = 5.0 * rng.standard_normal(st.theta.shape)
    return st


def _first(st, R, n):
    """The state of the first n of R replicas."""
    out = copy.copy(st)
    for k, v in vars(st).items():
        if isinstance(v, np.ndarray) and v.ndim > 1 and v.shape[-1] == R:
            setattr(out, k, np.ascontiguousarray(v[..., :n]))
    return out


# 64 replicas: passes of 73 to 23360 tasks, by threads and by warps; 3 replicas: by warps, but for short
# blocks of the longest year. 600 points: a thread's layout in global memory. 8 points: walks that run over
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("edge", [False, True])
@pytest.mark.parametrize("N,T,kw", [(12, 292, {}), (6, 1460, {}), (12, 292, {"max_points": 600}),
                                    (12, 292, {"max_points": 8})])
def test_replica_independent_of_route(N, T, kw, edge, precision):
    m = make_model(N, (3 * N) // 2, T, seed=3)
    R, n = 64, 3
    st = _state(m, R, edge)
    out = []
    for r in (R, n):
        d = DeviceChain(m, r, precision=precision, seed=9, **kw)
        d.upload(_first(st, R, r))
        d.storage_ms(1)
        out.append(d.download())
        d.close()
    for k in ("g", "e"):
        assert not np.array_equal(out[0][k], getattr(st, k)), k
        assert np.array_equal(out[0][k][..., :n], out[1][k]), k


@pytest.mark.parametrize("N,T,R", [(12, 24, 8), (12, 219, 8), (12, 292, 8), (5, 8760, 2)])
def test_storage_long_routes(N, T, R):
    """Every task whose draws differ from the oracle's is a round-off flip at its first differing move, with
    the bounds of test_storage_long_flips_explained."""
    m = make_model(N, (3 * N) // 2, T, seed=3)
    st = _state(m, R)
    d = DeviceChain(m, R, precision=64, seed=5)
    d.upload(st)
    d.set_move_log(R)
    o = Oracle(m, R, seed=5)
    o.set_state(st)
    nu = len({p[0] for p in o.storage_long_plan(9)})
    sd = d.storage_long(9)
    tdev = d.storage_long_log(nu)                       # [unit, move, replica]
    torc = np.full((nu, 5, R), np.nan)
    o.storage_long_log(9, torc)
    assert sd[0] == nu * 5 * R
    first = first_diffs(tdev.transpose(1, 0, 2), torc.transpose(1, 0, 2), 1e-9, 1e-12)   # [unit, replica]
    o2 = Oracle(m, R, seed=5)
    o2.set_state(st)
    o2.rebuild()
    flips = []
    for ui, rep in zip(*np.nonzero(first >= 0)):
        mi = int(first[ui, rep])
        o2.sl_task(9, int(ui), int(rep), 0, mi)
        e = o2.sl_explain(9, int(ui), int(rep), mi, float(np.nan_to_num(tdev[ui, mi, rep])))
        assert e is not None
        e["t_dev"] = float(tdev[ui, mi, rep])
        kind, margin = classify(e, 40.0)
        flips.append(dict(kind=kind, margin=margin))
    assert (first < 0).any()
    assert all(f["margin"] <= (1e-6 if f["kind"] == "offset" else 1e-8) for f in flips), summary(flips)
