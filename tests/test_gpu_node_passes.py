"""Branches of the passes over nodes: the rebuild with one and with four (step, replica) pairs a thread, which
must give the same bits, and the FP32 score pass at nodes of more lines than it keeps in shared memory (12),
with fewer replicas than a warp has lanes, one more, and a whole one, against the FP64 oracle by its bounds."""
import copy

import numpy as np
import pytest

from esmgb.device import DeviceChain
from esmgb.model import initial_state, make_model
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _state(m, R):
    st = initial_state(m, R, seed=3)
    rng = np.random.Generator(np.random.PCG64(5))
    st.g = st.g + 0.05 * rng.standard_normal(st.g.shape)
    st.e = rng.uniform(-0.02, 1.02, st.e.shape)
    st.theta = 30.0 * rng.standard_normal(st.theta.shape)
    return st


# 33 replicas of 1460 steps: four pairs, the last block ragged; one replica of them: one pair
@pytest.mark.parametrize("precision", [32, 64])
def test_rebuild_pairs_per_thread(precision):
    m = make_model(40, 60, 1460, seed=3)
    st = _state(m, 33)
    out = []
    for rep in (None, 0, 32):
        s = copy.copy(st)
        if rep is not None:
            for k, v in vars(st).items():
                if isinstance(v, np.ndarray) and v.ndim > 1 and v.shape[-1] == 33:
                    setattr(s, k, np.ascontiguousarray(v[..., rep:rep + 1]))
        d = DeviceChain(m, 33 if rep is None else 1, precision=precision, seed=9)
        d.upload(s)
        d.rebuild()
        out.append(d.caches())
        d.close()
    for i, rep in ((1, 0), (2, 32)):
        for a, b in zip(out[0], out[i]):
            assert np.array_equal(np.asarray(a)[..., rep:rep + 1], b)


@pytest.mark.parametrize("R", [1, 32, 33])
def test_scores_of_dense_nodes(R):
    m = make_model(16, 110, 24, seed=3)
    assert np.bincount(np.concatenate([m.bus0, m.bus1])).max() > 12
    d = DeviceChain(m, R, precision=32, seed=9)
    d.upload(_state(m, R))
    o = Oracle(m, R, seed=9)
    o.set_state(d.download())
    sk, _, parts = d.scores()
    ek, ep = d.score_errors()
    sk0, _, parts0 = o.scores()
    # (within the bounds that the pass reports, as test_capacity_scores)
    assert np.all(np.abs(sk - sk0) <= ek)
    assert np.all(np.abs(parts[:, :7] - parts0[:, :7]) <= ep[:, :7] + 1e-9)
