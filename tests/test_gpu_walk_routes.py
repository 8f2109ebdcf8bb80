"""Which walk a line move takes (esm_set_sep_walk, esm_set_move_schedule, a batch): every route gives the
same states and counts, bit for bit, also where a point cap cuts a group of breakpoints at one t. (Before the
block walk left such walks to the one-lane walk, the two ended them differently in FP32, and these tests
showed by it which walk had run.)"""
import numpy as np
import pytest

from esmgb.device import DeviceBatch, DeviceChain
from esmgb.model import ROLE_GEN, ROLE_SE, Atoms, initial_state, make_model

pytestmark = pytest.mark.gpu


def _state(m, R, seed, edge):
    st = initial_state(m, R, seed=seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    st.g = st.g + 0.02 * rng.standard_normal(st.g.shape)
    st.theta = 5.0 * rng.standard_normal(st.theta.shape)
    st.e = rng.uniform(-0.02, 1.02, st.e.shape)
    if edge:                                            # many clamps at one time
        st.e = np.round(4.0 * st.e) / 4.0
    return st


def _chain(m, R, st, precision=32, sep=None, schedule="move", **kw):
    d = DeviceChain(m, R, precision=precision, seed=9, **kw)
    d.upload(st)
    if sep is not None:
        d.set_sep_walk(sep)
    d.set_move_schedule(schedule)
    return d


def _run(*a, **kw):
    d = _chain(*a, **kw)
    counts = d.sweeps(1, 0)
    out = d.download()
    d.close()
    return counts, out


def _same(x, y):
    return np.array_equal(x[0], y[0]) and all(np.array_equal(x[1][k], y[1][k]) for k in ("theta", "g", "e"))


def _ties():
    """A model and state whose walks the cap cuts inside groups of events of one time."""
    m = make_model(40, 60, 24, seed=3)
    return m, 8, _state(m, 8, 7, True), {"max_points": 8}


def test_sep_walk_zero_is_off():
    """0 keeps the one-lane walk (the walk of the whole-class launch); the default is 1."""
    m, R, st, kw = _ties()
    one_lane = _run(m, R, st, schedule="class", **kw)
    for sep in (0, 1, None):
        assert _same(_run(m, R, st, sep=sep, **kw), one_lane), sep
    # a setting above 0 that was asked for keeps the launches per move, the default does not
    for sep in (0, 1):
        assert _same(_run(m, R, st, sep=sep, schedule="class", **kw), one_lane), sep
    d = DeviceChain(m, R, seed=9)
    assert d.sep_walk()[0] == 1
    d.set_sep_walk(0)
    assert d.sep_walk()[0] == 0
    d.close()


def test_batch_takes_the_chains_walk():
    """A batch walks a chain's separable moves as the chain's own sweeps do, also when the setting changes
    after the batch was made."""
    m, R, st, kw = _ties()
    m2 = make_model(12, 18, 73, seed=5)
    st2 = _state(m2, 4, 8, False)
    a, b = _chain(m, R, st, **kw), _chain(m2, 4, st2)
    batch = DeviceBatch([a, b])
    for sep in (0, 41, 1, 13):                          # (no move has 41 units)
        a.set_sep_walk(sep)
        a.upload(st)
        b.upload(st2)
        counts = batch.sweeps(1, sweep0=0)
        assert _same((counts[0], a.download()), _run(m, R, st, sep=sep, **kw)), sep
        assert _same((counts[1], b.download()), _run(m2, 4, st2)), sep
    batch.close()
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_single_unit_below_the_threshold(precision):
    """Atoms of one storage unit, below the set number of units, keep the one-lane walk's bits."""
    m = make_model(12, 18, 73, seed=3)
    for f, a in enumerate(m.atoms):
        if a.role == ROLE_SE:
            idx = np.unique(a.idx).astype(np.int32)
            m.atoms[f] = Atoms(ROLE_SE, np.arange(len(idx) + 1, dtype=np.int32), idx, np.ones(len(idx)))
    st = _state(m, 8, 7, False)
    one_lane = _run(m, 8, st, precision, schedule="class")
    for sep in (0, 1, 2):
        assert _same(_run(m, 8, st, precision, sep=sep), one_lane), sep


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("cap", [10, 13, 0])
def test_equal_roots_beyond_the_buffer(precision, cap):
    """More node-balance roots at one time than the walk takes at once are all points of the walk: with a
    cap between the buffer and their number it ends in a guard event."""
    m = make_model(12, 18, 24, seed=3)
    for a in m.atoms:                                   # the one generator atom of all nodes, no other move
        n = np.diff(a.ptr)
        keep = int(np.flatnonzero(n == 12)[0]) if a.role == ROLE_GEN else 0
        s = slice(a.ptr[keep], a.ptr[keep + 1] if a.role == ROLE_GEN else a.ptr[keep])
        a.idx, a.val = a.idx[s].copy(), a.val[s].copy()
        a.ptr = np.array([0, len(a.idx)] if len(a.idx) else [0], np.int32)
    m.xbar[:m.N] = 2000.0                               # nodes alike: their balances vanish at one t
    m.wscale[:] = 0.0
    m.unit_mc[:] = 40.0
    st = initial_state(m, 4, seed=7)
    st.z[:] = 0.0
    st.g[:] = 0.3
    st.k[:] = 0.0
    st.k[m.disp] = 5000.0
    out = [_run(m, 4, st, precision, schedule=s, extra=0.0, max_points=cap) for s in ("move", "class")]
    assert out[1][0][:-1:2].sum() == m.T * 4
    assert out[1][0][-1] == (m.T * 4 if 0 < cap < 13 else 0)
    assert _same(*out)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("cap", [8, 20, 45, 0])
@pytest.mark.parametrize("N,T,R", [(40, 24, 8), (12, 73, 3)])
def test_equal_times_at_the_cap(N, T, R, cap, precision):
    """States of charge at quarters, and all at one half: many events of one time, which the cap cuts."""
    m = make_model(N, (3 * N) // 2, T, seed=3)
    for seed, steps in ((7, 4.0), (11, 4.0), (13, 2.0)):
        st = _state(m, R, seed, True)
        if steps == 2.0:
            st.e[:] = 0.5
        one_lane = _run(m, R, st, precision, schedule="class", max_points=cap)
        assert _same(_run(m, R, st, precision, max_points=cap), one_lane), seed
        other = make_model(20, 30, 24, seed=5)          # (another split of the block's lists)
        a = _chain(m, R, st, precision, max_points=cap)
        b = _chain(other, 16, _state(other, 16, 8, False), precision)
        batch = DeviceBatch([a, b])
        counts = batch.sweeps(1, sweep0=0)
        assert _same((counts[0], a.download()), one_lane), seed
        batch.close()
        a.close()
        b.close()
