"""The weather step's recursion, whose innovations are formed in chunks of 56 steps by 32 replicas: years
below, at a remainder of and beyond a chunk, replicas below and beyond a warp, and more regimes than the
kernel keeps coefficients of (8), against the oracle with the bounds of test_weather_step."""
import copy

import numpy as np
import pytest

from esmgb.device import DeviceChain
from esmgb.model import initial_state, make_model
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _regimes(m, K):
    """The model with its regimes repeated to K."""
    m = copy.copy(m)
    idx = np.arange(K) % m.K
    for k in ("phi", "mu", "sig", "sig0"):
        v = getattr(m, k)
        if v.ndim and v.shape[0] == m.K:
            setattr(m, k, np.ascontiguousarray(v[idx]))
    P = m.Ptr[np.ix_(idx, idx)]
    m.Ptr = np.ascontiguousarray(P / P.sum(1, keepdims=True))
    m.pi0 = np.ascontiguousarray(m.pi0[idx] / m.pi0[idx].sum())
    m.K = K
    return m


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("T,R,K", [(24, 1, 2), (60, 33, 2), (219, 5, 2), (120, 33, 9)])
def test_weather_step_chunks(T, R, K, prec):
    m = make_model(8, 12, T, seed=4)
    if K != m.K:
        m = _regimes(m, K)
    st = initial_state(m, R, seed=3)
    d = DeviceChain(m, R, precision=prec, seed=5)
    d.upload(st)
    o = Oracle(m, R, seed=5)
    o.set_state(st)
    moved = (np.arange(R) % 3 != 1).astype(np.int32)
    theta = np.where(np.arange(R) % 2 == 0, 0.3, 0.1)
    window = np.where(np.arange(R) % 4 == 0, min(12, T), 0)
    wstart = 1 + (np.arange(R) * 7) % T
    for it in (4, 5):
        d.weather_step(moved, theta, window, wstart, it=it)
        o.weather_step(moved, theta, window, wstart, it=it)
    a, b = d.download(), o.get_state()
    assert np.array_equal(a["reg"], b["reg"])
    tz = 1e-9 if prec == 64 else 2 * 2e-5   # (two steps)
    assert np.abs(a["z"] - b["z"]).max() < tz * (1 + np.abs(b["z"]).max())
