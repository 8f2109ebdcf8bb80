"""The framework's work as a user's program has it do, case by case, for timing and comparison.

A case is a dict of plain values; ``prepare`` makes what a running program holds (a chain on the GPU
with its state uploaded, a batch of chains, a surrogate network and a minibatch), ``run`` makes one
pass through the public calls and returns what they give the caller. The networks are the seeded
synthetic models of ``esmgb.model`` (three lines per two nodes); the states are made here from the
case's seed: weather by its prior recursion, dispatch covering the residual load, storage half full,
each with a spread, as a chain meets them in its first sweeps.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "esm-sampling_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from esmgb import replicas as RP  # noqa: E402
from esmgb.device import DeviceBatch, DeviceChain  # noqa: E402
from esmgb.model import LANGEVIN_KAPPA, make_model  # noqa: E402
from esmgb.surrogate import MLP  # noqa: E402

NET = 1234                      # the networks' seed, the one of the benchmark
STEPS = (24, 73, 120, 219, 365, 584, 1095, 1460, 2920, 4380, 8760)  # steps per year (divisors of 8760)


def listed():
    return [
        # the smallest chain in use (the marginal comparisons' model): launches and latency count
        {"name": "sweep_n12_t24_r4", "kind": "sweep", "N": 12, "T": 24, "R": 4, "precision": 32, "read": "state"},
        # the plain replica sampler's configuration, FP64: 40 nodes, 6-hourly steps, 4 replicas
        {"name": "sweep_n40_t1460_r4_f64", "kind": "sweep", "N": 40, "T": 1460, "R": 4, "precision": 64,
         "read": "state"},
        # odd node and step counts (three colour classes), replicas that fill no warp evenly
        {"name": "sweep_n33_t1095_r24", "kind": "sweep", "N": 33, "T": 1095, "R": 24, "precision": 32,
         "read": "state"},
        # a large network: 128 nodes, the top of the uneven batch's range
        {"name": "sweep_n128_t1460_r16", "kind": "sweep", "N": 128, "T": 1460, "R": 16, "precision": 32,
         "read": "scores"},
        # the production step: 40 nodes, hourly, 64 replicas; weather schedule, sweep, scores, Langevin step
        {"name": "step_n40_t8760_r64", "kind": "step", "N": 40, "T": 8760, "R": 64},
        # uneven models in one batch, as the batching configuration draws them (a few of its 96)
        {"name": "batch_4models_r16", "kind": "batch", "sizes": "10:2920 24:1460 45:1460 64:1460", "R": 16},
        # the two storage sweeps of the operation sweep, 3-hourly
        {"name": "storage_n40_t2920_r64", "kind": "storage", "N": 40, "T": 2920, "R": 64},
        # scores and one Langevin step with dispatch following, production size
        {"name": "capacity_n40_t8760_r64", "kind": "capacity", "N": 40, "T": 8760, "R": 64, "precision": 32},
        # a weather burst of every replica (half of them with a regime window) and the replicas'
        # weather features, 3-hourly
        {"name": "weather_n40_t2920_r64", "kind": "weather", "N": 40, "T": 2920, "R": 64, "precision": 32,
         "read": "features"},
        # the surrogate of the learned proposal: one training step, and one evaluation in the chain
        {"name": "train_3x512_b1024", "kind": "train", "K": 212, "layers": 3, "width": 512, "batch": 1024},
        {"name": "predict_3x512_b1", "kind": "predict", "K": 212, "layers": 3, "width": 512, "batch": 1},
        # the surrogate of the full-scale configuration (256 nodes)
        {"name": "train_5x1024_b1024", "kind": "train", "K": 1357, "layers": 5, "width": 1024, "batch": 1024},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("sweep", "sweep", "sweep", "step", "batch", "storage", "capacity", "weather", "train",
                       "predict"))
    if kind in ("train", "predict"):
        return {"kind": kind, "K": _logint(rng, 53, 1357), "layers": rng.randint(1, 5),
                "width": _logint(rng, 48, 1024), "batch": _logint(rng, 1, 1024)}
    if kind == "batch":
        sizes = ["%d:%d" % (_logint(rng, 10, 97), rng.choice((73, 365, 1460))) for _ in range(rng.randint(2, 4))]
        return {"kind": kind, "sizes": " ".join(sizes), "R": _logint(rng, 4, 16)}
    precision = 64 if kind in ("sweep", "capacity", "weather") and rng.random() < 0.2 else 32
    most = 8e6 if precision == 64 else 1.5e8 if kind == "storage" else 5e8
    while True:
        N, T, R = _logint(rng, 10, 128), rng.choice(STEPS[2:] if kind == "storage" else STEPS), _logint(rng, 2, 64)
        if N * N * T * R <= most:
            break
    case = {"kind": kind, "N": N, "T": T, "R": R}
    if kind in ("sweep", "capacity", "weather"):
        case["precision"] = precision
    if kind in ("sweep", "weather"):
        small = 7 * N * T * R <= 7e6
        case["read"] = "state" if small else ("scores" if kind == "sweep" else "features")
    return case


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _model(N, T):
    return make_model(N, (3 * N) // 2, T, seed=NET)


def _device():
    return torch.device("cuda")


def _weather(m, R, seed, gen):
    """Regimes [T, R] (Markov chain) and anomalies [n0, T, R] (the switching VAR(1)) of the prior,
    the anomalies as FP32 values."""
    dev = _device()
    rng = np.random.default_rng([seed, 11])
    u = rng.random((m.T, R))
    cum = np.cumsum(m.Ptr, axis=1)
    reg = np.zeros((m.T, R), np.int32)
    reg[0] = np.minimum(np.searchsorted(np.cumsum(m.pi0), u[0]), m.K - 1)
    for t in range(1, m.T):
        reg[t] = np.minimum((u[t][:, None] > cum[reg[t - 1]]).sum(1), m.K - 1)
    f = dict(dtype=torch.float32, device=dev)
    z = torch.randn((m.T, m.n0, R), generator=gen, **f)
    phi, sig = (torch.as_tensor(x, **f) for x in (m.phi[0], m.sig[0]))   # the same in every regime
    mu0 = torch.as_tensor(m.mu[:, :, 0].T.copy(), **f)                    # [n0, K], no seasonal part
    k = torch.as_tensor(reg, dtype=torch.long, device=dev)
    z[0] *= torch.as_tensor(m.sig0, **f)[:, None]
    for t in range(1, m.T):
        z[t].mul_(sig[:, None]).addcmul_(z[t - 1], phi[:, None].expand(-1, R)).add_(mu0[:, k[t]])
    return reg, z.permute(1, 0, 2).contiguous()


def _start(m, R, seed):
    """A chain's state (torch, on the GPU, FP32 values): dispatch covers the residual load of its
    own weather, storage half full, flows small, each with a spread."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    reg, z = _weather(m, R, seed, gen)
    f = dict(dtype=torch.float32, device=dev)
    shape = (m.T, R)

    def randn(n):
        return torch.randn((n, *shape), generator=gen, **f)

    sc, xb = torch.as_tensor(m.wscale, **f), torch.as_tensor(m.xbar, **f)
    res = [torch.relu(xb[n][:, None] + sc[n] * z[n]) for n in range(m.N)]
    for i in m.ren:
        s = int(m.unit_series[i])
        res[m.unit_bus[i]] -= float(m.k0[i]) * torch.sigmoid(xb[s][:, None] + sc[s] * z[s])
    g = torch.stack([(res[m.unit_bus[i]] / max(float(m.k0[i]), 1e-9)).clamp(0, 1) for i in m.disp])
    return {"theta": 5.0 * randn(m.N), "g": g + 0.02 * randn(m.D), "e": 0.5 + 0.02 * randn(m.S), "z": z,
            "reg": reg, "k": np.asarray(m.k0, np.float64)}


def _host(st):
    return {k: v.double().cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in st.items()}


def _chain(m, R, seed, precision=32):
    d = DeviceChain(m, R, precision=precision, seed=1 + seed % 1000003)
    d.upload(_host(_start(m, R, seed)))
    return d


def _minibatch(case, seed):
    """Weights, inputs (capacities over their bound and regime occupancies) and standardised score
    targets of a surrogate of K capacities."""
    rng = np.random.default_rng([seed, 5])
    dims = [case["K"] + 8] + [case["width"]] * case["layers"] + [case["K"]]
    layers = []
    for i, o in zip(dims[:-1], dims[1:]):
        W = rng.standard_normal((o, i)) * math.sqrt(2.0 / i) * (0.1 if o == case["K"] else 1.0)
        layers.append((W.astype(np.float32), (0.05 * rng.standard_normal(o)).astype(np.float32)))
    x = rng.random((case["batch"], dims[0])).astype(np.float32)
    t = rng.standard_normal((case["batch"], dims[-1])).astype(np.float32)
    return dims, layers, x, t


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "it": 1, "read": case.get("read")}
    if kind in ("train", "predict"):
        dims, layers, s["x"], s["t"] = _minibatch(case, seed)
        s["net"] = MLP(dims, batch_max=case["batch"], seed=1)
        for l, (W, b) in enumerate(layers):
            s["net"].set_layer(l, W, b)
        return s
    if kind == "batch":
        s["chains"] = []
        for i, spec in enumerate(case["sizes"].split()):
            N, T = (int(x) for x in spec.split(":"))
            s["chains"].append(_chain(_model(N, T), case["R"], seed + 101 * i))
        s["batch"] = DeviceBatch(s["chains"])
        s["batch"].sweeps(1, 0)
        return s
    m = _model(case["N"], case["T"])
    R = case["R"]
    s["m"], s["d"] = m, _chain(m, R, seed, case.get("precision", 32))
    if kind in ("sweep", "storage"):               # a running chain: one sweep behind it
        s["d"].sweeps(1, 0)
    if kind in ("step", "capacity"):
        s["kappa_s"] = np.array([LANGEVIN_KAPPA.get(c, 100.0) for c in m.carriers])
        s["eta"] = np.full(len(m.carriers), RP.LANGEVIN_ETA)
        s["w"] = np.full(R, 1.0 / R)
    if kind == "step":
        s["ctl"] = RP.ReplicaCtl(M=R)
        s["rs"] = RP.ReplicaSet(R, eta_w=list(s["eta"]))
        s["rng"] = np.random.default_rng([seed, 3])
    if kind == "weather":
        s["moved"] = np.ones(R, np.int32)
        s["theta"] = np.full(R, 0.3)
        s["window"] = np.where(np.arange(R) % 2 == 0, min(60, m.T), 0).astype(np.int32)
        s["wstart"] = (1 + np.random.default_rng([seed, 4]).integers(0, m.T, R)).astype(np.int32)
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "train":
        loss, grads = s["net"].train_step(s["x"], s["t"], 1e-3, grads=True)
        return {"loss": loss, "grads": grads}
    if kind == "predict":
        return s["net"].forward(s["x"])
    it = s["it"]
    s["it"] += 1
    if kind == "batch":
        counts = s["batch"].sweeps(1, it)
        return [counts, [d.scores() for d in s["chains"]]]
    d = s["d"]
    if kind == "sweep":
        counts = d.sweeps(1, it)
        return [counts, d.download() if s["read"] == "state" else d.scores()]
    if kind == "step":
        m = s["m"]
        rec = RP.replica_step(d, s["rs"], s["ctl"], it, s["rng"], s["kappa_s"], m.beta_k / m.beta_v, m.unit_hi,
                              m.unit_group)
        return {k: rec[k] for k in ("sk", "fk", "parts", "wts", "kraw", "knew", "rs", "nclip")}
    if kind == "storage":
        counts = [d.storage_ms(it), d.storage_long(it)]
        return [counts, d.scores()]
    if kind == "capacity":
        scores = d.scores()
        return [scores, d.langevin_step(s["w"], s["eta"], s["kappa_s"], it=it)]
    d.weather_step(s["moved"], s["theta"], s["window"], s["wstart"], it=it)
    return [d.replica_features(s["m"].k0), d.download() if s["read"] == "state" else None]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _moves(N):
    """Line moves of one colour-class pass: the basis atoms (angles N - 1; dispatch N; two storage
    fields of N) and 4 N family draws."""
    return (4 * N - 1) + 4 * N


def _state_values(N, T, R):
    off = 12 if N == 40 else max(1, round(0.3 * N))
    fields = N + N + 2 * N + (3 * N + off)      # angles, dispatch, storage, weather
    return fields * T * R


def _sweep(N, T, R, size):
    """One operation sweep: the state and its caches read and written once (the lower bound on
    traffic); per move and task the line conditional of its terms, evaluated at no fewer than its
    ends and kinks (about 6 terms a move, 8 points, 20 operations a term and point)."""
    cache = (N + (3 * N) // 2) * T * R
    moved = 4 * N * T * R
    return {"bytes": size * (_state_values(N, T, R) + moved + 2 * cache), "flops": 960.0 * _moves(N) * T * R}


def work(case):
    kind = case["kind"]
    if kind in ("train", "predict"):
        dims = [case["K"] + 8] + [case["width"]] * case["layers"] + [case["K"]]
        B, w = case["batch"], sum(i * o + o for i, o in zip(dims[:-1], dims[1:]))
        io = 4 * B * (dims[0] + dims[-1])
        if kind == "predict":
            return {"bytes": 2 * w + io, "flops": 2.0 * B * w}
        # weights and both moments read and written, the gradients written
        return {"bytes": 28 * w + io, "flops": 6.0 * B * w - 2.0 * B * dims[0] * dims[1]}
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for spec in case["sizes"].split():
            N, T = (int(x) for x in spec.split(":"))
            w = _sweep(N, T, case["R"], 4)
            total = {k: total[k] + w[k] for k in total}
        return total
    N, T, R = case["N"], case["T"], case["R"]
    size = case.get("precision", 32) // 8
    if kind in ("sweep", "step"):
        return _sweep(N, T, R, size)
    n = _state_values(N, T, R)
    if kind == "storage":
        # every storage unit's states and its node's dispatch and balance, read and written once
        return {"bytes": 2 * 4 * 4 * N * T * R, "flops": 200.0 * 2 * N * T * R * 8}
    if kind == "capacity":
        # the scores read the state once, the following writes dispatch and residuals
        return {"bytes": size * (n + 4 * N * T * R), "flops": 30.0 * n}
    return {"bytes": 2 * size * n, "flops": 60.0 * n}     # weather: anomalies rotated, dispatch compensated


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------------------------
def _exact_scores(m, st, R):
    """Capacity scores d/dk of -beta_v (operational cost) plus the reference measure's gradient, the
    capacity prior's term and the cost parts, per replica."""
    dev = _device()
    D = dict(dtype=torch.float64, device=dev)
    theta, g, e, z = (st[k].double() for k in ("theta", "g", "e", "z"))
    k = torch.as_tensor(st["k"], **D)
    lo, hi = torch.as_tensor(m.unit_lo, **D), torch.as_tensor(m.unit_hi, **D)
    kc = torch.minimum(torch.maximum(k, lo), hi)
    inside = ((lo < k) & (k < hi)).double()
    dt, cv = m.dt, m.c_viol
    xb, sc = torch.as_tensor(m.xbar, **D), torch.as_tensor(m.wscale, **D)

    def series(i):
        return xb[i][:, None] + sc[i] * z[i]

    r = torch.stack([torch.relu(series(n)) for n in range(m.N)])
    pen = torch.zeros(R, **D)
    for a, b, lb, ls in zip(m.bus0, m.bus1, m.line_b, m.line_s):
        f = lb * (theta[a] - theta[b])
        r[a] += f
        r[b] -= f
        pen += cv * dt * torch.relu(f.abs() - ls).sum(0)
    cgen, cst = torch.zeros(R, **D), torch.zeros(R, **D)
    inj, own = {}, {}                 # injection per unit capacity, other cost per unit capacity
    for j, u in enumerate(m.disp):
        y = g[j].clamp(0, 1)
        inj[u] = m.unit_avail[u] * y
        out = cv * dt * (g[j] - y).abs()
        own[u] = dt * m.unit_mc[u] * inj[u] + out
        cgen += dt * m.unit_mc[u] * kc[u] * inj[u].sum(0)
        pen += (kc[u] + m.kappa0) * out.sum(0)
    for u in m.ren:
        inj[u] = torch.sigmoid(series(int(m.unit_series[u])))
        own[u] = dt * m.unit_mc[u] * inj[u]
        cgen += kc[u] * own[u].sum(0)
    for j, u in enumerate(m.stor):
        h, ein, eout, qt = (float(x[u]) for x in (m.unit_hours, m.unit_eta_in, m.unit_eta_out, m.unit_qt))
        ec = e[j].clamp(0, 1)
        dd = h * (torch.roll(ec, -1, 0) - ec) / dt - qt
        ch, di = torch.relu(dd) / ein, torch.relu(-dd) * eout
        dic = di.clamp(max=1.0)
        over = cv * dt * torch.relu(ch - 1) + (cv * dt * torch.relu(di - 1) if qt <= 0 else 0.0)
        box = cv * h * (e[j] - ec).abs()
        inj[u] = dic - ch
        run_ = dt * m.unit_mc[u] * (ch + dic)
        own[u] = run_ + over + box
        cst += kc[u] * run_.sum(0)
        pen += (kc[u] + m.kappa0) * (over + box).sum(0)
    for u in inj:
        r[m.unit_bus[u]] -= kc[u] * inj[u]
    shed, dump = dt * torch.relu(r).sum((1,)), dt * torch.relu(-r).sum((1,))
    G = dt * torch.where(r > 0, m.c_shed, torch.where(r < 0, -m.c_dump, 0.0))
    sk = torch.zeros((R, m.Kunits), **D)
    ren = set(int(u) for u in m.ren)
    for u in inj:
        dk = (own[u] - inj[u] * G[m.unit_bus[u]]).sum(0)
        sk[:, u] = -m.beta_v * inside[u] * dk
        if m.physical and int(u) not in ren:
            sk[:, u] += inside[u] * m.T / (k[u] + m.kappa0)
    shed, dump = shed.sum(0), dump.sum(0)
    cap = torch.as_tensor(m.unit_capex, **D)
    capex = (cap * k + m.gamma_k * cap * (k - kc).abs()).sum()
    op = cgen + cst + m.c_shed * shed + m.c_dump * dump + pen
    parts = torch.stack([capex.expand(R), op, cgen, cst, shed, dump, pen, torch.zeros(R, **D)], dim=1)
    fk = m.beta_k * cap * (1 + m.gamma_k * torch.sign(k - kc))
    return [sk, fk, parts]


def _exact_net(case, seed, train):
    dev = _device()
    _, layers, x, t = _minibatch(case, seed)
    p = [[torch.as_tensor(v, dtype=torch.float64, device=dev).requires_grad_(train) for v in wb] for wb in layers]
    a = torch.as_tensor(x, dtype=torch.float64, device=dev)
    for l, (W, b) in enumerate(p):
        a = a @ W.T + b
        if l + 1 < len(p):
            a = torch.nn.functional.silu(a)
    if not train:
        return a
    loss = ((a - torch.as_tensor(t, dtype=torch.float64, device=dev)) ** 2).sum() / (2 * case["batch"])
    loss.backward()
    return {"loss": float(loss.detach()), "grads": [(W.grad, b.grad) for W, b in p]}


def exact(case, seed):
    # sweeps and steps are chains of random discrete choices: their values in 64 bits are other chains'
    if case["kind"] in ("train", "predict"):
        return _exact_net(case, seed, case["kind"] == "train")
    if case["kind"] == "capacity":
        m = _model(case["N"], case["T"])
        return [_exact_scores(m, _start(m, case["R"], seed), case["R"]), None]
    return None
