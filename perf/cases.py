"""Measured cases: the calls a fit or a sampler makes on this framework.

Two families, as in use:

* ``engine``: one evaluation of K parameter points over an event sample that
  is already loaded (``Engine.from_workload`` + ``autotune``, as the sampler
  and the benchmark do), through ``eval`` (host arrays in and out: minimisers,
  samplers) or ``eval_device`` (device pointers on the caller's stream:
  device-resident samplers, training sets).  The samples are taken from the
  benchmark's own synthetic configurations, with event weights, data and
  parameter points of the seed: c1 (3 splines and 2 norms per
  event, 400 bins, Poisson), c2 (mixed dials, 200 parameters, 3000 bins,
  Barlow-Beeston), c5 (400 parameters, 10,000 bins, a kriged table refilled
  from the parameters) and mixed (every dial type, mirrors, truncation,
  clamps, weight cap).
* ``surrogate``: the learned surrogate's calls: value and gradient of the
  stage-1 target (Hamiltonian trajectories), random-walk sub-chains, and the
  training loop over the device-resident set.
"""
from __future__ import annotations

import functools
import math
from types import SimpleNamespace

import numpy as np
import torch

from gundam_gb300 import _native as N
from gundam_gb300.engine import Engine
from gundam_gb300.surrogate import Surrogate
from gundam_gb300.workload import Workload

# events of each configuration's largest sample; smaller ones are its first events
MOST = {"c1": 100_000, "c2": 1_000_000, "c5": 300_000, "mixed": 20_000}


def _engine(name, config, events, points, precision, io="host", graph=False):
    return {"name": name, "family": "engine", "config": config, "events": events, "points": points,
            "precision": precision, "io": io, "graph": graph}


def _surrogate(name, call, params, bins, rows, steps=0):
    return {"name": name, "family": "surrogate", "call": call, "params": params, "bins": bins, "rows": rows,
            "steps": steps}


def listed():
    return [
        # the smallest exact call: one point of a small FP64 fit (a minimiser's function call)
        _engine("c1_fp64_1pt", "c1", 100_000, 1, "fp64"),
        # a small sample evaluated for 64 chains, the launch chain replayed from a CUDA graph
        _engine("c1_fp32_64pt_graph", "c1", 100_000, 64, "fp32", graph=True),
        # one point of a large mixed-dial sample: the memory-bound call, in each precision
        _engine("c2_fp32_1pt", "c2", 1_000_000, 1, "fp32"),
        _engine("c2_fp64_1pt", "c2", 500_000, 1, "fp64"),
        # a few points at once (finite differences of a fit), and double-float for 16
        _engine("c2_fp32_3pt", "c2", 499_979, 3, "fp32"),
        _engine("c2_df64_16pt", "c2", 250_000, 16, "df64"),
        # the sampler's call: 64 chains on the mixed-dial sample, FP32 dials and FP64 sums; and in FP64
        _engine("c2_fp32_64pt", "c2", 1_000_000, 64, "fp32", io="device"),
        _engine("c2_fp64_64pt", "c2", 200_000, 64, "fp64", io="device"),
        # 400 parameters, 10,000 bins and a table recomputed per point, a ragged number of points
        _engine("c5_fp32_100pt", "c5", 299_993, 100, "fp32"),
        # the surrogate at the c2 sizes: stage-1 value and gradient of 64 chains,
        # 64 random-walk sub-chains, and Adam steps on the device-resident set
        _surrogate("surrogate_value_grad", "value_grad", 200, 3000, 64),
        _surrogate("surrogate_substeps", "substeps", 200, 3000, 64, 10),
        _surrogate("surrogate_train", "train", 200, 3000, 2048, 24),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    u = rng.random()
    if u < 0.7:
        config = rng.choice(["c1", "c1", "c2", "c2", "c2", "c5", "mixed"])
        precision = rng.choice(["fp32", "fp32", "fp64", "df64"])
        points = rng.choice([1, 64, _log_int(rng, 1, 256)])
        events = _log_int(rng, 2_000, MOST[config])
        # no dearer than the largest listed cases: the 8-byte precisions' batches on smaller samples
        room = {"fp32": 6.4e7, "fp64": 1.28e7, "df64": 1.28e7}[precision]
        events = max(1_000, min(events, int(room / points)))
        return {k: v for k, v in _engine("", config, events, points, precision, rng.choice(["host", "device"]),
                                         rng.random() < 0.3).items() if k != "name"}
    call = rng.choice(["value_grad", "substeps", "train"])
    params = 8 * _log_int(rng, 2, 50)
    bins = 8 * _log_int(rng, 25, 500)
    rows = 128 * rng.randint(2, 16) if call == "train" else _log_int(rng, 1, 256)
    steps = {"value_grad": 0, "substeps": rng.randint(1, 20), "train": 3 * rng.randint(1, 8)}[call]
    return {k: v for k, v in _surrogate("", call, params, bins, rows, steps).items() if k != "name"}


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _pool(config):
    return Workload(config, n_events=MOST[config], seed=11)


def _sample(case, seed):
    """The configuration's first events with weights and data of the seed, as the object Engine.from_workload takes."""
    wl, n = _pool(case["config"]), case["events"]
    rng = np.random.default_rng([seed, 1])
    d1 = int(wl.event_dial_start[n])
    w = SimpleNamespace()
    for k in ("config", "n_params", "n_bins", "n_tables", "max_weight", "mirror_lo", "mirror_hi", "clamp_lo",
              "clamp_hi", "truncate", "prior_mean", "prior_icov", "prior_chol", "table_size", "table_fn_par",
              "table_node_start", "table_nodes", "table_clamp"):
        setattr(w, k, getattr(wl, k))
    w.n_events, w.n_dials = n, d1
    w.event_bin, w.event_dial_start = wl.event_bin[:n], wl.event_dial_start[:n + 1]
    w.event_w0 = wl.event_w0[:n] * rng.uniform(0.5, 1.5, n)
    for k in ("dial_type", "dial_par0", "dial_par1"):
        setattr(w, k, getattr(wl, k)[:d1])
    w.dial_data_start, w.dial_data = wl.dial_data_start[:d1 + 1], wl.dial_data[:int(wl.dial_data_start[d1])]
    w.dial_result = lambda: np.repeat(np.arange(n, dtype=np.int32), np.diff(w.event_dial_start))
    w.data = rng.poisson(wl.data * (n / wl.n_events)).astype(np.float64)
    w.llh = N.GW_LLH_BARLOW_BEESTON_OA2021 if case["config"] != "c1" else N.GW_LLH_POISSON
    z = rng.standard_normal((case["points"], w.n_params))
    w.points = np.ascontiguousarray(w.prior_mean[None, :] + z @ w.prior_chol.T)
    return w


def _prepare_engine(case, seed):
    w = _sample(case, seed)
    K = case["points"]
    s = SimpleNamespace(case=case, points=w.points)
    s.engine = Engine.from_workload(w, precision=case["precision"], k_max=K, llh_type=w.llh)
    s.engine.autotune(K)
    if case["graph"]:
        s.engine.use_graph(True)
    if case["io"] == "device":
        f64 = dict(dtype=torch.float64, device="cuda")
        s.stream = torch.cuda.Stream()
        s.d_points = torch.from_numpy(w.points).cuda()
        s.out = [torch.zeros((K, w.n_bins), **f64), torch.zeros((K, w.n_bins), **f64), torch.zeros(K, **f64),
                 torch.zeros(K, **f64)]
        torch.cuda.synchronize()
    return s


def _network(case, seed):
    """Network, head and parameter points of a trained-like surrogate (FP64 host arrays)."""
    P, B = case["params"], case["bins"]
    rng = np.random.default_rng([seed, 2])
    m = SimpleNamespace(P=P, B=B, nodes=8, lim=3.0)
    dims = [P, 512, 512, 512, B]
    m.layers = []
    for i, o in zip(dims[:-1], dims[1:]):
        lim = math.sqrt(6.0 / (i + o))
        m.layers.append((rng.uniform(-lim, lim, (o, i)).astype(np.float32),
                         rng.uniform(-0.05, 0.05, o).astype(np.float32)))
    m.mu, m.sd = rng.normal(0, 0.2, P), rng.uniform(0.1, 0.4, P)
    x = np.linspace(-m.lim, m.lim, m.nodes)
    slope = rng.normal(0, 0.02, (P, 1, B))
    bend = rng.normal(0, 0.002, (P, 1, B))
    tab = (slope * x[None, :, None] + bend * x[None, :, None] ** 2).reshape(P * m.nodes, B)
    m.A = np.concatenate([rng.uniform(4.0, 7.0, (1, B)), tab])
    m.r_mu, m.r_sd = rng.normal(0, 0.002, B), rng.uniform(0.005, 0.02, B)
    m.rb, m.rw = rng.normal(0.0, 0.1, B), rng.normal(0.0, 0.01, (B, P))
    m.data = rng.poisson(np.exp(m.A[0])).astype(np.float64)
    m.icov = np.eye(P) * 1.5 + 0.5 / P
    m.chol = np.linalg.cholesky(np.diag((0.02 * m.sd) ** 2) + 1e-6)
    m.rng = rng
    return m


def _points(m, rows):
    return m.mu + m.sd * m.rng.standard_normal((rows, m.P))


def _train_set(m, n):
    theta = _points(m, n)
    z = (theta - m.mu) / m.sd
    dev = dict(dtype=torch.float64, device="cuda")
    zt = torch.as_tensor(z, **dev)
    pairs = torch.as_tensor(m.rng.normal(0, 1.0 / m.P, (m.P, m.B)), **dev)
    logs = _base(m, zt) + torch.as_tensor(m.r_sd, **dev) * ((zt * zt.roll(1, 1)) @ pairs * math.sqrt(m.P))
    return theta, torch.exp(logs).cpu().numpy()


def _set_size(case):
    return 3 * case["rows"]  # three batches an epoch


def _prepare_surrogate(case, seed):
    m = _network(case, seed)
    rows = case["rows"]
    s = SimpleNamespace(case=case)
    sur = s.sur = Surrogate(m.P, m.B, batch_max=2048, seed=5)
    for l, (w, b) in enumerate(m.layers):
        sur.mlp.set_layer(l, w, b)
    sur.kind, sur.nodes, sur.lim = "additive", m.nodes, m.lim
    sur.mu, sur.sd, sur.A, sur.r_mu, sur.r_sd, sur.rb, sur.rw = m.mu, m.sd, m.A, m.r_mu, m.r_sd, m.rb, m.rw
    sur.attach(m.data, None, N.GW_LLH_BARLOW_BEESTON_OA2021)
    if case["call"] == "train":
        theta, sums = _train_set(m, _set_size(case))
        sur.reserve(_set_size(case))
        sur.append(theta, sums)
        return s
    s.theta = _points(m, rows)
    sur.set_chain(m.chol, m.mu, m.icov)
    if case["call"] == "substeps":
        _, s.f0, _ = sur.substeps(s.theta, None, 0, 1)
    return s


def prepare(case, seed):
    return _prepare_engine(case, seed) if case["family"] == "engine" else _prepare_surrogate(case, seed)


# ---------------------------------------------------------------- one pass
def run(state):
    case = state.case
    if case["family"] == "engine":
        if case["io"] == "device":
            o = state.out
            state.engine.eval_device(state.d_points.data_ptr(), case["points"], o[0].data_ptr(), o[1].data_ptr(),
                                     o[2].data_ptr(), o[3].data_ptr(), state.stream.cuda_stream)
            return o
        return list(state.engine.eval(state.points))
    sur = state.sur
    if case["call"] == "value_grad":
        return list(sur.value_grad(state.theta))
    if case["call"] == "substeps":
        return list(sur.substeps(state.theta, state.f0, case["steps"], 77))
    losses = sur.train(epochs=case["steps"] // 3, batch=case["rows"], seed=9)
    out = [np.asarray(losses, dtype=np.float32)]
    for l in range(sur.mlp.n_layers):
        out += list(sur.mlp.get_layer(l))
    return out


# ---------------------------------------------------------------- what a pass cannot do without
# per event and configuration: dials, values in them, operations per point
_PER_EVENT = {"c1": (5.0, 3 * 9.0, 3 * 31 + 4), "c2": (8.0, 8 * 15.4, 8 * 27.0), "c5": (11.0, 10 * 15.3 + 8, 10 * 28.0),
              "mixed": (4.0, 4 * 18.0, 4 * 25.0)}
_PARAMS = {"c1": (22, 400), "c2": (200, 3000), "c5": (400, 10000), "mixed": (16, 60)}


def work(case):
    if case["family"] == "engine":
        dials, values, ops = _PER_EVENT[case["config"]]
        P, B = _PARAMS[case["config"]]
        size = 4 if case["precision"] == "fp32" else 8
        n, K = case["events"], case["points"]
        return {"bytes": n * (values * size + dials * 6 + 8 + size) + K * (8 * P + 16 * B), "flops": n * K * ops}
    P, B, rows = case["params"], case["bins"], case["rows"]
    weights = P * 512 + 2 * 512 * 512 + 512 * B
    if case["call"] == "train":
        return {"bytes": case["steps"] * (weights * 28 + rows * 4 * (P + B)), "flops": case["steps"] * 6.0 * rows * weights}
    head = B * P * 4 * (8 + 1)
    passes = 1 if case["call"] == "value_grad" else case["steps"]
    flops = (4.0 if case["call"] == "value_grad" else 2.0) * rows * weights + rows * B * P * 6.0
    return {"bytes": passes * (2 * weights + head + rows * 16 * P), "flops": passes * flops}


# ---------------------------------------------------------------- the same in 64 bits
def _interval(x, knots):
    """Index i of the interval (knots [.., n], x [.., 1] broadcast), 0 .. n - 2, from x > knots[1 .. n - 2]."""
    return (x.unsqueeze(-1) > knots[:, 1:-1].unsqueeze(0)).sum(-1)


def _take(a, i):
    """a [D, n] at i [K, D] -> [K, D]."""
    return a.unsqueeze(0).expand(i.shape[0], -1, -1).gather(2, i.unsqueeze(-1)).squeeze(-1)


def _hermite(p1, m1, p2, m2, t):
    return p1 + t * (m1 + t * (3 * (p2 - p1) - 2 * m1 - m2 + t * (m1 + m2 - 2 * (p2 - p1))))


def _uniform_knots(y, low, step, x, trunc, slopes=None, limit=False):
    n = y.shape[1]
    u = (x - low) / step
    u = torch.where(trunc, u.clamp(0, n - 1), u)
    i = u.trunc().clamp(0, n - 2).long()
    t = u - i
    own = slopes is None
    if own:
        d = y[:, 1:] - y[:, :-1]
        slopes = torch.cat([d[:, :1], 0.5 * (d[:, 1:] + d[:, :-1]), d[:, -1:]], 1)
        if limit:
            top = 3 * torch.minimum(d[:, 1:].abs(), d[:, :-1].abs())
            mid = torch.where(d[:, 1:] * d[:, :-1] <= 0, torch.zeros_like(top), slopes[:, 1:-1])
            slopes = torch.cat([d[:, :1], torch.maximum(torch.minimum(mid, top), -top), d[:, -1:]], 1)
    p1, p2, m1, m2 = _take(y, i), _take(y, i + 1), _take(slopes, i), _take(slopes, i + 1)
    if own:  # beyond the ends the outer slope is the end difference
        m2 = torch.where(t < 0, p2 - p1, m2)
        m1 = torch.where(t >= 1, p2 - p1, m1)
    return _hermite(p1, m1, p2, m2, t)


def _bicubic(gx, gy, z, x, y):
    """Catmull-Rom rows along x, then along y, the grid extended linearly by one knot on each side."""
    def wide(a, dim):
        lo, hi = a.narrow(dim, 0, 1), a.narrow(dim, a.shape[dim] - 1, 1)
        return torch.cat([2 * lo - a.narrow(dim, 1, 1), a, 2 * hi - a.narrow(dim, a.shape[dim] - 2, 1)], dim)

    def segment(v, q, p):
        t = (v - q[1]) / (q[2] - q[1])
        step = q[2] - q[1]
        m1, m2 = step * (p[2] - p[0]) / (q[2] - q[0]), step * (p[3] - p[1]) / (q[3] - q[1])
        m2 = torch.where(t < 0, m1, m2)
        m1 = torch.where(t > 1, m2, m1)
        return _hermite(p[1], m1, p[2], m2, t)

    ny = gy.shape[1] + 2
    i = (x.unsqueeze(-1) >= gx[:, 1:-1].unsqueeze(0)).sum(-1)
    j = (y.unsqueeze(-1) >= gy[:, 1:-1].unsqueeze(0)).sum(-1)
    ex, ey, ez = wide(gx, 1), wide(gy, 1), wide(wide(z, 2), 1).flatten(1)
    qx, qy = [_take(ex, i + k) for k in range(4)], [_take(ey, j + k) for k in range(4)]
    rows = [segment(x, qx, [_take(ez, (i + k) * ny + j + r) for k in range(4)]) for r in range(4)]
    return segment(y, qy, rows)


def _respond(kind, v, x, y, trunc, tables):
    """Responses [K, D] of dials of one type and length: v [D, len] their data, x, y [K, D] their parameters."""
    if kind == N.GW_DIAL_NORM:
        return x
    if kind in (N.GW_DIAL_MONOTONIC, N.GW_DIAL_COMPACT):
        return _uniform_knots(v[:, 2:], v[:, 0], v[:, 1], x, trunc, limit=kind == N.GW_DIAL_MONOTONIC)
    if kind == N.GW_DIAL_UNIFORM:
        return _uniform_knots(v[:, 2::2], v[:, 0], v[:, 1], x, trunc, slopes=v[:, 3::2] * v[:, 1:2])
    if kind == N.GW_DIAL_GENERAL:
        p, s, q = v[:, 2::3], v[:, 3::3], v[:, 4::3]
        x = torch.where(trunc, torch.minimum(torch.maximum(x, q[:, 0]), q[:, -1]), x)
        i = _interval(x, q)
        a = _take(q, i)
        step = _take(q, i + 1) - a
        return _hermite(_take(p, i), _take(s, i) * step, _take(p, i + 1), _take(s, i + 1) * step, (x - a) / step)
    if kind == N.GW_DIAL_GRAPH:
        p, q = v[:, 0::2], v[:, 1::2]
        if p.shape[1] == 1:
            return p[:, 0].expand_as(x)
        x = torch.where(trunc, torch.minimum(torch.maximum(x, q[:, 0]), q[:, -1]), x)
        i = _interval(x, q)
        a, p1 = _take(q, i), _take(p, i)
        return p1 + (x - a) / (_take(q, i + 1) - a) * (_take(p, i + 1) - p1)
    if kind in (N.GW_DIAL_BILINEAR, N.GW_DIAL_BICUBIC):
        nx, ny = int(v[0, 0]), int(v[0, 1])
        gx, gy, z = v[:, 2:2 + nx], v[:, 2 + nx:2 + nx + ny], v[:, 2 + nx + ny:]
        x = torch.where(trunc, torch.minimum(torch.maximum(x, gx[:, 0]), gx[:, -1]), x)
        y = torch.where(trunc, torch.minimum(torch.maximum(y, gy[:, 0]), gy[:, -1]), y)
        if kind == N.GW_DIAL_BICUBIC:
            return _bicubic(gx, gy, z.reshape(-1, nx, ny), x, y)
        i, j = _interval(x, gx), _interval(y, gy)
        a, b = _take(gx, i), _take(gy, j)
        fx, fy = (x - a) / (_take(gx, i + 1) - a), (y - b) / (_take(gy, j + 1) - b)
        at = lambda di, dj: _take(z, (i + di) * ny + j + dj)  # noqa: E731
        v0, v1 = at(0, 0) + (at(1, 0) - at(0, 0)) * fx, at(0, 1) + (at(1, 1) - at(0, 1)) * fx
        return v0 + (v1 - v0) * fy
    t = tables[int(v[0, 0])]  # [K, size]
    if kind == N.GW_DIAL_TABULATED:
        i = v[:, 1].long()
        return v[:, 2] * t[:, i] + (1 - v[:, 2]) * t[:, i + 1]
    k = (v.shape[1] - 2) // 2
    return sum(v[:, 2 + k + q] * t[:, v[:, 2 + q].long()] for q in range(k))


def _exact_engine(case, seed):
    w = _sample(case, seed)
    dev = lambda a, dtype=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")  # noqa: E731
    raw = dev(w.points)
    lo, hi = dev(w.mirror_lo), dev(w.mirror_hi)
    both = (lo > -1e300) & (hi < 1e300)
    span = torch.where(both, hi - lo, torch.ones_like(lo))
    t = torch.fmod(raw - torch.where(both, lo, torch.zeros_like(lo)), 2 * span).abs()
    x = torch.where(both, torch.where(t > span, 2 * span - t, t) + lo.clamp(min=-1e300), raw)
    tables = []
    for k in range(w.n_tables):
        nodes = dev(w.table_nodes[w.table_node_start[k]:w.table_node_start[k + 1]])
        if w.table_fn_par[k, 0] >= 0:
            q = [x[:, int(p), None] for p in w.table_fn_par[k]]
            s = torch.sin(q[1] * 1.267 / nodes + q[2])
            tables.append(1 - q[0] * s * s * (1 + q[3] * (torch.log(nodes) - q[4])) * q[5])
        else:
            tables.append(nodes[None, :].expand(len(x), -1))
    E = w.n_events
    lens = np.diff(w.dial_data_start)
    rank = np.arange(w.n_dials) - np.repeat(w.event_dial_start[:-1], np.diff(w.event_dial_start))
    event = w.dial_result()
    # dials of one type, length, rank in their event and table are answered together
    key = (w.dial_type.astype(np.int64) * 64 + lens) * 64 + rank
    order = np.argsort(key, kind="stable")
    edges = np.concatenate([[0], np.flatnonzero(np.diff(key[order])) + 1, [w.n_dials]])
    values, trunc_all = dev(w.dial_data), dev(w.truncate, torch.bool)
    clo, chi = dev(w.clamp_lo), dev(w.clamp_hi)
    groups = sorted(((int(rank[order[a]]), order[a:b]) for a, b in zip(edges[:-1], edges[1:]) if b > a), key=lambda g: g[0])
    K = len(x)
    sums = torch.zeros((K, w.n_bins), dtype=torch.float64, device="cuda")
    sums2 = torch.zeros_like(sums)
    bins, w0 = dev(w.event_bin, torch.int64), dev(w.event_w0)
    step = max(1, int(2.5e7 // max(E, 1)))
    for k0 in range(0, K, step):
        xk, tk = x[k0:k0 + step], [t[k0:k0 + step] for t in tables]
        W = torch.ones((len(xk), E), dtype=torch.float64, device="cuda")
        for _, g in groups:
            kind, L = int(w.dial_type[g[0]]), int(lens[g[0]])
            v = values[dev(w.dial_data_start[g], torch.int64)[:, None] + torch.arange(L, device="cuda")]
            if kind >= N.GW_DIAL_TABULATED:
                r = _respond(kind, v, None, None, None, tk)
                c = w.table_clamp[int(v[0, 0])]
                r = r.clamp(float(c[0]), float(c[1]))
            else:
                p = dev(w.dial_par0[g], torch.int64)
                y = xk[:, dev(w.dial_par1[g], torch.int64)] if kind in (N.GW_DIAL_BILINEAR, N.GW_DIAL_BICUBIC) else None
                r = _respond(kind, v, xk[:, p], y, trunc_all[p], tk)
                r = torch.minimum(torch.maximum(r, clo[p]), chi[p])
            e = dev(event[g], torch.int64)
            W[:, e] *= r
        if w.max_weight > 0:
            W = W.clamp(max=w.max_weight)
        W *= w0
        sums[k0:k0 + step].index_add_(1, bins, W)
        sums2[k0:k0 + step].index_add_(1, bins, W * W)
    stat = _llh(w.llh, dev(w.data), sums, sums2).sum(1)
    d = raw - dev(w.prior_mean)
    return [sums, sums2, stat + ((d @ dev(w.prior_icov)) * d).sum(1), stat]


def _llh(kind, data, mu, s2):
    """-2 log L per bin."""
    safe = torch.clamp(mu, min=1e-300)
    full = torch.clamp(data, min=1e-300)
    if kind == N.GW_LLH_POISSON:
        r = torch.where(data > 0, 2 * (mu - data + data * torch.log(full / safe)), 2 * mu)
        return torch.where(mu > 0, r, torch.full_like(r, math.inf))
    f2 = torch.where(s2 > 0, s2 / safe ** 2, torch.ones_like(s2))
    t = safe * f2 - 1
    beta = torch.where(s2 > 0, 0.5 * (torch.sqrt(t * t + 4 * data * f2) - t), torch.ones_like(s2))
    mc = torch.clamp(torch.where(s2 > 0, safe * beta, mu), min=2.2250738585072014e-308)
    stat = torch.where(data > 2.3e-16, mc - data + data * (torch.log(full) - torch.log(mc)), mc)
    return 2 * stat + torch.where(s2 > 0, (beta - 1) ** 2 / f2, torch.zeros_like(s2))


def _base(m, z):
    """The additive piecewise-linear base at standardised points z [n, P]."""
    tab = torch.as_tensor(m.A[1:], dtype=torch.float64, device="cuda")
    u = (z.clamp(-m.lim, m.lim) + m.lim) * ((m.nodes - 1) / (2 * m.lim))
    i = u.detach().floor().clamp(max=m.nodes - 2).long()
    t = (u - i).unsqueeze(-1)
    j = torch.arange(m.nodes, device="cuda")
    hat = torch.where(j == i.unsqueeze(-1), 1 - t, torch.where(j == i.unsqueeze(-1) + 1, t, torch.zeros_like(t)))
    return torch.as_tensor(m.A[0], dtype=torch.float64, device="cuda") + hat.flatten(1) @ tab


def _forward(layers, z):
    for l, (w, b) in enumerate(layers):
        z = z @ w.T + b
        if l + 1 < len(layers):
            z = z * torch.sigmoid(z)
    return z


def _exact_surrogate(case, seed):
    if case["call"] == "substeps":
        return None  # accept / reject decisions on the device's own random numbers
    m = _network(case, seed)
    dev = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    layers = [(dev(w), dev(b)) for w, b in m.layers]
    if case["call"] == "value_grad":
        theta = dev(_points(m, case["rows"])).requires_grad_(True)
        z = (theta - dev(m.mu)) / dev(m.sd)
        lr = _base(m, z) + dev(m.r_mu) + dev(m.r_sd) * _forward(layers, z)
        s2 = torch.exp(lr + dev(m.rb) + z @ dev(m.rw).T)
        d = theta - dev(m.mu)
        f = _llh(N.GW_LLH_BARLOW_BEESTON_OA2021, dev(m.data), torch.exp(lr), s2).sum(1) + ((d @ dev(m.icov)) * d).sum(1)
        f.sum().backward()
        return [f.detach(), theta.grad]
    n, batch = _set_size(case), case["rows"]
    theta, sums = _train_set(m, n)
    z = (dev(theta) - dev(m.mu)) / dev(m.sd)
    target = (torch.log(dev(sums)) - _base(m, z) - dev(m.r_mu)) / dev(m.r_sd)
    params = [p.clone().requires_grad_(True) for wb in layers for p in wb]
    mom = [[torch.zeros_like(p), torch.zeros_like(p)] for p in params]
    state, mask = 9, (1 << 64) - 1
    losses, steps, spe = [], 0, n // batch
    total = case["steps"] // 3 * spe
    for _ in range(case["steps"] // 3):
        perm = list(range(n))
        for i in range(n - 1, 0, -1):  # splitmix64 and Fisher-Yates, as documented for the training loop
            state = (state + 0x9E3779B97F4A7C15) & mask
            h = state
            h = ((h ^ (h >> 30)) * 0xBF58476D1CE4E5B9) & mask
            h = ((h ^ (h >> 27)) * 0x94D049BB133111EB) & mask
            j = (h ^ (h >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        loss_sum = 0.0
        for b in range(spe):
            at = torch.as_tensor(perm[b * batch:(b + 1) * batch], device="cuda")
            y = _forward(list(zip(params[0::2], params[1::2])), z[at])
            loss = ((y - target[at]) ** 2).mean()
            grads = torch.autograd.grad(loss, params)
            loss_sum += float(loss.detach())
            lr = 0.5 * 1e-3 * (1 + math.cos(math.pi * steps / total))
            steps += 1
            with torch.no_grad():
                for p, g, (a, v) in zip(params, grads, mom):
                    a.mul_(0.9).add_(0.1 * g)
                    v.mul_(0.999).add_(0.001 * g * g)
                    p -= lr * (a / (1 - 0.9 ** steps)) / (torch.sqrt(v / (1 - 0.999 ** steps)) + 1e-8)
        losses.append(loss_sum / spe)
    return [torch.tensor(losses, dtype=torch.float64)] + [p.detach() for p in params]


def exact(case, seed):
    return _exact_engine(case, seed) if case["family"] == "engine" else _exact_surrogate(case, seed)
