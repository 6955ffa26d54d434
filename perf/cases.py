"""The workloads this engine's speed is measured on, each through a public entry point.

Five ways in, as programs use the library:

* ``host``   — :func:`ps26119.solve_lp` (the reference-facing C call) on host arrays: presolve, the
  solve, the in-process check and the certified bound, x, y, z back on the host.
* ``device`` — :func:`ps26119.solve_lp_device`: model and solution stay in device memory.
* ``batch``  — :func:`ps26119.solve_batch`: scenarios that share one matrix.
* ``serve``  — :class:`ps26119.Server`: independent requests in flight together.
* ``plugin`` — :class:`ps26119.Backend`: the op-by-op interface a host-driven loop calls.

LPs are the two families of :mod:`ps26119.generators` (the random equality LP and the staircase
planning LP), with the same shapes and value distributions but drawn on the GPU, so that new inputs
are quick to make. ``iterations`` is a solve's budget; a solve that reaches its 1e-8 tolerance ends sooner.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ps26119-solver_b200"))

import ps26119
from ps26119.generators import Lp

F64 = {"dtype": torch.float64, "device": "cuda"}

LISTED = [
    # The smallest request of a serving stream, with an iteration budget: launch latency and the checks.
    {"name": "solve_1k", "way": "host", "lp": "random", "size": 1000, "precision": "fp64", "iterations": 9600},
    # A small model in the middle of such a stream, mixed precision, an iteration budget, ragged size.
    {"name": "solve_4k_mixed", "way": "host", "lp": "random", "size": 4001, "precision": "mixed", "iterations": 3840},
    # The 10,000-row benchmark LP, plain fp64.
    {"name": "solve_10k", "way": "host", "lp": "random", "size": 10000, "precision": "fp64", "iterations": 6400},
    # A week of hourly planning periods through the other first-order algorithm.
    {"name": "pdlp_staircase_168", "way": "host", "lp": "staircase", "size": 168, "precision": "fp64",
     "algorithm": "pdlp", "iterations": 3840},
    # A large request, ragged size, with model and result resident on the device.
    {"name": "device_100k", "way": "device", "lp": "random", "size": 100003, "precision": "fp64", "iterations": 1280},
    # The benchmark's headline workload and its mixed-precision form.
    {"name": "device_1m", "way": "device", "lp": "random", "size": 1000000, "precision": "fp64", "iterations": 640},
    {"name": "device_1m_mixed", "way": "device", "lp": "random", "size": 1000000, "precision": "mixed",
     "iterations": 640},
    # The year of hourly planning periods.
    {"name": "device_staircase_8760", "way": "device", "lp": "staircase", "size": 8760, "precision": "fp64",
     "iterations": 1920},
    # The benchmark's scenario batch, and a smaller one in mixed precision.
    {"name": "batch_720x64", "way": "batch", "lp": "staircase", "size": 720, "precision": "fp64", "scenarios": 64,
     "iterations": 640},
    {"name": "batch_10kx16_mixed", "way": "batch", "lp": "random", "size": 10000, "precision": "mixed",
     "scenarios": 16, "iterations": 640},
    # Requests of a serving stream in flight together.
    {"name": "serve_16", "way": "serve", "lp": "random", "size": 20000, "low": 1000, "precision": "mixed",
     "requests": 16, "iterations": 1280},
    # A host-driven loop over the plugin's operations: 64 iterations and one check.
    {"name": "plugin_10k", "way": "plugin", "lp": "random", "size": 10000, "precision": "fp64", "iterations": 64},
]


def listed():
    return [dict(c) for c in LISTED]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    way = rng.choice(["host", "host", "device", "device", "batch", "serve", "plugin"])
    lp = rng.choice(["random", "random", "staircase"])
    case = {"way": way, "lp": lp, "precision": rng.choice(["fp64", "mixed"])}
    # staircase sizes are periods of 49 x 60; random sizes are rows
    if way == "host":
        case["size"] = _size(rng, 1000, 60000) if lp == "random" else _size(rng, 24, 1200)
        if rng.random() < 0.25:
            case["algorithm"] = "pdlp"
    elif way == "device":
        case["size"] = _size(rng, 20000, 900000) if lp == "random" else _size(rng, 400, 8000)
    elif way == "batch":
        case["size"] = _size(rng, 1000, 12000) if lp == "random" else _size(rng, 24, 600)
        case["scenarios"] = _size(rng, 4, 64)
    elif way == "serve":
        case["lp"] = "random"
        case["low"] = 1000
        case["size"] = _size(rng, 4000, 20000)
        case["requests"] = rng.randint(4, 16)
    else:
        case["size"] = _size(rng, 1000, 200000) if lp == "random" else _size(rng, 24, 2000)
    rows = case["size"] * (1 if case["lp"] == "random" else 49)
    budget = {"host": 3840, "device": 1280, "batch": 640, "serve": 1280, "plugin": 64}[way]
    if way == "device" and rows > 300000:
        budget = 640
    case["iterations"] = budget if way == "plugin" else 64 * rng.randint(budget // 128, budget // 64)
    return case


# ------------------------------------------------------------------------------------ inputs
def _csc(m, n, rows, cols, vals):
    order = torch.argsort(cols * m + rows)
    start = torch.zeros(n + 1, dtype=torch.int64, device=rows.device)
    start[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0)
    return start.int(), rows[order].int(), vals[order].contiguous()


def _random_lp(m, g):
    """6 nonzeros a row at distinct uniform columns, N(0, 1); feasible x0, bounded by its box."""
    n, kw = (3 * m) // 2, {"generator": g, "device": "cuda"}
    f64 = dict(kw, dtype=torch.float64)
    cols = torch.randint(0, n, (m, 6), **kw)
    while True:
        s = torch.sort(cols, 1).values
        bad = torch.nonzero((s[:, 1:] == s[:, :-1]).any(1)).flatten()
        if not len(bad):
            break
        cols[bad] = torch.randint(0, n, (len(bad), 6), **kw)
    cols = cols.flatten()
    rows = torch.arange(m, device="cuda").repeat_interleave(6)
    vals, x0, y0 = torch.randn(6 * m, **f64), torch.rand(n, **f64), torch.randn(m, **f64)
    z = torch.where(torch.rand(n, **f64) < 0.5, torch.rand(n, **f64), 0.0)
    start, ri, v = _csc(m, n, rows, cols, vals)
    col_of = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.diff(start.long()))
    b = _sorted_product(m, ri.long(), col_of, v, x0)
    c = _sorted_product(n, col_of, ri.long(), v, y0) + z
    full = lambda a: torch.full((n,), a, dtype=torch.float64, device="cuda")
    return {"m": m, "n": n, "c": c, "col_lower": full(0.0), "col_upper": full(10.0), "row_lower": b,
            "row_upper": b.clone(), "col_start": start, "row_index": ri, "value": v, "x0": x0}


def _sorted_product(size, to, by, vals, x):
    """Σ vals·x[by] into `to`, summed on the host: the same inputs whatever the GPU's atomics do."""
    out = np.bincount(to.cpu().numpy(), weights=(vals * x[by]).cpu().numpy(), minlength=size)
    return torch.from_numpy(out).cuda()


def _staircase_lp(T, g):
    """T periods of 49 x 60, about 175 nonzeros each, linked by 5 inventory columns."""
    R, C, inventory = 49, 60, 5
    m, n, f64 = T * R, T * C, {"generator": g, "device": "cuda", "dtype": torch.float64}
    at = torch.rand((T, R * C), generator=g, device="cuda").topk(160, 1).indices
    present = torch.zeros((T, R * C), dtype=torch.bool, device="cuda").scatter_(1, at, True).view(T, R, C)
    t, i = torch.nonzero(~present.any(2), as_tuple=True)  # every row and column gets an entry
    present[t, i, torch.randint(0, C, (len(t),), generator=g, device="cuda")] = True
    t, j = torch.nonzero(~present.any(1), as_tuple=True)
    present[t, torch.randint(0, R, (len(t),), generator=g, device="cuda"), j] = True
    k = torch.arange(inventory, device="cuda")
    present[:, k, C - inventory + k] = True
    t, i, j = torch.nonzero(present, as_tuple=True)
    vals = 10.0 ** (4.0 * torch.rand(len(t), **f64) - 2.0)
    vals = torch.where(torch.rand(len(t), **f64) < 0.5, -vals, vals)
    vals[(i < inventory) & (j == C - inventory + i)] = 1.0
    later = torch.arange(1, T, device="cuda").repeat_interleave(inventory)
    k = k.repeat(T - 1)
    rows = torch.cat([t * R + i, later * R + k])
    cols = torch.cat([t * C + j, (later - 1) * C + C - inventory + k])
    vals = torch.cat([vals, -torch.ones(len(k), dtype=torch.float64, device="cuda")])
    start, ri, v = _csc(m, n, rows, cols, vals)
    ub = 10.0 + 990.0 * torch.rand(n, **f64)
    x0 = ub * (0.2 + 0.6 * torch.rand(n, **f64))
    ax = _sorted_product(m, rows, cols, vals, x0)
    hour = torch.arange(T, device="cuda") % 24
    demand = (50.0 + 100.0 * torch.rand(T, **f64)) * (1.0 + 0.3 * torch.sin(2.0 * math.pi * hour / 24.0))
    slack = demand.repeat_interleave(R) * torch.rand(m, **f64)
    kind = torch.rand(m, **f64)
    rl = torch.where(kind < 0.3, ax, torch.where(kind < 0.65, ax - slack, -math.inf))
    ru = torch.where(kind < 0.3, ax, torch.where(kind < 0.65, math.inf, ax + slack))
    return {"m": m, "n": n, "c": torch.randn(n, **f64), "col_lower": torch.zeros(n, **F64),
            "col_upper": ub, "row_lower": rl, "row_upper": ru, "col_start": start, "row_index": ri, "value": v, "x0": x0}


def _make(kind, size, g):
    return _random_lp(size, g) if kind == "random" else _staircase_lp(size, g)


def _host(d):
    """The LP of _make as a generators.Lp in host memory."""
    a = {k: v.cpu().numpy() for k, v in d.items() if torch.is_tensor(v)}
    x0 = a.pop("x0")
    return Lp(d["m"], d["n"], meta={"x0": x0}, **a)


def _generator(seed):
    return torch.Generator("cuda").manual_seed(seed)


DATA = ("c", "col_lower", "col_upper", "row_lower", "row_upper", "col_start", "row_index", "value")


def _sizes(case, seed):
    """Rows of a stream's requests: log-uniform, the same for every seed (the seed makes the LPs)."""
    k, lo, hi = case["requests"], math.log(case["low"]), math.log(case["size"])
    return [int(math.exp(lo + (hi - lo) * ((0.5 + 7 * i) % k) / k)) for i in range(k)]


def prepare(case, seed):
    g, way = _generator(seed), case["way"]
    if way == "serve":
        return {"case": case, "lps": [_host(_random_lp(m, g)) for m in _sizes(case, seed)], "server": ps26119.Server(slots=16)}
    d = _make(case["lp"], case["size"], g)
    state = {"case": case}
    if way == "device":
        new = lambda k: torch.empty(k, dtype=torch.float64, device="cuda")
        state.update(model=d, x=new(d["n"]), y=new(d["m"]), z=new(d["n"]), stream=torch.cuda.Stream())
        return state
    lp = _host(d)
    state["lp"] = lp
    if way == "batch":
        from ps26119.generators import feasible_scenarios
        state["scenarios"] = feasible_scenarios(lp, case["scenarios"], seed=seed)
    if way == "plugin":
        be = ps26119.Backend(lp)
        state["backend"] = be
        state["eta"] = 0.998 / be.norm2_estimate()
        state["vec"] = {k: be.create(dual) for dual, names in ((False, ("x", "x0", "xh", "xb")), (True, ("y", "y0", "yh", "yb")))
                        for k in names}
        rng = np.random.default_rng(seed)
        be.upload(state["vec"]["x0"], np.clip(rng.uniform(0.0, 0.1, lp.num_cols), be.scaled(3), be.scaled(4)))
        be.upload(state["vec"]["y0"], np.zeros(lp.num_rows))
        be.set_precision(case["precision"] == "mixed")
    return state


def _said(r, **points):
    """A solve's outputs: the point, the objectives and residuals, how it ended."""
    return dict(points, objective=r.objective, dual_objective=r.dual_objective, primal_residual=r.primal_residual,
                dual_residual=r.dual_residual, iterations=r.iterations, status=r.status)


def run(state):
    case = state["case"]
    way = case["way"]
    if way == "device":
        d = state["model"]
        r = ps26119.solve_lp_device(d["m"], d["n"], 1, 0.0, [d[k].data_ptr() for k in DATA], precision=case["precision"],
                                    iteration_limit=case["iterations"], stream=state["stream"].cuda_stream,
                                    out=[state[k].data_ptr() for k in "xyz"])
        return _said(r, x=state["x"], y=state["y"], z=state["z"])
    if way == "serve":
        srv = state["server"]
        ids = [srv.submit(lp, precision=case["precision"], iteration_limit=case["iterations"]) for lp in state["lps"]]
        got = [srv.result(i)[0] for i in ids]
        return {"x": [r.x for r in got], "y": [r.y for r in got], "iterations": [r.iterations for r in got]}
    lp = state["lp"]
    if way == "plugin":
        be, v, K = state["backend"], state["vec"], case["iterations"]
        be.copy(v["x"], v["x0"])
        be.copy(v["y"], v["y0"])
        for k in range(K):
            w = (k + 1) / (k + 2)
            be.fused_primal(v["y"], v["x"], v["x0"], state["eta"], w, 1.0, v["xh"], v["xb"])
            be.fused_dual(v["xb"], v["y"], v["y0"], state["eta"], w, 1.0, v["yh"], v["yb"])
        k = be.kkt(v["xh"], v["yh"])
        return {"x": be.download(v["x"]), "y": be.download(v["y"]), "moved": be.diff_norm2(v["xh"], v["x0"]),
                "primal": k["primal_residual"], "dual": k["dual_residual"], "primal_obj": k["primal_obj"],
                "dual_obj": k["dual_obj"]}
    model = (lp.c, (lp.col_start, lp.row_index, lp.value), lp.row_lower, lp.row_upper, lp.col_lower, lp.col_upper)
    if way == "batch":
        got = ps26119.solve_batch(*model, scenarios=state["scenarios"], iteration_limit=case["iterations"],
                                  precision=case["precision"])
        return {"x": np.stack([r.x for r in got]), "y": np.stack([r.y for r in got]),
                "objective": np.array([r.objective for r in got]), "iterations": np.array([r.iterations for r in got])}
    r = ps26119.solve_lp(*model, algorithm=case.get("algorithm", "r2hpdhg"), precision=case["precision"],
                         iteration_limit=case["iterations"])
    return _said(r, x=r.x, y=r.y, z=r.z, bound=r.certified_bound)


def work(case):
    """Per iteration both products' matrices and the update's vectors once, as bench.py's roofline
    counts them; the model in and the point out once."""
    s = 8 if case["precision"] == "fp64" else 4
    K = case["iterations"]
    lots = case.get("scenarios", 1)
    total = {"bytes": 0, "flops": 0}
    for size in (_sizes(case, 0) if case["way"] == "serve" else [case["size"]]):
        if case["lp"] == "random":
            m, n, nnz = size, (3 * size) // 2, 6 * size
        else:
            m, n, nnz = 49 * size, 60 * size, 175 * size
        model = 12 * nnz + 4 * (n + 1) + lots * (24 * n + 16 * m)
        step = 2 * nnz * (s + 4) + 4 * (m + n) + lots * s * (9 * n + 7 * m)
        total["bytes"] += model + K * step + lots * 8 * (2 * n + m)
        total["flops"] += K * lots * (4 * nnz + 10 * (m + n))
    return total


# ------------------------------------------------------------------------------ 64-bit values
class _Scaled:
    """The scaled problem of an LP (geometric mean, Ruiz, Pock-Chambolle, bound and objective scalars)."""

    def __init__(self, d):
        self.m, self.n = m, n = d["m"], d["n"]
        self.rows = d["row_index"].long()
        self.cols = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.diff(d["col_start"].long()))
        self.value = d["value"]
        self.R, self.C = torch.ones(m, **F64), torch.ones(n, **F64)
        a = self.value.abs()
        v = a[a > 0]
        self.a = self.value.clone()
        if torch.log10(v.max() / v.min()) >= 4.5:
            for _ in range(12):
                self.R = self._middle(a * self.C[self.cols], self.rows, self.R)
                self.C = self._middle(a * self.R[self.rows], self.cols, self.C)
            self.a = self.a * (self.R[self.rows] * self.C[self.cols])
        for step in range(11):
            a = self.a.abs()
            if step < 10:
                r, c = (torch.zeros(k, **F64).scatter_reduce_(0, i, a, "amax") for k, i in ((m, self.rows), (n, self.cols)))
            else:
                r, c = (torch.zeros(k, **F64).index_add_(0, i, a) for k, i in ((m, self.rows), (n, self.cols)))
            r, c = (torch.where(k > 0, k.rsqrt(), 1.0) for k in (r, c))
            self.a = self.a * (r[self.rows] * c[self.cols])
            self.R, self.C = self.R * r, self.C * c
        self.c = self.C * d["c"]
        self.l, self.u = d["col_lower"] / self.C, d["col_upper"] / self.C
        self.rl, self.ru = self.R * d["row_lower"], self.R * d["row_upper"]
        self.bs = 1.0 / (_bounds_norm(self.rl, self.ru) + 1.0)
        self.os = 1.0 / (float(torch.linalg.norm(self.c)) + 1.0)
        self.l, self.u, self.rl, self.ru = (k * self.bs for k in (self.l, self.u, self.rl, self.ru))
        self.c = self.c * self.os
        self.A, self.At = self._matrix(self.a)
        self.A0, self.At0 = self._matrix(self.value)

    def _middle(self, v, index, old):
        lo = torch.full_like(old, math.inf).scatter_reduce_(0, index, v, "amin")
        hi = torch.zeros_like(old).scatter_reduce_(0, index, v, "amax")
        return torch.where(hi > 0, (1.0 / (lo.sqrt() * hi.sqrt())).clamp(1e-20, 1e20), old)

    def _matrix(self, a):
        at = torch.sparse_coo_tensor(torch.stack([self.cols, self.rows]), a, (self.n, self.m)).coalesce()
        return at.t().coalesce().to_sparse_csr(), at.to_sparse_csr()

    def norm(self):
        """||A||_2 by Lanczos on A'A: the largest eigenvalue once it stands still."""
        state, v = 0x9E3779B97F4A7C15, np.empty(self.n)
        for j in range(self.n):
            state ^= state >> 12
            state = (state ^ (state << 25)) & (2**64 - 1)
            state ^= state >> 27
            v[j] = (state * 0x2545F4914F6CDD1D % 2**64 >> 11) / 2.0**53 * 2.0 - 1.0
        v = torch.from_numpy(v).cuda()
        v, old, b = v / torch.linalg.norm(v), torch.zeros_like(v), 0.0
        alpha, beta, last, still, theta = [], [], -1.0, 0, 0.0
        for k in range(400):
            w = self.At @ (self.A @ v)
            alpha.append(float(w @ v))
            w = w - (alpha[-1] * v + b * old)
            b = float(torch.linalg.norm(w))
            theta = float(np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1))[-1])
            if b <= 1e-14 * max(1.0, theta):
                break
            beta.append(b)
            still = still + 1 if theta - last <= 1e-12 * theta else 0
            if still >= 5 and k >= 20:
                break
            last, old, v = theta, v, w / b
        return math.sqrt(max(theta, 0.0)) * (1.0 + 1e-4)

    def step(self, x, x0, y, y0, tau, sigma, w):
        """One reflected Halpern step: the new x and y, the projected and the extrapolated points."""
        xh = (x - tau * (self.c - self.At @ y)).clamp(self.l, self.u)
        xb = 2 * xh - x
        ax = self.A @ xb
        yh = y - sigma * ax + sigma * (ax - y / sigma).clamp(self.rl, self.ru)
        yb = 2 * yh - y
        return w * (2 * xh - x) + (1 - w) * x0, w * (2 * yh - y) + (1 - w) * y0, xh, xb, yh, yb

    def unscaled(self, d, x, y):
        return (self.C * x / self.bs).clamp(d["col_lower"], d["col_upper"]), self.R * y / self.os

    def kkt(self, d, x, y):
        """Residual norms and objectives of (x, y) on the original LP."""
        ax, lam = self.A0 @ x, d["c"] - self.At0 @ y
        viol = (d["row_lower"] - ax).clamp(min=0) + (ax - d["row_upper"]).clamp(min=0)
        side = torch.where(y > 0, d["row_lower"], d["row_upper"])
        open_ = (y != 0) & ~torch.isfinite(side)
        dual = torch.where((y == 0) | open_, 0.0, y * torch.where(torch.isfinite(side), side, 0.0)).sum()
        dual = dual + torch.where(lam > 0, lam * d["col_lower"], lam * d["col_upper"]).sum()
        return {"primal": float(torch.linalg.norm(viol)), "dual": float(torch.linalg.norm(y * open_)),
                "primal_obj": float(d["c"] @ x), "dual_obj": float(dual),
                "worst": float((viol / (1.0 + torch.where(ax < d["row_lower"], d["row_lower"], d["row_upper"]).abs())).max())}


def _bounds_norm(lo, up):
    lo, up = (torch.where(torch.isfinite(k), k.abs(), 0.0) for k in (lo, up))
    return float(torch.linalg.norm(torch.maximum(lo, up)))


def _solve(d, iterations, b_norm, c_norm):
    """The restarted reflected Halpern PDHG with PID primal weight, a check every 64 iterations."""
    S, K = _Scaled(d), 64
    eta = 0.998 / S.norm()
    x, y = torch.zeros(S.n, **F64).clamp(S.l, S.u), torch.zeros(S.m, **F64)
    x0, y0 = x, y
    omega, integral, best_omega, best_balance = 1.0, 0.0, 1.0, 1e300
    it, inner, r0, r_last = 0, 0, -1.0, math.inf

    def residual(xh, xb, yh, yb):
        dx, dy = xb - xh, yb - yh
        return math.sqrt(max(float(omega * (dx @ dx) + (dy @ dy) / omega + 2.0 * eta * (dy @ (S.A @ dx))), 0.0))

    while True:
        for k in range(K):
            w = (inner + 1) / (inner + 2)
            x, y, xh, xb, yh, yb = S.step(x, x0, y, y0, eta / omega, eta * omega, w)
            if inner == 0:
                r0 = residual(xh, xb, yh, yb)
            inner += 1
        it += K
        r = residual(xh, xb, yh, yb)
        xo, yo = S.unscaled(d, xh, yh)
        q = S.kkt(d, xo, yo)
        rp, rd = q["primal"] / (1.0 + b_norm), q["dual"] / (1.0 + c_norm)
        gap = abs(q["primal_obj"] - q["dual_obj"]) / (1.0 + abs(q["primal_obj"]) + abs(q["dual_obj"]))
        done = max(rp, rd, gap) <= 1e-8 and q["worst"] <= 1e-6
        if done or it == iterations:
            return {"x": xo, "y": yo, "z": d["c"] - S.At0 @ yo, "objective": q["primal_obj"],
                    "dual_objective": q["dual_obj"], "primal_residual": rp, "dual_residual": None, "iterations": it,
                    "status": ps26119.OPTIMAL if done else ps26119.ITERATION_LIMIT}
        if not (r <= 0.2 * r0 or (r <= 0.5 * r0 and r > r_last) or inner >= 0.36 * it):
            r_last = r
            continue
        dx, dy = float(torch.linalg.norm(xh - x0)), float(torch.linalg.norm(yh - y0))
        ratio = rd / rp if rd > 0 and rp > 0 else 1.0
        if 1e-16 < dx < 1e12 and 1e-16 < dy < 1e12 and 1e-8 < ratio < 1e8:
            e = math.log(dy) - math.log(dx) - math.log(omega)
            integral = 0.3 * integral + e
            omega *= math.exp(min(max(0.99 * e + 0.01 * integral, -math.log(10.0)), math.log(10.0)))
        else:
            omega, integral = best_omega, 0.0
        if rd > 0 and rp > 0 and abs(math.log10(ratio)) < best_balance:
            best_balance, best_omega = abs(math.log10(ratio)), omega
        x = x0 = xh
        y = y0 = yh
        inner, r_last = 0, math.inf


def exact(case, seed):
    """Plain torch in 64 bits: the fp64 r2HPDHG solves and the plugin's operations. No value for mixed
    precision (its fp32 phase follows another path), the batch, the server and PDLP, nor for the staircase
    through presolve, whose reductions would have to be written out here as well. The dual residual of
    these LPs is what rounding leaves of zero: no value either."""
    if case["precision"] != "fp64" or case["way"] in ("batch", "serve") or "algorithm" in case:
        return None
    if case["way"] == "host" and (case["lp"] != "random" or case["size"] > 20000):
        return None
    d = _make(case["lp"], case["size"], _generator(seed))
    if case["way"] == "plugin":
        S = _Scaled(d)
        eta = 0.998 / S.norm()
        x0 = torch.from_numpy(np.random.default_rng(seed).uniform(0.0, 0.1, S.n)).cuda().clamp(S.l, S.u)
        x, y = x0, torch.zeros(S.m, **F64)
        y0 = y
        for k in range(case["iterations"]):
            x, y, xh, _, yh, _ = S.step(x, x0, y, y0, eta, eta, (k + 1) / (k + 2))
        q = S.kkt(d, *S.unscaled(d, xh, yh))
        return {"x": x, "y": y, "moved": float(torch.linalg.norm(xh - x0)), "primal": q["primal"], "dual": None,
                "primal_obj": q["primal_obj"], "dual_obj": q["dual_obj"]}
    b_norm, c_norm = _bounds_norm(d["row_lower"], d["row_upper"]), float(torch.linalg.norm(d["c"]))
    if case["way"] == "device":
        return _solve(d, case["iterations"], b_norm, c_norm)
    # presolve takes the empty columns out (their cost is never negative: they stay at 0)
    kept = torch.diff(d["col_start"].long()) > 0
    small = dict(d, n=int(kept.sum()), **{k: d[k][kept] for k in ("c", "col_lower", "col_upper")})
    small["col_start"] = torch.cat([d["col_start"][:1], d["col_start"][1:][kept]])
    r = _solve(small, case["iterations"], b_norm, c_norm)
    x, z = torch.zeros(d["n"], **F64), d["c"].clone()
    x[kept], z[kept] = r["x"], r["z"]
    return dict(r, x=x, z=z, bound=None)
