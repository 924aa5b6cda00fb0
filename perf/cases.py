"""The measured work of the LP solver, as a user's program calls it.

A case is one call through the library's public entry points on inputs made from a seed:

  solve   DeviceProblem.solve on a resident problem: the first `iterations` iterations of the
          restarted PDHG loop from the zero start, and the averaged iterate on the host.
  batch   DeviceBatch.solve on packed problems of mixed sizes, the same way.
  load    DeviceProblem.from_csc (upload, transpose, rescaling on the GPU), a short solve, the
          rescaling vectors and the solution read back, and the handle closed.
  check   gpdhg_convergence_noalloc: the termination statistics of a candidate solution.

Iterations are counted instead of solving to a tolerance: the loop amplifies rounding until
iterates of two summation orders have nothing in common, so only a short run has values that
can be compared. FP32 runs are shorter for the same reason, and hand out FP32 values.
"""
import ctypes
import math
import os
import sys
import types

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cupdlp.jl_gb300"))

import cupdlp  # noqa: E402
from cupdlp import _abi  # noqa: E402
from cupdlp.solver import DeviceBatch, DeviceProblem, _Desc  # noqa: E402

EVALUATE_EVERY = 64   # PdhgParameters' default


def listed():
    return [
        # the termination statistics of one candidate of the power-law LP's size
        {"name": "check", "kind": "check", "m": 1_000_000, "n": 2_000_000},
        # the smallest LPs of the batch and of the serving mixture: a lone solve is latency
        {"name": "tiny_fp64", "kind": "solve", "lp": "random", "m": 203, "n": 406, "per_row": 20.0,
         "precision": "fp64", "iterations": 128},
        # the plain benchmark LP: 1,000 x 2,000, 0.5% dense
        {"name": "plain_fp64", "kind": "solve", "lp": "random", "m": 1000, "n": 2000, "per_row": 10.0,
         "precision": "fp64", "iterations": 128},
        # a medium request of the serving mixture (10,000 to 100,000 rows), in both precisions
        {"name": "medium_fp64", "kind": "solve", "lp": "random", "m": 20_011, "n": 40_022, "per_row": 20.0,
         "precision": "fp64", "iterations": 96},
        {"name": "medium_fp32", "kind": "solve", "lp": "random", "m": 90_007, "n": 180_014, "per_row": 22.0,
         "precision": "fp32", "iterations": 32},
        # the transportation benchmark LP: 500 x 2,000, two nonzeros per column
        {"name": "transport_fp64", "kind": "solve", "lp": "transport", "m": 500, "n": 2000, "per_row": 0.0,
         "precision": "fp64", "iterations": 64},
        # the power-law benchmark LP, whose iterations run in FP32 first, and the serving
        # mixture's large LP in FP64, which the benchmark's second phase runs in
        {"name": "power_law_fp32", "kind": "solve", "lp": "power_law", "m": 1_000_000, "n": 2_000_000,
         "per_row": 20.0, "precision": "fp32", "iterations": 32},
        {"name": "power_law_fp64", "kind": "solve", "lp": "power_law", "m": 500_000, "n": 1_000_000,
         "per_row": 20.0, "precision": "fp64", "iterations": 64},
        # the batch benchmark's mixture (median 2,000 rows, a quarter transportation LPs)
        {"name": "batch_fp32", "kind": "batch", "count": 48, "m_lo": 200, "m_hi": 50_000, "median": 2000, "sizes": 3,
         "precision": "fp32", "iterations": 24},
        # a cohort of the serving loop's small requests (200 to 2,000 rows)
        {"name": "batch_small_fp64", "kind": "batch", "count": 40, "m_lo": 200, "m_hi": 2000, "median": 700, "sizes": 4,
         "precision": "fp64", "iterations": 64},
        # one problem from host arrays to its solution, as optimize() runs it
        {"name": "load", "kind": "load", "lp": "random", "m": 60_013, "n": 120_026, "per_row": 20.0,
         "precision": "fp64", "iterations": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["check", "solve", "solve", "solve", "solve", "batch", "load"])
    if what == "check":
        n = _log(rng, 400, 4_000_000)
        return {"kind": "check", "m": max(1, int(n * rng.uniform(0.2, 1.0))), "n": n}
    precision = rng.choice(["fp64", "fp32"])
    short = 32 if precision == "fp32" else 64
    if what == "batch":
        lo = _log(rng, 200, 1000)
        hi = _log(rng, 2 * lo, 30_000)
        return {"kind": "batch", "count": rng.randint(3, 48), "m_lo": lo, "m_hi": hi, "median": _log(rng, lo, min(hi, 2500)),
                "sizes": rng.randrange(1 << 30), "precision": precision,
                "iterations": 24 if precision == "fp32" else 64}
    lp = rng.choice(["random", "random", "transport", "power_law"])
    if lp == "transport":   # an FP64 workload: a lone one's FP32 iterates part within a few dozen steps
        precision, short = "fp64", 64
        case = {"lp": lp, "m": _log(rng, 10, 600), "n": _log(rng, 40, 2000), "per_row": 0.0}
    elif lp == "power_law":
        m = _log(rng, 3000, 500_000)
        case = {"lp": lp, "m": m, "n": 2 * m + rng.randint(0, 1), "per_row": rng.uniform(10.0, 20.0)}
    else:
        m = _log(rng, 200, 100_000)
        case = {"lp": lp, "m": m, "n": 2 * m + rng.randint(0, 3), "per_row": rng.uniform(5.0, 40.0)}
    if what == "load":
        return {"kind": "load", **case, "precision": "fp64", "iterations": 20}
    return {"kind": "solve", **case, "precision": precision, "iterations": short}


# ---- inputs -----------------------------------------------------------------------------


class _Lp:
    """min c'x, A x = b (the first neq rows), A x >= b (the rest), l <= x <= u; A in
    compressed sparse columns, each column's rows increasing."""

    def __init__(self, m, n, neq, colptr, rows, vals, l, u, c, b):
        self.m, self.n, self.neq = m, n, neq
        self.colptr, self.rows, self.vals = colptr, rows, vals
        self.l, self.u, self.c, self.b = l, u, c, b

    def cols(self):
        return np.repeat(np.arange(self.n, dtype=np.int32), np.diff(self.colptr))


def _planted(g, host, m, n, rows, cols, value, ub):
    """An LP on the pattern (rows, cols) whose optimum is planted: 30% of x at 0, 10% at the
    upper bound; half of the '>=' rows slack; 60% of the rows equalities. `host` draws the
    m- and n-vectors; the matrix is drawn on the GPU with g."""
    key = torch.unique(cols.long() * m + rows.long())   # sorted by column, then row
    cols, rows = torch.div(key, m, rounding_mode="floor"), key % m
    colptr = np.zeros(n + 1, dtype=np.int64)
    colptr[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0).cpu().numpy()
    vals = value(key.numel()).cpu().numpy()
    rows, cols = rows.cpu().numpy(), cols.cpu().numpy()
    neq = int(round(0.6 * m))
    kind = host.random(n)
    x = ub * host.uniform(0.01, 0.99, n)
    x[kind < 0.3] = 0.0
    hi = (kind >= 0.3) & (kind < 0.4)
    x[hi] = ub[hi]
    b = np.bincount(rows, weights=vals * x[cols], minlength=m)
    slack = np.zeros(m, dtype=bool)
    slack[neq:] = host.random(m - neq) < 0.5
    b[slack] -= host.uniform(0.0, 1.0, int(slack.sum()))
    y = host.standard_normal(m)
    y[neq:] = np.abs(y[neq:])
    y[slack] = 0.0
    c = np.bincount(cols, weights=vals * y[rows], minlength=n)
    c[kind < 0.3] += np.abs(host.standard_normal(int((kind < 0.3).sum())))
    c[hi] -= np.abs(host.standard_normal(int(hi.sum())))
    return _Lp(m, n, neq, colptr, rows, vals, np.zeros(n), ub, c, b)


def _lp(lp, m, n, per_row, seed):
    host = np.random.default_rng(seed)
    if lp == "transport":   # m supplies, n demands: x[s, d] >= 0
        S, D = m, n
        j = np.arange(S * D)
        rows = np.stack([j % D, D + j // D], 1).reshape(-1)   # demand rows '=', supply rows '>='
        demand = host.uniform(10.0, 50.0, D)
        supply = host.uniform(50.0, 150.0, S)
        supply *= 1.1 * demand.sum() / supply.sum()
        return _Lp(S + D, S * D, D, np.arange(0, 2 * S * D + 1, 2), rows, np.tile([1.0, -1.0], S * D),
                   np.zeros(S * D), np.full(S * D, np.inf), host.uniform(1.0, 100.0, S * D),
                   np.concatenate([demand, -supply]))
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda k: torch.rand(k, generator=g, device="cuda", dtype=torch.float64)   # noqa: E731
    normal = lambda k: torch.randn(k, generator=g, device="cuda", dtype=torch.float64)   # noqa: E731
    nnz = int(m * per_row)
    if lp == "random":   # uniform pattern, N(0, 1) values, 0 <= x <= 10
        rows = torch.randint(0, m, (nnz,), generator=g, device="cuda")
        cols = torch.randint(0, n, (nnz,), generator=g, device="cuda")
        return _planted(g, host, m, n, rows, cols, normal, np.full(n, 10.0))
    # power law: column degrees with the tail of Zipf(1.5) up to 5,000, row popularity
    # proportional to rank^-0.5, values N(0, 1) x 10^U(-2, 2), 0 <= x <= U(1, 100)
    deg = torch.clamp(torch.floor(rand(n) ** -2.0), max=5000.0)
    deg = deg * (nnz / deg.sum().item())
    deg = torch.clamp(torch.floor(deg) + (rand(n) < deg - torch.floor(deg)), min=1.0, max=float(m)).long()
    cols = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    place = torch.argsort(rand(m))
    rows = place[torch.clamp((rand(cols.numel()) ** 2 * m).long(), max=m - 1)]
    return _planted(g, host, m, n, rows, cols, lambda k: normal(k) * 10.0 ** (4.0 * rand(k) - 2.0),
                    host.uniform(1.0, 100.0, n))


def _csr(p):
    """(row pointer, columns, values) of p's matrix, each row's columns increasing."""
    order = np.argsort(p.rows, kind="stable")
    ptr = np.zeros(p.m + 1, dtype=np.int32)
    np.cumsum(np.bincount(p.rows, minlength=p.m), out=ptr[1:])
    return ptr, p.cols()[order], p.vals[order]


def _members(case, seed):
    """(lp, m, n, per_row, seed) of each LP of a batch; a batch takes its LPs as they are. The
    sizes belong to the case, the data to the seed."""
    host = np.random.default_rng(case["sizes"])
    out = []
    for k in range(case["count"]):
        m = int(np.clip(round(case["median"] * math.exp(host.normal())), case["m_lo"], case["m_hi"]))
        per_row, transport = host.uniform(5.0, 40.0), host.random() < 0.25
        if transport:
            m = min(m, 2000)
            out.append(("transport", max(2, m // 5), max(2, m - m // 5), 0.0, seed * 1009 + k))
        else:
            out.append(("random", m, 2 * m, per_row, seed * 1009 + k))
    return out


def _params(case):
    p = cupdlp.default_parameters(tolerance=1e-12, iteration_limit=case["iterations"], verbosity=0)
    p.precision = cupdlp.Precision.FP64 if case["precision"] == "fp64" else cupdlp.Precision.FP32
    return p


def _vectors(p):
    none = np.zeros(0)
    return _Desc(p.n, p.m, p.neq, np.zeros(0, np.int32), np.zeros(0, np.int32), none, p.l, p.u, p.c, p.b, 0.0)


def _candidate(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    m, n = case["m"], case["n"]
    normal = lambda k: torch.randn(k, generator=g, device="cuda", dtype=torch.float64)   # noqa: E731
    u = 1.0 + 99.0 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    u[torch.rand(n, generator=g, device="cuda") < 0.2] = math.inf
    x = torch.where(u.isinf(), normal(n).abs(), 0.6 * u * normal(n).abs())
    d = {"l": torch.zeros(n, device="cuda", dtype=torch.float64), "u": u, "c": normal(n), "b": normal(m), "x": x,
         "y": normal(m)}
    d["ax"] = d["b"] + 0.1 * normal(m)
    d["aty"] = d["c"] - 0.1 * normal(n)
    return d, int(round(0.6 * m))


def prepare(case, seed):
    if case["kind"] == "check":
        d, neq = _candidate(case, seed)
        p = {k: ctypes.cast(v.data_ptr(), ctypes.POINTER(ctypes.c_double)) for k, v in d.items()}
        torch.cuda.synchronize()
        return {"kind": "check", "lib": _abi.load(), "keep": d, "out": _abi.ConvergenceInformation(),
                "args": (case["n"], case["m"], neq, 0.0, p["l"], p["u"], p["c"], p["b"], p["x"], p["y"], p["ax"],
                         p["aty"], 1e-4, 1e-4, None)}
    state = {"kind": case["kind"], "params": _params(case), "narrow": case["precision"] == "fp32"}
    if case["kind"] == "batch":
        descs = []
        for member in _members(case, seed):
            p = _lp(*member)
            descs.append(_Desc(p.n, p.m, p.neq, *_csr(p), p.l, p.u, p.c, p.b, 0.0))
        state["handle"] = DeviceBatch(descs)
        return state
    p = _lp(case["lp"], case["m"], case["n"], case["per_row"], seed)
    csc = types.SimpleNamespace(indptr=p.colptr, indices=p.rows, data=p.vals)
    if case["kind"] == "load":
        state.update(desc=_vectors(p), csc=csc)
    else:
        state["handle"] = DeviceProblem.from_csc(_vectors(p), csc, unscaled_params=state["params"])
    return state


# ---- one pass ---------------------------------------------------------------------------

_CHECKED = [f for f, t in _abi.ConvergenceInformation._fields_ if t is ctypes.c_double and f != "corrected_dual_objective"]


def _answer(state, res, x, y):
    if state["narrow"]:   # an FP32 solve's values, widened by the call
        x, y = torch.from_numpy(x).float(), torch.from_numpy(y).float()
    return {"x": x, "y": y, "iterations": int(res.iteration_count), "attempts": int(res.total_number_iterations)}


def run(state):
    if state["kind"] == "check":
        _abi.check(state["lib"].gpdhg_convergence_noalloc(*state["args"], ctypes.byref(state["out"])), state["lib"])
        return {f: getattr(state["out"], f) for f in _CHECKED}
    if state["kind"] == "load":
        with DeviceProblem.from_csc(state["desc"], state["csc"], unscaled_params=state["params"]) as handle:
            con, var = handle.rescaling()
            return {**_answer(state, *handle.solve(state["params"])), "con": con, "var": var}
    if state["kind"] == "batch":
        results, xs, ys = state["handle"].solve(state["params"])
        x, y = torch.from_numpy(np.concatenate(xs)), torch.from_numpy(np.concatenate(ys))
        return {"x": x.float() if state["narrow"] else x, "y": y.float() if state["narrow"] else y,
                "iterations": np.array([r.iteration_count for r in results]),
                "attempts": np.array([r.total_number_iterations for r in results])}
    return _answer(state, *state["handle"].solve(state["params"]))


def _sizes(lp, m, n, per_row):
    """(rows, columns, nonzeros) of one LP."""
    return (m + n, m * n, 2 * m * n) if lp == "transport" else (m, n, int(m * per_row))


def work(case):
    if case["kind"] == "check":
        return {"bytes": 8.0 * (5 * case["n"] + 3 * case["m"]), "flops": 16.0 * case["n"] + 14.0 * case["m"]}
    if case["kind"] == "batch":
        sizes = [_sizes(*member[:4]) for member in _members(case, 1)]
    else:
        sizes = [_sizes(case["lp"], case["m"], case["n"], case["per_row"])]
    m, n, nnz = (sum(s[q] for s in sizes) for q in range(3))
    t = 8 if case["precision"] == "fp64" else 4
    # an iteration: A and A' once, the step's vectors read and written once, and its operations
    step = 2 * nnz * (t + 4) + t * (11 * n + 10 * m)
    flops = 4 * nnz + 9 * n + 13 * m
    load = 2 * (12 * nnz + 8 * (4 * n + m)) if case["kind"] == "load" else 0
    return {"bytes": float(case["iterations"] * step + load + 8 * (m + n)), "flops": float(case["iterations"] * flops)}


# ---- the same in 64 bits ----------------------------------------------------------------


class _Exact:
    """rescale_problem (10 Ruiz passes, Pock-Chambolle with alpha 1) and the restarted PDHG
    loop with the default parameters, in FP64 torch."""

    def __init__(self, p, rescale):
        cuda = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device="cuda")   # noqa: E731
        self.m, self.n, self.neq = p.m, p.n, p.neq
        order = np.argsort(p.rows, kind="stable")
        rows, cols = torch.from_numpy(p.rows.astype(np.int64)).cuda(), torch.from_numpy(p.cols().astype(np.int64)).cuda()
        v = cuda(p.vals)
        self.l, self.u, self.c, self.b = cuda(p.l), cuda(p.u), cuda(p.c), cuda(p.b)
        self.con, self.var = torch.ones_like(self.b), torch.ones_like(self.c)

        def scale(v, e, d):
            e, d = torch.where(e > 0, e, 1.0).sqrt(), torch.where(d > 0, d, 1.0).sqrt()
            self.con, self.var = self.con * e, self.var * d
            self.c, self.l, self.u, self.b = self.c / d, self.l * d, self.u * d, self.b / e
            return v / (e[rows] * d[cols])

        zero = lambda like: torch.zeros_like(like)   # noqa: E731
        for _ in range(10 if rescale else 0):
            v = scale(v, zero(self.b).scatter_reduce(0, rows, v.abs(), "amax"),
                      zero(self.c).scatter_reduce(0, cols, v.abs(), "amax"))
        if rescale:
            v = scale(v, zero(self.b).index_add(0, rows, v.abs()), zero(self.c).index_add(0, cols, v.abs()))
        perm = torch.from_numpy(order).cuda()
        ptr = lambda k, size: torch.cat([zero(k[:1]), torch.bincount(k, minlength=size).cumsum(0)])   # noqa: E731
        self.A = torch.sparse_csr_tensor(ptr(rows, p.m), cols[perm], v[perm], (p.m, p.n))
        self.At = torch.sparse_csr_tensor(ptr(cols, p.n), rows, v, (p.n, p.m))
        self.amax = v.abs().max().item()

    def kkt(self, omega, x, y, kx, grad):
        """The restart scheme's score of a point."""
        fl, fu = self.l.isfinite(), self.u.isfinite()
        primal = torch.cat([self.b[:self.neq] - kx[:self.neq], (self.b - kx)[self.neq:].clamp(min=0.0),
                            (self.l - x).clamp(min=0.0), (x - self.u).clamp(min=0.0)]).norm()
        rc = torch.where(fl, grad.clamp(min=0.0), 0.0) + torch.where(fu, grad.clamp(max=0.0), 0.0)
        dual = torch.cat([(-y[self.neq:]).clamp(min=0.0), grad - rc]).norm()
        bound = torch.where(rc > 0, self.l, torch.where(rc < 0, self.u, 0.0))
        gap = (self.c.dot(x) - self.b.dot(y) - (bound * rc).sum()).abs()
        return (omega * primal ** 2 + dual ** 2 / omega + gap ** 2).sqrt().item()

    def solve(self, iterations):
        x, y = torch.zeros_like(self.c), torch.zeros_like(self.b)
        kx, kty = torch.zeros_like(y), torch.zeros_like(x)
        tau, omega = 1.0 / self.amax, 1.0
        if self.c.norm() > 0 and self.b.norm() > 0:
            omega = (self.c.norm() / self.b.norm()).item()
        sx, sy, skx, weight, count = torch.zeros_like(x), torch.zeros_like(y), torch.zeros_like(y), 0.0, 0
        last, last_ratio, attempts, it = (x, y, kx, self.c - kty), 1.0, 0, 1
        while True:
            if (it - 1) % EVALUATE_EVERY == 0 or it == iterations + 1 or it <= 10:
                ax, ay, akx = (sx / weight, sy / weight, skx / weight) if count else (x, y, kx)
                if it - 1 >= iterations:
                    return ax, ay, it - 1, attempts
                if count:
                    agrad = self.c - self.At @ ay
                    cur, avg = self.kkt(omega, x, y, kx, self.c - kty), self.kkt(omega, ax, ay, akx, agrad)
                    restart, best = count >= 0.36 * (it - 1), min(cur, avg)
                    if not restart:
                        ratio = best / self.kkt(omega, *last)
                        restart = ratio < 0.8 and (ratio < 0.2 or ratio > last_ratio)
                        last_ratio = ratio
                    if restart:
                        dx, dy = (ax - last[0]).norm().item(), (ay - last[1]).norm().item()
                        if cur >= avg:
                            x, y, kx, kty = ax, ay, akx, self.c - agrad
                        last = (x, y, kx, self.c - kty)
                        sx, sy, skx = torch.zeros_like(x), torch.zeros_like(y), torch.zeros_like(y)
                        weight, count = 0.0, 0
                        if dx / math.sqrt(tau) > 2.3e-16 and dy / math.sqrt(tau) > 2.3e-16:
                            omega = math.exp(0.5 * math.log(dy / dx) + 0.5 * math.log(omega))
            begin = tau
            while True:
                nx = torch.minimum(self.u, torch.maximum(self.l, x - (tau / omega) * (self.c - kty)))
                dx = nx - x
                kdx = self.A @ dx
                ny = y + (omega * tau) * (self.b - 2.0 * kdx - kx)
                ny[self.neq:].clamp_(min=0.0)
                dy = ny - y
                cross = abs(dy.dot(kdx).item())
                move = 0.5 * omega * dx.dot(dx).item() + 0.5 / omega * dy.dot(dy).item()
                limit = move / cross if cross > 0 else math.inf
                attempts += 1
                accept = tau <= limit
                tau = min((1.0 - (attempts + 1.0) ** -0.3) * limit, (1.0 + (attempts + 1.0) ** -0.6) * tau)
                if accept:
                    break
            x, y, kx = nx, ny, kx + kdx
            kty = self.At @ y
            sx, sy, skx = sx + begin * x, sy + begin * y, skx + begin * kx
            weight, count, it = weight + begin, count + 1, it + 1


def exact(case, seed):
    if case["kind"] == "check":
        d, neq = _candidate(case, seed)
        x, y, c, b, u = d["x"], d["y"], d["c"], d["b"], d["u"]
        cv = b - d["ax"]
        cv[neq:].clamp_(min=0.0)
        primal = torch.cat([cv, (-x).clamp(min=0.0), (x - u).clamp(min=0.0)])
        grad = c - d["aty"]
        rc = torch.where(u.isinf(), grad.clamp(min=0.0), grad)
        dual = torch.cat([(-y[neq:]).clamp(min=0.0), grad - rc])
        pobj = c.dot(x).item()
        dobj = (b.dot(y) + torch.where(rc < 0, u * rc, 0.0).sum()).item()
        inf = lambda v: v.abs().max().item()   # noqa: E731
        pi, p2, di, d2 = inf(primal), primal.norm().item(), inf(dual), dual.norm().item()
        return dict(zip(_CHECKED, [
            pobj, dobj, pi, p2, di, d2, pi / (1 + inf(b)), p2 / (1 + b.norm().item()), di / (1 + inf(c)),
            d2 / (1 + c.norm().item()), abs(pobj - dobj) / (1 + abs(pobj) + abs(dobj)), inf(x), x.norm().item(), inf(y),
            y.norm().item()]))
    if case["kind"] == "batch":
        out = [_Exact(_lp(*member), False).solve(case["iterations"]) for member in _members(case, seed)]
        return {"x": torch.cat([o[0] for o in out]), "y": torch.cat([o[1] for o in out]),
                "iterations": np.array([o[2] for o in out]), "attempts": np.array([o[3] for o in out])}
    e = _Exact(_lp(case["lp"], case["m"], case["n"], case["per_row"], seed), True)
    x, y, iterations, attempts = e.solve(case["iterations"])
    out = {"x": x, "y": y, "iterations": iterations, "attempts": attempts}
    return {**out, "con": e.con, "var": e.var} if case["kind"] == "load" else out
