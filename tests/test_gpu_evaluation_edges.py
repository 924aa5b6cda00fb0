"""The evaluation statistics at the edges of their segments, on values that take every selection of
the reduced-cost and bound arithmetic: infinite and finite bounds (zero among them), violated and
exactly met bounds, zero, negative and subnormal entries."""
import ctypes as C

import numpy as np
import pytest

import cupdlp
from cupdlp import _abi

pytestmark = pytest.mark.gpu


def _reference(l, u, c, b, x, y, ax, aty, neq):
    cv = b - ax
    cv[neq:] = np.maximum(cv[neq:], 0.0)
    primal = np.concatenate([cv, np.maximum(l - x, 0.0), np.maximum(x - u, 0.0)])
    g = c - aty
    rc = np.maximum(g, 0.0) * np.isfinite(l) + np.minimum(g, 0.0) * np.isfinite(u)
    dual = np.concatenate([np.maximum(-y[neq:], 0.0), g - rc])
    with np.errstate(invalid="ignore"):
        terms = np.where(rc > 0, l * rc, np.where(rc < 0, u * rc, 0.0))
    inf = lambda v: float(np.max(np.abs(v), initial=0.0))  # noqa: E731
    values = dict(primal_objective=c @ x, dual_objective=b @ y + terms.sum(), l_inf_primal_residual=inf(primal),
                  l2_primal_residual=np.linalg.norm(primal), l_inf_dual_residual=inf(dual),
                  l2_dual_residual=np.linalg.norm(dual), l_inf_primal_variable=inf(x),
                  l2_primal_variable=np.linalg.norm(x), l_inf_dual_variable=inf(y), l2_dual_variable=np.linalg.norm(y))
    # a sum of k terms rounds by at most k eps times the sum of magnitudes; norms are relative
    slack = dict(primal_objective=np.abs(c * x).sum(), dual_objective=np.abs(b * y).sum() + np.abs(terms).sum())
    return values, slack


@pytest.mark.parametrize("n,m", [(1, 0), (1, 1), (31, 33), (255, 256), (257, 511), (153_600, 1), (100_003, 60_001),
                                 (1, 200_000)])
def test_noalloc_statistics(n, m):
    import torch
    rng = np.random.default_rng(n * 7 + m)
    l = np.where(rng.random(n) < 0.3, -np.inf, rng.choice([0.0, -1.5, 2.0], n))
    u = np.where(rng.random(n) < 0.3, np.inf, np.maximum(np.where(np.isfinite(l), l, 0.0), 0.0) + rng.choice([0.0, 3.0], n))
    x = rng.choice([0.0, -0.0, 1.0, -2.5, 2.0, 3.0, 5e-310], n) + rng.choice([0.0, 1e-3], n)
    c, aty = rng.standard_normal(n), rng.standard_normal(n)
    aty[rng.random(n) < 0.2] = 0.0
    c[rng.random(n) < 0.2] = 0.0
    b, ax = rng.standard_normal(m), rng.standard_normal(m)
    y = rng.choice([0.0, -0.0, 1.0, -0.25, -5e-310], m)
    neq = m // 2
    want, slack = _reference(l, u, c, b.copy(), x, y, ax, aty, neq)
    dev = [torch.from_numpy(v).cuda() if v.size else None for v in (l, u, c, b, x, y, ax, aty)]
    ptr = [C.cast(d.data_ptr() if d is not None else None, _abi._dp) for d in dev]
    out = _abi.ConvergenceInformation()
    lib = _abi.load()
    torch.cuda.synchronize()
    _abi.check(lib.gpdhg_convergence_noalloc(n, m, neq, 0.0, *ptr, 1e-4, 1e-4, None, C.byref(out)), lib)
    eps = np.finfo(np.float64).eps
    for name, value in want.items():
        got = getattr(out, name)
        tol = (n + m) * eps * (slack.get(name, 0.0) + abs(value)) if not name.startswith("l_inf") else 2 * eps * abs(value)
        assert abs(got - value) <= tol, (name, got, value)


@pytest.mark.parametrize("precision", [cupdlp.Precision.FP64, cupdlp.Precision.FP32])
@pytest.mark.parametrize("n", [255, 257, 33_001, 120_000])
def test_solver_statistics_match_noalloc(n, precision):
    """The statistics a solve reports for its averaged iterate are those of that iterate computed
    anew (FP64 from the returned point, so FP32 differs by its products' rounding)."""
    import torch
    from cupdlp import synthetic
    lp = synthetic.known_optimum_lp(n, m=n // 2, n=n, density=min(0.05, 8.0 / n)).problem
    lp.variable_upper_bound[::3] = np.inf
    lp.variable_lower_bound[::5] = -np.inf
    params = cupdlp.default_parameters(tolerance=1e-12, iteration_limit=20, precision=precision)
    sq = cupdlp.rescale_problem(10, False, 1.0, 0, lp)
    with cupdlp.DeviceProblem(cupdlp.scaled_desc(sq)) as dp:
        res, xs, ys = dp.solve(params)
    x, y = xs / sq.variable_rescaling, ys / sq.constraint_rescaling
    A = lp.constraint_matrix
    arrays = (lp.variable_lower_bound, lp.variable_upper_bound, lp.objective_vector, lp.right_hand_side, x, y, A @ x,
              A.T @ y)
    dev = [torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64)).cuda() for v in arrays]
    out = _abi.ConvergenceInformation()
    lib = _abi.load()
    torch.cuda.synchronize()
    _abi.check(lib.gpdhg_convergence_noalloc(n, n // 2, lp.num_equalities, 0.0,
                                             *[C.cast(d.data_ptr(), _abi._dp) for d in dev], 1e-4, 1e-4, None,
                                             C.byref(out)), lib)
    got = res.last_iteration_stats.convergence_information
    rtol = 1e-9 if precision == cupdlp.Precision.FP64 else 1e-4
    for name in ("primal_objective", "l2_primal_residual", "l2_dual_residual", "l2_primal_variable", "l2_dual_variable"):
        a, b = getattr(got, name), getattr(out, name)
        assert abs(a - b) <= rtol * max(1.0, abs(b)), (name, a, b)
