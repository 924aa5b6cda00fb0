"""The plain product on rows of A' around the lengths at which a warp, a warp of a run of long rows or
a whole CTA sums them: integer data, exact in FP32 in any order, through the statistics of a warm
start's own point (dual residual c - A'y of free variables)."""
import numpy as np
import pytest
import scipy.sparse as sp

import cupdlp
from cupdlp.solver import DeviceProblem, unscaled_desc

import instances
from test_gpu_long_row_runs import RUNS

pytestmark = pytest.mark.gpu


def _lp(order, m=2300, seed=4):
    rng = np.random.default_rng(seed)
    lengths = [k for run in order for k in run + (0, 1, 3)]
    rows = np.concatenate([rng.choice(m, size=k, replace=False) for k in lengths])
    cols = np.repeat(np.arange(len(lengths)), lengths)
    a = sp.csc_matrix((rng.integers(1, 9, rows.size) * rng.choice([-1.0, 1.0], rows.size), (rows, cols)),
                      shape=(m, len(lengths)))
    n = len(lengths)
    free = np.full(n, np.inf)
    return instances.lp(a, np.zeros(m), rng.integers(-50, 50, n), -free, free, m), rng.integers(-20, 20, m).astype(float)


@pytest.mark.parametrize("precision", [cupdlp.Precision.FP64, cupdlp.Precision.FP32])
@pytest.mark.parametrize("order", [RUNS, RUNS[::-1], ((257,) * 8, (2048,) * 3, (2049,) * 4, (1, 512) * 5)])
def test_exact_products(order, precision):
    p, y = _lp(order)
    want = p.objective_vector - p.constraint_matrix.T @ y
    params = cupdlp.default_parameters(iteration_limit=0, precision=precision)
    with DeviceProblem(unscaled_desc(p)) as dp:
        dp.set_warm_start(None, y)
        res, _, _ = dp.solve(params)
    ci = res.last_iteration_stats.convergence_information
    assert (res.iteration_count, ci.l_inf_dual_residual) == (0, np.abs(want).max())
    assert ci.l2_dual_residual == pytest.approx(np.sqrt((want ** 2).sum()), rel=1e-15)
