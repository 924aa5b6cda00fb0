"""Runs of rows of 257 to 2,048 nonzeros are summed by a warp each in the plain product (A' of the
average), isolated and longer ones by a whole CTA: lengths at the edges of a
warp's rounds, in runs on both sides of the rule, against the oracle."""
import numpy as np
import pytest
import scipy.sparse as sp

import instances
from test_gpu_parity import _params, compare_strict, solve_both

pytestmark = pytest.mark.gpu

RUNS = ((257, 288, 289, 300), (511, 512, 513, 2047, 2048), (2049, 256, 257), (600,) * 9, (255, 1025, 700, 2100, 2048))


def _lp(seed=13, m=2200, n=600):
    """Column lengths in the order of RUNS, short columns between."""
    rng = np.random.default_rng(seed)
    cols, rows = [], []
    j = 0
    for run in RUNS:
        for length in run + (2, 3):
            rows.append(rng.choice(m, size=length, replace=False))
            cols.append(np.full(length, j))
            j += 1
    rest = np.repeat(np.arange(j, n), 4)
    rows.append(rng.integers(0, m, rest.size))
    cols.append(rest)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    a = sp.csc_matrix((rng.uniform(0.5, 1.5, rows.size) * rng.choice([-1.0, 1.0], rows.size), (rows, cols)), shape=(m, n))
    x = rng.uniform(0.0, 1.0, n)
    b = a @ x
    y = rng.standard_normal(m)
    y[1000:] = np.abs(y[1000:])
    return instances.lp(a, b, a.T @ y, np.zeros(n), np.full(n, 10.0), 1000)


@pytest.mark.parametrize("iters", [1, 12])
def test_matches_oracle(iters):
    p = _lp()
    sq, (res, xa, ya, stats, xc, yc), orc, _ = solve_both(p, _params(tolerance=1e-10, iteration_limit=iters))
    assert res.iteration_count == orc.result.iteration_count
    compare_strict(stats, orc, rtol=1e-9)
    for got, want in ((xc, orc.x_cur), (yc, orc.y_cur)):
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-9 * max(1.0, np.abs(want).max()))
