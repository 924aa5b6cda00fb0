"""Small LPs run their step attempts on one thread-block cluster, larger ones (and every profiled
solve) as launches of the step kernels: both routes add every sum in the same order, so their
results are the same bits, on either side of the rule and at the edges of tiles and vectors."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import cupdlp
from cupdlp import _abi, synthetic
from cupdlp.solver import DeviceProblem, scaled_desc

import instances

pytestmark = pytest.mark.gpu


def _solve(dp, params, profile):
    cp = cupdlp.params_to_c(params)
    cp.profile_kernels = int(profile)
    res = _abi.Result()
    x, y = np.empty(dp.n), np.empty(dp.m)
    _abi.check(dp.lib.gpdhg_solve(dp.handle, C.byref(cp), C.byref(res), _abi.dptr(x), _abi.dptr(y)), dp.lib)
    return res, x, y, dp.current_iterate()


def _random(m, n, density, seed=3):
    return lambda: synthetic.known_optimum_lp(seed, m=m, n=n, density=density).problem


def _one_dense_row(n, m=40, seed=9):
    rng = np.random.default_rng(seed)
    a = sp.random(m, n, density=0.02, random_state=seed, format="lil")
    a[m - 1, :] = rng.uniform(0.5, 1.5, n)
    return lambda: instances.lp(sp.csc_matrix(a), np.full(m, -1.0), rng.standard_normal(n), np.zeros(n), np.full(n, 5.0), 3)


# (problem, on the cluster in FP64, in FP32); None: either
CASES = {
    "tiny": (lambda: instances.tiny()[0], True, True),
    "no_constraints": (instances.no_constraints, None, None),
    "empty_rows_and_columns": (instances.empty_rows_and_columns, True, True),
    "1x1": (_random(1, 1, 1.0), True, True),
    "31x33": (_random(31, 33, 0.3), True, True),
    "256x257": (_random(256, 257, 0.04), True, True),
    "1000x2000": (_random(1000, 2000, 0.005), True, True),
    "2100x300": (_random(2100, 300, 0.02), None, None),
    "several_rounds": (_random(6000, 7000, 0.0006), True, True),
    "too_many_rows": (_random(30_000, 20_000, 0.0002), False, False),
    "row_of_1500": (_one_dense_row(1500), None, None),
    "row_of_9000": (_one_dense_row(9000), False, False),
}


@pytest.mark.parametrize("precision", [cupdlp.Precision.FP64, cupdlp.Precision.FP32])
@pytest.mark.parametrize("name", list(CASES))
def test_same_bits_as_step_kernels(name, precision):
    make, on64, on32 = CASES[name]
    params = cupdlp.default_parameters(tolerance=1e-10, iteration_limit=230, precision=precision)
    sq = cupdlp.rescale_problem(10, False, 1.0, 0, make())
    with DeviceProblem(scaled_desc(sq)) as dp:
        got, x, y, cur = _solve(dp, params, False)
        again = _solve(dp, params, False)
        want, xw, yw, curw = _solve(dp, params, True)
    assert (got.iteration_count, got.termination_reason) == (want.iteration_count, want.termination_reason)
    for a, b in ((x, xw), (y, yw), (cur[0], curw[0]), (cur[1], curw[1]), (x, again[1]), (y, again[2])):
        np.testing.assert_array_equal(a, b)
    expected = on64 if precision == cupdlp.Precision.FP64 else on32
    if expected is not None:   # one launch per interval instead of two per attempt
        assert (got.kernels_launched < want.kernels_launched) == expected
