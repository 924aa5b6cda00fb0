"""Intervals of more step attempts than one launch of the cluster kernel takes (8,192): the launch that
ends short of its interval leaves the state from which the next goes on, and the evaluation between
them does nothing, so the results are the bits of the step kernels."""
import ctypes as C

import numpy as np
import pytest

import cupdlp
from cupdlp import _abi, synthetic
from cupdlp.solver import DeviceProblem, scaled_desc

pytestmark = pytest.mark.gpu

ITERATIONS = 17_000   # from the tenth on one interval: three launches


def _solve(dp, precision, constant, profile):
    params = cupdlp.default_parameters(tolerance=1e-15, iteration_limit=ITERATIONS, precision=precision)
    params.termination_evaluation_frequency = 1 << 20
    cp = cupdlp.params_to_c(params)
    cp.step_size_policy, cp.profile_kernels = int(constant), int(profile)
    res = _abi.Result()
    x, y = np.empty(dp.n), np.empty(dp.m)
    _abi.check(dp.lib.gpdhg_solve(dp.handle, C.byref(cp), C.byref(res), _abi.dptr(x), _abi.dptr(y)), dp.lib)
    return res, x, y, dp.current_iterate()


@pytest.mark.parametrize("constant", [False, True])
@pytest.mark.parametrize("precision", [cupdlp.Precision.FP64, cupdlp.Precision.FP32])
@pytest.mark.parametrize("m,n,density", [(31, 33, 0.3), (256, 257, 0.04)])
def test_same_bits_across_launches(m, n, density, precision, constant):
    p = synthetic.known_optimum_lp(3, m=m, n=n, density=density).problem
    with DeviceProblem(scaled_desc(cupdlp.rescale_problem(10, False, 1.0, 0, p))) as dp:
        got, x, y, cur = _solve(dp, precision, constant, False)
        want, xw, yw, curw = _solve(dp, precision, constant, True)
    assert got.iteration_count == want.iteration_count == ITERATIONS
    assert (got.accepted_steps, got.rejected_steps) == (want.accepted_steps, want.rejected_steps)
    assert got.kernels_launched < 200 < want.kernels_launched   # on the cluster
    for a, b in ((x, xw), (y, yw), (cur[0], curw[0]), (cur[1], curw[1])):
        np.testing.assert_array_equal(a, b)
