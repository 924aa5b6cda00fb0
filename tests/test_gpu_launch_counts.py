"""gpdhg_result.kernels_launched counts every kernel of a solve: those of the intervals' graphs and those
launched around them (a warm start's products, the power method of the constant step size, the
FP64 hand-off). One iteration from the zero start, whose launches can be added up by hand."""
import ctypes as C
import math

import numpy as np
import pytest

import cupdlp
from cupdlp import _abi, synthetic
from cupdlp.solver import DeviceProblem, scaled_desc

pytestmark = pytest.mark.gpu

EVALUATION = 5   # row pass, commit, A'y, column pass, sums
# (rows, columns, density, its attempts run on a cluster)
SIZES = [(300, 500, 0.02, True), (30_000, 20_000, 0.0002, False)]


def _launched(dp, precision, profile=False, constant=False, handoff=0.0):
    cp = cupdlp.params_to_c(cupdlp.default_parameters(tolerance=1e-12, iteration_limit=1, precision=precision))
    cp.profile_kernels, cp.step_size_policy, cp.fp64_handoff_relative_kkt = int(profile), int(constant), handoff
    for _ in range(2):   # the first solve also lays the workspace out
        res = _abi.Result()
        _abi.check(dp.lib.gpdhg_solve(dp.handle, C.byref(cp), C.byref(res), None, None), dp.lib)
    assert res.iteration_count == 1
    return res.kernels_launched, res.accepted_steps + res.rejected_steps


def _interval(attempts, cluster):
    """The state's copy, the attempts and the evaluation: a rejected attempt of the step kernels takes
    another launch."""
    return 1 + 1 + EVALUATION if cluster else attempts * (1 + 2 + EVALUATION)


def _power_iterations(n):
    """estimate_maximum_singular_value's, src/primal_dual_hybrid_gradient_gpu.jl:139-172."""
    eps, k = 1.0 - 0.8 ** 2, 0
    while (1.0 if k < 2 else min(0.824, 0.354 / math.sqrt(eps * (k - 1))) * math.sqrt(n) * (1 - eps) ** (k - 0.5)) > 0.001:
        k += 1
    return k


@pytest.mark.parametrize("m,n,density,cluster", SIZES)
def test_launches_add_up(m, n, density, cluster):
    p = synthetic.known_optimum_lp(6, m=m, n=n, density=density).problem
    first = 1 + 1 + EVALUATION   # the gradient, the state's copy, the evaluation of the start
    with DeviceProblem(scaled_desc(cupdlp.rescale_problem(10, False, 1.0, 0, p))) as dp:
        for precision in (cupdlp.Precision.FP64, cupdlp.Precision.FP32):
            got, attempts = _launched(dp, precision)
            assert got == first + _interval(attempts, cluster)
            got, attempts = _launched(dp, precision, profile=True)
            assert got == first + _interval(attempts, False)
            got, attempts = _launched(dp, precision, constant=True)
            k = _power_iterations(n)   # two products and the norm each, then two products and two dot products
            assert got == first + _interval(attempts, cluster) + 4 * k + 2 + 4
        got, attempts = _launched(dp, cupdlp.Precision.FP32_REFINE, handoff=1e30)   # at the start's evaluation
        handoff = 16 + 2 + 1   # vectors converted, exact products, gradient
        assert got == first + handoff + 1 + EVALUATION + _interval(attempts, cluster)
        dp.set_warm_start(np.zeros(n), np.zeros(m))
        got, attempts = _launched(dp, cupdlp.Precision.FP64)
        assert got == first + 2 + _interval(attempts, cluster)
