"""The line between the cluster kernel and the step kernels for a lone LP: two plan CTAs per CTA of the
cluster and side. Just inside and outside of it, the routes and their bits."""
import pytest

import cupdlp
from cupdlp import synthetic
from cupdlp.solver import DeviceProblem, scaled_desc

import numpy as np
from test_gpu_cluster_route import _solve

pytestmark = pytest.mark.gpu


# about 20 nonzeros per row: an FP64 plan CTA takes about 48 rows, an FP32 one about 98
@pytest.mark.parametrize("precision,m,cluster", [(cupdlp.Precision.FP64, 1450, True), (cupdlp.Precision.FP64, 1750, False),
                                                 (cupdlp.Precision.FP32, 2900, True), (cupdlp.Precision.FP32, 3600, False)])
def test_route_and_bits(precision, m, cluster):
    p = synthetic.known_optimum_lp(8, m=m, n=2 * m, density=10.0 / m).problem
    params = cupdlp.default_parameters(tolerance=1e-10, iteration_limit=150, precision=precision)
    with DeviceProblem(scaled_desc(cupdlp.rescale_problem(10, False, 1.0, 0, p))) as dp:
        got, x, y, _ = _solve(dp, params, False)
        want, xw, yw, _ = _solve(dp, params, True)
    assert (got.kernels_launched < want.kernels_launched) == cluster
    np.testing.assert_array_equal(x, xw)
    np.testing.assert_array_equal(y, yw)
