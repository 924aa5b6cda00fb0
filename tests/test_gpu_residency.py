"""A step kernel is compiled for 2, 3 and 4 resident CTAs per SM and chosen by its number of CTAs (up
to 304, up to 456, more). A lone LP of each size and the same LP three times in a batch, whose CTAs
then take another choice, give the same bits."""
import numpy as np
import pytest

import cupdlp
from cupdlp import synthetic
from cupdlp.solver import DeviceBatch, DeviceProblem, scaled_desc

pytestmark = pytest.mark.gpu


# rows of 20 nonzeros: an FP64 CTA takes about 47 rows, an FP32 CTA about 98
@pytest.mark.parametrize("precision,m", [(cupdlp.Precision.FP64, 8000), (cupdlp.Precision.FP64, 14_400),
                                         (cupdlp.Precision.FP64, 18_000), (cupdlp.Precision.FP64, 23_000),
                                         (cupdlp.Precision.FP32, 20_000), (cupdlp.Precision.FP32, 36_000)])
def test_choices_agree(precision, m):
    p = synthetic.known_optimum_lp(4, m=m, n=2 * m, density=10.0 / m).problem
    params = cupdlp.default_parameters(tolerance=1e-10, iteration_limit=25, precision=precision)
    sq = cupdlp.rescale_problem(10, False, 1.0, 0, p)
    with DeviceProblem(scaled_desc(sq)) as dp:
        res, x, y = dp.solve(params)
    with DeviceBatch([scaled_desc(sq)] * 3) as db:
        results, xs, ys = db.solve(params)
    for r, xb, yb in zip(results, xs, ys):
        assert (r.iteration_count, r.total_number_iterations) == (res.iteration_count, res.total_number_iterations)
        np.testing.assert_array_equal(xb, x)
        np.testing.assert_array_equal(yb, y)
