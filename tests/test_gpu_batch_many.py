"""A batch of more instances than a grid's second dimension takes (65,535): its instances give the
same bits as solved alone."""
import numpy as np
import pytest

import cupdlp
from cupdlp import synthetic
from cupdlp.solver import DeviceBatch, DeviceProblem, scaled_desc

import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [65_535, 65_536, 70_001])
def test_more_than_65535_instances(count):
    kinds = [instances.tiny()[0], instances.empty_rows_and_columns(),
             synthetic.known_optimum_lp(3, m=3, n=5, density=0.7).problem]
    params = cupdlp.default_parameters(tolerance=1e-10, iteration_limit=25)
    descs = [scaled_desc(cupdlp.rescale_problem(10, False, 1.0, 0, p)) for p in kinds]
    alone = []
    for d in descs:
        with DeviceProblem(d) as dp:
            alone.append(dp.solve(params))
    with DeviceBatch([descs[k % len(descs)] for k in range(count)]) as db:
        results, xs, ys = db.solve(params)
    for k in range(count):
        want, x, y = alone[k % len(descs)]
        assert (results[k].termination_reason, results[k].iteration_count, results[k].total_number_iterations) == \
            (want.termination_reason, want.iteration_count, want.total_number_iterations), k
        assert np.array_equal(xs[k], x) and np.array_equal(ys[k], y), k
