"""Handing a solution out allocates no device memory: what it needs is laid out with the workspace, so a
shortage shows before the iterations and the server's estimate of a request holds to its end."""
import numpy as np
import pytest

import cupdlp
from cupdlp import synthetic
from cupdlp.solver import DeviceBatch, DeviceProblem, scaled_desc

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _desc(seed):   # renumbered columns; vectors of several of the allocator's 2 MB pages
    p = synthetic.power_law_lp(seed, m=150_000, n=600_000, target_nnz=1_500_000).problem
    return scaled_desc(cupdlp.rescale_problem(2, False, 1.0, 0, p))


@pytest.mark.parametrize("precision", [cupdlp.Precision.FP64, cupdlp.Precision.FP32])
def test_no_allocation_at_the_end(precision):
    torch.zeros(1, device="cuda")
    params = cupdlp.default_parameters(tolerance=1e-12, iteration_limit=5, precision=precision)
    descs = [_desc(1), _desc(2)]
    with DeviceProblem(descs[0]) as dp:
        dp.solve(params, want_solution=False)
        before = _free()
        _, x, y = dp.solve(params)
        assert _free() == before
    with DeviceBatch(descs) as db:
        db.solve(params, want_solution=False)
        before = _free()
        _, xs, ys = db.solve(params)
        assert _free() == before
    np.testing.assert_array_equal(xs[0], x)
    np.testing.assert_array_equal(ys[0], y)
