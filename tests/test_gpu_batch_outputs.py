"""A batch hands its solutions out in runs of neighbouring instances that ended together: reordered and
plain instances, an instance that ends first (alone) between neighbours that end later, instances
without rows, and callers that want only some of the arrays."""
import ctypes as C

import numpy as np
import pytest

import cupdlp
from cupdlp import _abi, synthetic
from cupdlp.solver import DeviceBatch, DeviceProblem, scaled_desc

import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cupdlp.Precision.FP64, cupdlp.Precision.FP32])
def test_runs_and_null_outputs(precision):
    skewed = [synthetic.power_law_lp(seed, m=1500, n=5000, target_nnz=40_000).problem for seed in (1, 2, 3)]
    problems = [skewed[0], synthetic.known_optimum_lp(5, m=90, n=140, density=0.1).problem, instances.tiny()[0],
                instances.no_constraints(), skewed[1], skewed[2]]
    params = cupdlp.default_parameters(tolerance=1e-4, iteration_limit=70, precision=precision)
    scaled = [scaled_desc(cupdlp.rescale_problem(10, False, 1.0, 0, p)) for p in problems]
    alone = []
    for d in scaled:
        with DeviceProblem(d) as dp:
            alone.append(dp.solve(params))
    assert len({r.iteration_count for r, _, _ in alone}) > 1   # some end before the others
    fill = -7.25
    with DeviceBatch(scaled) as db:
        cp = cupdlp.params_to_c(params)
        for want_x, want_y in (([1] * 6, [1] * 6), ([1, 0, 1, 0, 1, 1], [0, 1, 1, 0, 0, 1]), ([0] * 6, [1] * 6), ([1] * 6, None)):
            results = (_abi.Result * 6)()
            xs = [np.full(d.desc.num_variables, fill) for d in scaled]
            ys = [np.full(max(d.desc.num_constraints, 1), fill) for d in scaled]
            xp = (_abi._dp * 6)(*[_abi.dptr(x if w else None) for x, w in zip(xs, want_x)])
            yp = (_abi._dp * 6)(*[_abi.dptr(y if w else None) for y, w in zip(ys, want_y)]) if want_y else None
            _abi.check(db.lib.gpdhg_batch_solve(db.handle, C.byref(cp), results, xp, yp), db.lib)
            for k, (r, x, y) in enumerate(alone):
                assert results[k].iteration_count == r.iteration_count, k
                np.testing.assert_array_equal(xs[k], x if want_x[k] else fill)
                np.testing.assert_array_equal(ys[k][:y.size], y if want_y and want_y[k] else fill)
