"""The evaluation passes at the edges of their items (1,024 elements, two CTAs of 128 threads each)."""
import pytest

import cupdlp
from test_gpu_evaluation_edges import test_solver_statistics_match_noalloc as _statistics_match

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cupdlp.Precision.FP64, cupdlp.Precision.FP32])
@pytest.mark.parametrize("n", [64, 127, 128, 129, 256, 1023, 1024, 1025, 2049])
def test_statistics_at_item_edges(n, precision):
    _statistics_match(n, precision)
