"""gpdhg_convergence_noalloc where its split over CTAs changes (256 elements per CTA up to 153,600 on
both sides together, 600 CTAs per side at most beyond) and at the longest vectors it takes."""
import ctypes as C

import pytest

import cupdlp
from cupdlp import _abi

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LIMIT = 16_777_216


@pytest.mark.parametrize("n,m", [(153_599, 1), (153_600, 1), (1, 153_599), (76_801, 76_800), (LIMIT, 1), (1, LIMIT),
                                 (LIMIT, LIMIT)])
def test_statistics(n, m):
    lib = _abi.load()
    g = torch.Generator(device="cuda").manual_seed(n ^ m)
    new = lambda k: torch.randn(k, generator=g, device="cuda", dtype=torch.float64)   # noqa: E731
    u = 1.0 + new(n).abs()
    c, b, x, y, ax, aty = new(n), new(m), 2.0 * new(n), new(m), new(m), new(n)
    low, neq = torch.zeros_like(u), m // 3
    ptr = lambda t: C.cast(C.c_void_p(t.data_ptr()), _abi._dp)   # noqa: E731
    out = _abi.ConvergenceInformation()
    torch.cuda.synchronize()
    _abi.check(lib.gpdhg_convergence_noalloc(n, m, neq, 0.0, *map(ptr, (low, u, c, b, x, y, ax, aty)), 1e-4, 1e-4, None,
                                             C.byref(out)), lib)
    cv = b - ax
    cv[neq:].clamp_(min=0.0)
    primal = torch.cat([cv, (-x).clamp(min=0.0), (x - u).clamp(min=0.0)])
    dual = (-y[neq:]).clamp(min=0.0)   # finite bounds: every reduced cost is kept
    want = {"l2_primal_variable": x.norm(), "l2_dual_variable": y.norm(), "l_inf_primal_variable": x.abs().max(),
            "l_inf_dual_variable": y.abs().max(), "l2_primal_residual": primal.norm(),
            "l_inf_primal_residual": primal.abs().max(), "l2_dual_residual": dual.norm(),
            "l_inf_dual_residual": dual.max() if m > neq else torch.zeros(())}
    # sums of non-negative terms, at most 2^16 roundings deep, in both: 2^17 x 2^-53 = 1.5e-11
    for field, value in want.items():
        assert getattr(out, field) == pytest.approx(value.item(), rel=1.5e-11), field
