"""Panel factorisation with one and with two levels of its pivot tree: random matrices (pivots from
every block of rows) at the edges of the row blocks (256 rows to a CTA, 32 CTAs, 512 rows), ragged last
panels, in mixed precision and FP64, judged by the residual of the solve.

Tolerance: the solve's own target 1e-12 (mixed: refined until it is met; a factor of a wrong
permutation or a missing pivot does not converge), times 10 for the norm (largest entry against the
solver's own)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 33, 256, 257, 289, 1025, 2050, 8200])
@pytest.mark.parametrize("form", ["SOLVE_MIXED_IR", "SOLVE_FP64"])
def test_solve_residual(n, form):
    import torch

    import ibemproject_gb300 as g
    if form == "SOLVE_FP64" and n > 2100:
        pytest.skip("the FP64 tree has two levels from three CTAs on")
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen)
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
    At = A.t().contiguous()   # column-major storage
    x = torch.empty_like(b)
    keep = At.clone()
    rep = g.SolveReport()
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    g.check(g.lib().ibem_e3d_solve(getattr(g, form), n, P(keep), n, P(b), P(x), 1e-12, ctypes.byref(rep), None))
    torch.cuda.synchronize()
    r = (b - A @ x).abs().max().item()
    scale = A.abs().sum(dim=1).max().item() * x.abs().max().item() + b.abs().max().item()
    assert r <= 1e-11 * scale, (r, scale)
