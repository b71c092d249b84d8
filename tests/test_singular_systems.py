"""Singular systems in the plain FP64 solve: equations given twice, in numbers that FP64 arithmetic
cancels exactly, are refused with a zero pivot, whatever unit the trailing updates run on; a
nearly singular system, whose pivots are as small, is still solved to its backward error.

Half of the rows are copies, so that a zero pivot does not hang on the rounding of one row: the
factorisation meets N / 2 of them.  Backward error of the nearly singular ones: N 2^-53, as for the
others."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(A, b, noalloc=False):
    import torch

    import ibemproject_gb300 as g
    n = len(b)
    At, bt = torch.from_numpy(np.ascontiguousarray(A.T)).cuda(), torch.from_numpy(b).cuda()
    x, rep = torch.zeros(n, dtype=torch.float64, device="cuda"), g.SolveReport()
    if noalloc:
        st = g.lib().ibem_e3d_solve_noalloc(n, At.data_ptr(), n, bt.data_ptr(), x.data_ptr(), ctypes.byref(rep), None)
    else:
        st = g.lib().ibem_e3d_solve(g.SOLVE_FP64, n, At.data_ptr(), n, bt.data_ptr(), x.data_ptr(), 1e-12, ctypes.byref(rep),
                                    None)
    return st, x.cpu().numpy(), rep


@pytest.mark.parametrize("n", [40, 64, 100, 128, 160, 256, 300, 400, 600, 1000, 2000])
def test_equations_given_twice(n):
    import ibemproject_gb300 as g
    rng = np.random.default_rng(n)
    A = np.repeat(rng.integers(-3, 4, (n // 2, n)).astype(float), 2, axis=0)
    st, _, rep = _solve(A, rng.standard_normal(n))
    assert st == g.IBEM_ERR_SINGULAR and 0 < rep.info <= n
    if n <= 1000:
        assert _solve(A, rng.standard_normal(n), noalloc=True)[0] == g.IBEM_ERR_SINGULAR


@pytest.mark.parametrize("n", [100, 700])
@pytest.mark.parametrize("cond", [1e13, 1e15])
def test_nearly_singular(n, cond):
    import ibemproject_gb300 as g
    rng = np.random.default_rng(n)
    u, v = (np.linalg.qr(rng.standard_normal((n, n)))[0] for _ in range(2))
    s = np.ones(n)
    s[-1] = 1 / cond
    A, b = (u * s) @ v, rng.standard_normal(n)
    st, x, rep = _solve(A, b)
    assert st == g.IBEM_OK and rep.backward_error <= n * 2.0 ** -53
    r = np.abs(b - A @ x).max() / (np.abs(A).sum(1).max() * np.abs(x).max() + np.abs(b).max())
    assert r <= n * 2.0 ** -53
