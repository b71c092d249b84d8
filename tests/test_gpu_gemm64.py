"""The plain FP64 solve at the sizes where its kernels can go wrong: panels and triangular
solves with ragged last blocks (multiples of 32, 64 and 128 and their neighbours), updates
smaller than one 128 x 64 tensor-core tile, one and several 256-column accumulation chunks,
several 2,048-column calls, operands whose entries spread over many decades, and non-finite
entries.

Tolerances: the matrices are sqrt(N) (2 I + G / sqrt(N)), G standard normal, with condition
number below 10; an LU solve in FP64 has relative forward error at most about
cond N 2^-53, so 10 N 2^-53 is asked (and its scaled backward error N 2^-53).  With rows and
columns scaled by powers of ten the solve equilibrates, so the same bound holds for each
entry of the unscaled solution against the largest.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [31, 33, 64, 65, 95, 127, 129, 160, 191, 257, 320, 449, 513, 1025, 2050]


def _solve(A, b):
    import torch

    import ibemproject_gb300 as g
    n = len(b)
    At = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()   # column-major
    bt, x = torch.from_numpy(b).cuda(), torch.zeros(n, dtype=torch.float64, device="cuda")
    rep = g.SolveReport()
    g.check(g.lib().ibem_e3d_solve(g.SOLVE_FP64, n, At.data_ptr(), n, bt.data_ptr(), x.data_ptr(), 1e-12,
                                   ctypes.byref(rep), None))
    return x.cpu().numpy(), rep


def _matrix(n, seed):
    rng = np.random.default_rng(seed)
    A = 2 * np.sqrt(n) * np.eye(n)[rng.permutation(n)] + rng.standard_normal((n, n))
    return A, rng.standard_normal(n), rng


@pytest.mark.parametrize("n", SIZES)
def test_fp64_solve_sizes(n):
    A, b, _ = _matrix(n, n)
    x, rep = _solve(A, b)
    want = np.linalg.solve(A, b)
    want += np.linalg.solve(A, b - A @ want)
    assert np.abs(x - want).max() <= 10 * n * 2.0 ** -53 * np.abs(want).max()
    assert rep.backward_error <= n * 2.0 ** -53


@pytest.mark.parametrize("n", [97, 700])
def test_fp64_solve_scaled(n):
    A, b, rng = _matrix(n, n)
    r, c = 10.0 ** rng.uniform(-12, 12, n), 10.0 ** rng.uniform(-12, 12, n)
    x, rep = _solve(r[:, None] * A * c, r * b)
    want = np.linalg.solve(A, b)
    assert np.abs(x * c - want).max() <= 10 * n * 2.0 ** -53 * np.abs(want).max()
    assert rep.backward_error <= n * 2.0 ** -53


def test_fp64_solve_smooth_digits():
    """Entries whose leading digits are all alike and of one sign: the accumulators' largest sums."""
    n = 600
    A, b, _ = _matrix(n, 3)
    A = 1.0 - 1e-3 * np.abs(A) / np.abs(A).max() + 4.0 * n * np.eye(n)
    x, _ = _solve(A, b)
    want = np.linalg.solve(A, b)
    assert np.abs(x - want).max() <= 10 * n * 2.0 ** -53 * np.abs(want).max()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_fp64_solve_non_finite(bad):
    """A non-finite entry must not come out as a finite solution."""
    import ibemproject_gb300 as g
    n = 300
    A, b, _ = _matrix(n, 5)
    A[n - 3, n // 2] = bad
    try:
        x, _ = _solve(A, b)
    except g.IbemError:
        return
    assert not np.isfinite(x).all()
