"""The FP64 trailing update on the tensor cores by itself (ibem_gemm_sub_f64): ragged sizes, one and
several accumulation chunks, several calls' worth of columns (k beyond 2,048 and 4,096), rows and
columns of very different size, entries far below their row's largest, and digits all of one sign
and near the largest, where the accumulators' sums are greatest; entry by entry against products
summed in extended precision.

Bound per entry (gemm_tc64.cu): 4.1 k 2^-53 max|a_i.| max|b_.j| for the digits and products left
out, and two roundings of the result (the sum, and the subtraction from C) in each call of 2,048
columns.  The reference's own rounding is below k 2^-63 of the sum of |a||b|.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _update(A, B, C):
    import torch

    import ibemproject_gb300 as g
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v.T)).cuda()   # column-major
    (m, k), n = A.shape, B.shape[1]
    a, b, c = dev(A), dev(B), dev(C)
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    g.check(g.lib().ibem_gemm_sub_f64(m, n, k, P(a), m, P(b), k, P(c), m, None))
    return c.cpu().numpy().T


def _check(A, B, C, rng, count=300):
    (m, k), n = A.shape, B.shape[1]
    got = _update(A, B, C)
    ij = np.stack([rng.integers(0, m, count), rng.integers(0, n, count)], 1)
    ij[:4] = [[0, 0], [m - 1, 0], [0, n - 1], [m - 1, n - 1]]
    ma, mb = np.abs(A).max(1), np.abs(B).max(0)
    for i, j in ij:
        want = np.longdouble(C[i, j]) - (A[i].astype(np.longdouble) * B[:, j].astype(np.longdouble)).sum()
        size = np.abs(A[i] * B[:, j]).sum()
        calls = -(-k // 2048)
        bound = 4.1 * k * 2.0 ** -53 * ma[i] * mb[j] + calls * 2.0 ** -53 * (abs(float(want)) + 2 * size + abs(C[i, j]))
        err = abs(float(want - np.longdouble(got[i, j])))
        assert err <= bound, (i, j, err, bound)


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 37, 45), (127, 63, 31), (128, 64, 32), (129, 65, 33), (128, 64, 256),
                                   (130, 70, 257), (257, 129, 192), (64, 200, 193), (300, 90, 2048), (70, 300, 2049),
                                   (150, 130, 4100), (40, 33, 6200)])
def test_sizes(m, n, k):
    rng = np.random.default_rng(m + n + k)
    _check(rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n)), rng)


@pytest.mark.parametrize("k", [70, 2100])
def test_scales(k):
    """Rows of A and columns of B between 1e-140 and 1e140, entries 1e-20 to 1 of their row's or column's largest."""
    rng = np.random.default_rng(k)
    m, n = 140, 100
    A = rng.standard_normal((m, k)) * 10.0 ** rng.uniform(-20, 0, (m, k)) * 10.0 ** rng.uniform(-140, 140, (m, 1))
    B = rng.standard_normal((k, n)) * 10.0 ** rng.uniform(-20, 0, (k, n)) * 10.0 ** rng.uniform(-140, 140, (1, n))
    A[5], B[:, 7] = 0.0, 0.0
    _check(A, B, np.zeros((m, n)), rng)


def _digits(rng, shape, lo, hi, sign):
    """Numbers in [2^54, 2^55) 2^-55 whose seven 8-bit digits all lie in lo .. hi (the last one a multiple of 4)."""
    f = np.zeros(shape, dtype=np.int64)
    for i in range(7):
        d = rng.integers(lo, hi + 1, shape)
        f = f * 256 + (d if i < 6 else d // 4 * 4)
    v = np.ldexp(f.astype(np.float64), -55)
    assert (v >= 0.5).all() and (v < 1).all() and (np.ldexp(v, 55).astype(np.int64) == f).all()
    return sign * v


@pytest.mark.parametrize("lo,hi", [(124, 127), (120, 127), (127, 127), (100, 127)])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("k", [192, 256, 1000, 2300])
def test_largest_sums(lo, hi, sign, k):
    rng = np.random.default_rng(k + lo)
    A, B = _digits(rng, (130, k), lo, hi, 1), _digits(rng, (k, 66), lo, hi, sign)
    _check(A, B, np.zeros((130, 66)), rng)


def test_smallest_maximum_with_dropped_products():
    """Rows and columns whose largest entry is just above a power of two and whose products left
    out are all of one sign: digits 65, then -128 six times (2.96 of the bound's 4.1)."""
    f = 65 * 2 ** 48 - 128 * sum(256 ** i for i in range(6))
    v = np.ldexp(np.float64(f), -55)
    assert int(np.ldexp(v, 55)) == f
    rng = np.random.default_rng(1)
    k = 512
    _check(np.full((130, k), v), np.full((k, 70), v), np.zeros((130, 70)), rng)


def test_non_finite_rows_and_columns():
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal((140, 50)), rng.standard_normal((50, 80))
    A[17, 3], B[20, 30] = np.nan, np.inf
    got = _update(A, B, np.zeros((140, 80)))
    bad = np.zeros(got.shape, dtype=bool)
    bad[17], bad[:, 30] = True, True
    assert np.isnan(got[bad]).all() and np.isfinite(got[~bad]).all()
