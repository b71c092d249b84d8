"""The layout-24 pair contraction from a source's record (mf_contract.cuh), which the matrix-free
products evaluate: in double-float numbers against FP64 on the host (FP64 itself is compared with the
generated block elsewhere), inside the source, at its surface and far away; and on the GPU the products
against the assembled matrix where target tiles, source slices and their pieces are ragged (1 to
129 particles: slices of 32, pieces of 8) and where spheres overlap.

Tolerances, per row order: double-float on the host 64 units of 2^-44 (about 60 dependent operations of a
few such units) of the result's largest entry, times 10 where the terms cancel (entries of up to ten
times the result near the surface).  On the GPU relative to the largest row sum of absolute
products: FP64 2e-13 (the assembled blocks are off by up to 4e-14 of their largest entry), double-float
4e-12 (the host's bound), FP32 2e-5.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HG = os.path.join(ROOT, "tests", "hostgen")
SO = os.path.join(HG, "_build", "libhostmf24.so")


@pytest.fixture(scope="module")
def hm():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "ibemproject_gb300", "csrc"), "-o", SO, os.path.join(HG, "hostmf24.cpp")], check=True)
    return ctypes.CDLL(SO)


@pytest.mark.parametrize("lo,hi", [(0.0, 0.99), (1.0, 1.0 + 1e-6), (1.01, 2.5), (4.0, 60.0)])
@pytest.mark.parametrize("nu0", [0.0, 0.3, 0.49])
def test_double_float_against_fp64(hm, lo, hi, nu0):
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    d = ctypes.c_double
    rng = np.random.default_rng(3)
    f = 2.0 * float(np.float32(1.0 - nu0))
    for _ in range(50):
        x = rng.standard_normal(3)
        x *= (lo + (hi - lo) * rng.random()) / np.linalg.norm(x)
        x = np.float32(x).astype(float)   # exact in both types
        coef = rng.standard_normal(24)
        y64, ydf = np.zeros(24), np.zeros(24)
        hm.hm_raw24(0, p(x), d(f), p(coef), d(0.75), p(y64))
        hm.hm_raw24(1, p(x), d(f), p(coef), d(0.75), p(ydf))
        for sel in (slice(0, 6), slice(6, 24)):
            assert np.abs(ydf - y64)[sel].max() <= 640 * 2.0**-44 * np.abs(y64[sel]).max(), (x, sel)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,overlap", [((1,), False), ((8, 1, 9), False), ((31, 33), False), ((64, 65), False),
                                           ((129, 3), False), ((40, 7), True)])
def test_products_against_matrix(sizes, overlap):
    import torch

    from ibemproject_gb300 import batch as B, cases
    cs = [cases.generated_case(n, 0.01, 0.2, seed=n, E1=70e9 * (2 + k)) for k, n in enumerate(sizes)]
    rng = np.random.default_rng(2)
    if overlap:   # half the spheres swallow the centre of another one
        for c in cs:
            for i in range(0, c.num - 1, 2):
                c.centers[i] = c.centers[i + 1] + 0.4 * c.radius[i] * rng.uniform(-1, 1, 3)
    bt = B.DeviceBatch(cs)
    dr, dc = bt.scalings()
    xs = rng.standard_normal(bt.N)
    x = torch.from_numpy(xs * dc).cuda()
    order = np.tile(np.repeat([0, 1], [6, 18]), bt.num)
    for precision, tol in ((64, 2e-13), (48, 4e-12), (32, 2e-5)):
        y = B.matvec(bt, x, precision).cpu().numpy() * dr
        for s, c in enumerate(cs):
            rows = bt.seg_rows(s)
            A = B.dense_system(c).cpu().numpy().T
            want = dr[rows] * (A @ (xs[rows] * dc[rows]))
            for o in range(2):
                sel = order[rows] == o
                scale = np.abs(dr[rows][:, None] * A * dc[rows])[sel].sum(axis=1).max()
                assert np.abs(y[rows] - want)[sel].max() <= tol * scale, (precision, s, o)
