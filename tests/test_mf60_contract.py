"""The layout-60 pair product in the frame of the offset (mf60_contract.cuh, gen_mf60.cuh)
against the generated dense block, on the host: offsets from contact to far, along the axes and
in every octant (the frame has a sign change at n_z = 0 and no square root), several Poisson
ratios, radii of different size.  And on the GPU the batched products against the assembled
matrix, where target tiles and source slices are ragged and where spheres overlap.

Tolerances per row order, relative to its largest entry: FP64 2e-13 (the dense block itself is
off by up to 4e-14 of it), FP32 2e-5 (as for layout 24: about 2,000 operations with rounding
6e-8, of random sign, on entries up to 6 times the result).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HG = os.path.join(ROOT, "tests", "hostgen")
SO = os.path.join(HG, "_build", "libhostmf60.so")
ORDERS = ((0, 6), (6, 24), (24, 60))


@pytest.fixture(scope="module")
def hg():
    from ibemproject_gb300 import codegen
    codegen.generate()
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.run(["g++", "-O0", "-shared", "-fPIC", "-I", os.path.join(ROOT, "ibemproject_gb300", "csrc"), "-o", SO,
                    os.path.join(HG, "hostmf60.cpp")], check=True)
    return ctypes.CDLL(SO)


@pytest.mark.parametrize("nu0", [0.0, 0.3, 0.49])
def test_contraction_against_dense_block(hg, nu0):
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    d = ctypes.c_double
    rng = np.random.default_rng(17)
    axes = [s * np.eye(3)[i] for i in range(3) for s in (1.0, -1.0)] + [np.array([1.0, -1.0, 0.0]), np.array([0.0, 1.0, -1e-9])]
    for t in range(60):
        x = axes[t] if t < len(axes) else rng.standard_normal(3)
        ah, as_ = 0.01 * (0.5 + rng.random()), 0.01 * (0.5 + rng.random())
        x = np.ascontiguousarray(x / np.linalg.norm(x) * ah * (1.001 + 20 * rng.random() ** 3))
        e = rng.standard_normal(60)
        want, y64, y32 = np.zeros(60), np.zeros(60), np.zeros(60)
        hg.hg_mf60(p(x), d(as_), d(ah), d(70e9), d(nu0), d(400e9), d(0.2), p(e), p(want), p(y64), p(y32))
        for a, b in ORDERS:
            scale = np.abs(want[a:b]).max()
            assert np.abs(y64 - want)[a:b].max() <= 2e-13 * scale, (t, a)
            assert np.abs(y32 - want)[a:b].max() <= 2e-5 * scale, (t, a)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,overlap", [((1,), False), ((2, 1, 63), False), ((64, 65), False), ((129, 3), False),
                                           ((40, 7), True)])
def test_products_against_matrix(sizes, overlap):
    import torch

    from ibemproject_gb300 import batch as B, cases
    cs = [cases.generated_case(n, 0.01, 0.2, seed=n, E1=70e9 * (2 + k)) for k, n in enumerate(sizes)]
    rng = np.random.default_rng(2)
    if overlap:   # half the spheres swallow the centre of another one
        for c in cs:
            for i in range(0, c.num - 1, 2):
                c.centers[i] = c.centers[i + 1] + 0.4 * c.radius[i] * rng.uniform(-1, 1, 3)
    bt = B.DeviceBatch(cs, layout=60)
    dr, dc = bt.scalings()
    xs = rng.standard_normal(bt.N)
    x = torch.from_numpy(xs * dc).cuda()
    order = np.tile(np.repeat([0, 1, 2], [6, 18, 36]), bt.num)
    for precision, tol in ((64, 2e-13), (32, 2e-5)):
        y = B.matvec(bt, x, precision).cpu().numpy() * dr
        for s, c in enumerate(cs):
            rows = bt.seg_rows(s)
            A = B.dense_system(c, layout=60).cpu().numpy().T
            want = dr[rows] * (A @ (xs[rows] * dc[rows]))
            for o in range(3):
                sel = order[rows] == o
                scale = np.abs(dr[rows][:, None] * A * dc[rows])[sel].sum(axis=1).max()
                assert np.abs(y[rows] - want)[sel].max() <= tol * scale, (precision, s, o)


@pytest.mark.gpu
@pytest.mark.parametrize("nu0", [0.0, 0.3, 0.49])
def test_block_jacobi_inverts_the_own_block(nu0):
    """A realisation of one particle is its own block: the FP32 inverse leaves 1e-4 of a residual at
    most (rounding times the block's condition, about 100), so refinement to 1e-11 takes at most
    three GMRES calls of at most two steps."""
    import torch

    from ibemproject_gb300 import batch as B, cases
    cs = [cases.generated_case(1, 0.01, 0.2, seed=k, E1=70e9 * (0.2 + 4 * k), nu0=nu0) for k in range(5)]
    bt = B.DeviceBatch(cs, layout=60)
    dr, _ = bt.scalings()
    b = torch.from_numpy(np.random.default_rng(4).standard_normal(bt.N) / dr).cuda()
    _, reps = B.solve(bt, b, B.PRECOND_BLOCK_JACOBI, tol=1e-11)
    for r in reps:
        assert r.rel_residual <= 1e-11 and r.outer <= 3 and r.inner <= 6, (r.outer, r.inner)
