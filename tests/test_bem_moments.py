"""The boundary rows from moments of the derivatives of R (bem_moments.cuh) and the stress sums'
per-pair form (bem_contract.cuh) against the generated stress kernels, on the host; the
assembled boundary matrices against the oracle on the GPU, where particles fill a pair, a group
of eight and one more, and where elements share nodes and hold the collocation node.

Tolerances: host 1e-13 of the largest entry of an order (derivatives of order up to 6 are sums
of at most 15 products, each combination of at most 20: 300 roundings of 1e-16, the largest
terms a few times the result); GPU 1e-11 of the block's largest entry, as for the other blocks.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HG = os.path.join(ROOT, "tests", "hostgen")
D = ctypes.c_double


def p(a):
    return a.ctypes.data_as(ctypes.POINTER(D))


def _lib(src, opt):
    so = os.path.join(HG, "_build", "lib" + src.replace(".cpp", ".so"))
    os.makedirs(os.path.dirname(so), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", opt, "-shared", "-fPIC", "-I", os.path.join(ROOT, "ibemproject_gb300", "csrc"),
                    "-o", so, os.path.join(HG, src)], check=True)
    return ctypes.CDLL(so)


@pytest.fixture(scope="module")
def libs():
    from ibemproject_gb300 import codegen
    codegen.generate()
    return _lib("hostbem.cpp", "-O1"), _lib("hostgen.cpp", "-O0")


@pytest.mark.parametrize("nu0", [0.0, 0.3, 0.45])
def test_entries_against_generated(libs, nu0):
    hb, hg = libs
    mat = (70e9, nu0, 400e9, 0.2)
    mu = [mat[0] / 2 / (1 + nu0), mat[2] / 2.4]
    dlam = 2 * mu[0] * nu0 / (1 - 2 * nu0) - 2 * mu[1] * 0.2 / 0.6
    rng = np.random.default_rng(3)
    pairs = [0, 1, 2, 4, 5, 8]   # (w, z), w <= z, of the nine
    for t in range(40):
        x, nv = rng.standard_normal(3) * (0.05, 0.4, 1.5)[t % 3], rng.standard_normal(3)
        if t < 3:
            x = np.roll(np.array([0.3, 0.0, 0.0]), t)
        nv /= np.linalg.norm(nv)
        su, st = np.zeros((60, 3)), np.zeros((60, 3))
        hb.hb_entries(p(x), p(nv), *[D(v) for v in mat], p(su), p(st))
        for o, nw, sl in ((0, 1, slice(0, 6)), (1, 3, slice(6, 24)), (2, 9, slice(24, 60))):
            a, b = np.zeros((6, nw, 3)), np.zeros((6, nw, 3))
            hg.hg_bem_stress(o, p(x), p(nv), *[D(v) for v in mat], D(dlam), D(mu[0] - mu[1]), p(a), p(b))
            for got, want in ((su[sl], a), (st[sl], b)):
                want = (want[:, pairs] if o == 2 else want).reshape(-1, 3)
                assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max(), (t, o)


@pytest.mark.parametrize("nu0", [0.0, 0.3, 0.45])
def test_post_sum_against_pair(libs, nu0):
    hb, _ = libs
    rng = np.random.default_rng(4)
    for t in range(60):
        r = rng.standard_normal(13)
        r[6] = abs(r[6])
        pt = r[:3] + rng.standard_normal(3) * (0.02, 0.5, 3.0)[t % 3]
        a, b = np.zeros(6), np.zeros(6)
        hb.hb_post(p(pt), p(r), D(70e9), D(nu0), D(400e9), D(0.2), p(a), p(b))
        assert np.abs(a - b).max() <= 1e-13 * np.abs(a).max()


@pytest.mark.gpu
@pytest.mark.parametrize("num,layout", [(1, 24), (2, 60), (7, 78), (8, 24), (9, 60), (17, 78)])
def test_boundary_blocks(oracle_mod, num, layout):
    import torch

    import ibemproject_gb300 as g
    from ibemproject_gb300 import cases
    c = cases.bounded_cube_case(n_face=3, num=num, radius=0.04, grid=0, seed=num)
    H, G = (np.asarray(v) for v in oracle_mod.assemble(c, layout)[:2])
    N, n3 = 3 * c.NN + layout * num, 3 * c.NN
    m = g.material(c.E0, c.nu0, c.E1, c.nu1)
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, dtype=t)).cuda()
    nodes, conn, cen = dev(c.nodes, np.float64), dev(c.conn, np.int32), dev(c.centers, np.float64)
    Hd = torch.zeros((N, N), dtype=torch.float64, device="cuda")           # column-major
    Gd = torch.zeros((12 * c.NE, N), dtype=torch.float64, device="cuda")
    L = g.lib()
    g.check(L.ibem_e3d_bem_hg(nodes.data_ptr(), c.NN, conn.data_ptr(), c.NE, ctypes.byref(m), Hd.data_ptr(), N, 0, 0,
                              Gd.data_ptr(), N, 0, 0, None))
    g.check(L.ibem_e3d_bem_to_incl(nodes.data_ptr(), c.NN, conn.data_ptr(), c.NE, cen.data_ptr(), num, ctypes.byref(m),
                                   layout, Hd.data_ptr(), N, 0, Gd.data_ptr(), N, 0, n3, None))
    Hg, Gg = Hd.cpu().numpy().T, Gd.cpu().numpy().T
    for got, want, rows in ((Hg[:, :n3], H[:, :n3], slice(0, n3)), (Gg, G, slice(0, n3))):
        assert np.abs(got[rows] - want[rows]).max() <= 1e-11 * np.abs(want[rows]).max()
    order = np.repeat([0, 1, 2], [6, 18, layout - 24])
    for o in range(3 if layout > 24 else 2):
        rows = n3 + np.flatnonzero(np.tile(order, num) == o)
        for got, want in ((Hg[:, :n3], H[:, :n3]), (Gg, G)):
            assert np.abs(got[rows] - want[rows]).max() <= 1e-11 * np.abs(want[rows]).max(), o
