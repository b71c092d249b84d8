"""The short route of the ellipsoid pair block (ellipsoid_ext.cuh: target outside the source)
against the general one, on the host: spheres, needles, discs and general shapes, offsets from
the centre to far away, along principal axes and planes (zero components of the
offset) and in general position, and the integrals at the borders of the quadrature's node
counts.  On the GPU: assembled blocks where warps are ragged, where a batch holds both routes
(flat close neighbours, a centre inside another particle) against the host's general route.

Tolerances: the general route's error, estimated in FP32, is 2 to 8e-6 (100 roundings), so in
FP64 1e-14 of a row order's largest entry on average and 1e-13 at contact, where it evaluates
differences of fourth derivatives; 1e-12 is asked.  Integrals: 1e-13 (Carlson's third
parameter derivatives lose a digit or two).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HG = os.path.join(ROOT, "tests", "hostgen")
SO = os.path.join(HG, "_build", "libhostellext.so")
D = ctypes.c_double


def p(a):
    return a.ctypes.data_as(ctypes.POINTER(D))


@pytest.fixture(scope="module")
def hx():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "ibemproject_gb300", "csrc"),
                    "-o", SO, os.path.join(HG, "hostellext.cpp")], check=True)
    return ctypes.CDLL(SO)


def _quat(rng):
    q = rng.standard_normal(4)
    return q / np.linalg.norm(q)


SHAPES = [(1, 1, 1), (1, 1, 0.3), (1, 0.3, 0.3), (1, 0.7, 0.4), (0.3, 1, 0.6), (1, 0.999999, 0.9999), (1, 0.5, 0.21)]


def _close(got, want, tol):
    for rows in (slice(0, 6), slice(6, 24)):
        for cols in (slice(0, 6), slice(6, 24)):
            if np.abs(got[rows, cols] - want[rows, cols]).max() > tol * np.abs(want[rows, cols]).max():
                return False
    return True


@pytest.mark.parametrize("shape", SHAPES)
def test_routes_agree(hx, shape):
    rng = np.random.default_rng(11)
    taken = 0
    for t in range(36):
        a = np.array(shape) * 0.01
        q = _quat(rng) if t % 3 else np.array([1.0, 0, 0, 0])
        d = rng.standard_normal(3)
        if t % 3 == 0:   # axes and planes of the principal frame
            d = np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 1, 0], [0, -1, 1], [1, 0, -1]][t // 3 % 6], dtype=float)
        d *= a.max() * (1.02, 1.2, 1.7, 3.0, 9.0, 60.0)[t % 6] / np.linalg.norm(d)
        if t > 30:   # inside and at the centre
            d = (0.2 if t < 35 else 0.0) * a.min() * rng.uniform(-1, 1, 3)
        g, e = np.zeros(576), np.zeros(576)
        if hx.hx_block24(p(d), p(q), p(a), D(0.3), p(g), p(e)):
            taken += 1
            assert _close(e.reshape(24, 24), g.reshape(24, 24), 1e-12), (shape, t)
    assert taken >= 30


def test_route_refused(hx):
    g, e, q = np.zeros(576), np.full(576, 7.0), np.array([1.0, 0, 0, 0])
    for a, d in (((1, 0.7, 0.19), (0.3, 0.1, 0.1)), ((1, 0.7, 0.1), (1.0, 0, 0)), ((1, 0.9, 0.01), (0, 0, 0.02)),
                 ((1, 0.8, 0.5), (np.nan, 0, 2.0))):
        assert not hx.hx_block24(p(np.array(d, dtype=float)), p(q), p(np.array(a, dtype=float)), D(0.3), p(g), p(e))
        assert (e == 7.0).all()


@pytest.mark.parametrize("kappa", [0.0, 0.01, 0.2, 0.2000001, 0.55, 0.5500001, 0.85, 0.8500001, 0.96])
def test_integrals(hx, kappa):
    rng = np.random.default_rng(5)
    for _ in range(10):
        X = rng.uniform(0.1, 30)
        x = np.array([X, X * (1 - kappa * rng.random()), X * (1 - kappa)])
        rng.shuffle(x)
        a, b = np.zeros(20), np.zeros(20)
        hx.hx_ik(p(x), D(kappa), p(a), p(b))
        assert np.abs(a / b - 1).max() <= 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("num", [1, 2, 31, 33, 65])
def test_assembled_blocks(hx, num):
    import torch

    import ibemproject_gb300 as g
    rng = np.random.default_rng(num)
    cen = rng.uniform(0, 0.05 * num ** (1 / 3), (num, 3))
    axes = 0.01 * np.stack([np.ones(num), rng.uniform(0.5, 1, num), rng.uniform(0.05, 1, num)], 1)
    quats = np.array([_quat(rng) for _ in range(num)])
    if num > 2:   # the last pair's own blocks go through the self term too
        cen[1] = cen[0] + 0.003   # inside one another
        axes[2, 2], cen[2] = 0.0001, cen[3 % num] + [0, 0, 0.0105]
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    c, a, q = dev(cen), dev(axes), dev(quats)
    n = 24 * num
    A = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    m = g.material(70e9, 0.3, 400e9, 0.2)
    g.check(g.lib().ibem_e3d_ell_pair_blocks(c.data_ptr(), a.data_ptr(), q.data_ptr(), num, ctypes.byref(m), A.data_ptr(),
                                             n, 0, 0, None))
    got = A.cpu().numpy().T
    pick = rng.integers(0, num, (40, 2)).tolist() + [[0, 1 % num], [1 % num, 0]]
    for s, h in pick:
        if s == h:
            continue
        want, e = np.zeros(576), np.zeros(576)
        hx.hx_block24(p(np.ascontiguousarray(cen[s] - cen[h])), p(quats[h]), p(axes[h]), D(0.3), p(want), p(e))
        assert _close(got[24 * s:24 * s + 24, 24 * h:24 * h + 24], want.reshape(24, 24), 1e-11), (s, h)
