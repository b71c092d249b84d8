"""An ellipsoid's own block (target at the source's centre, with the self term C0): the short route
and its self term against the general route, on the host; and the own blocks of assembled
matrices, where one batch holds both routes, against the host's general one.

Tolerances as for the pairs of different particles: 1e-12 of a row and column order's largest
entry on the host (two routes of about 100 roundings each), 1e-11 on the device.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HG = os.path.join(ROOT, "tests", "hostgen")
SO = os.path.join(HG, "_build", "libhostellself.so")
D = ctypes.c_double
# the last two are too flat for the short route
SHAPES = [(1, 1, 1), (1, 1, 0.3), (1, 0.3, 0.3), (1, 0.7, 0.4), (0.3, 1, 0.6), (0.5, 0.21, 1), (1, 0.7, 0.19), (1, 0.9, 0.02)]


def p(a):
    return a.ctypes.data_as(ctypes.POINTER(D))


@pytest.fixture(scope="module")
def he():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "ibemproject_gb300", "csrc"),
                    "-o", SO, os.path.join(HG, "hostellself.cpp")], check=True)
    return ctypes.CDLL(SO)


def _quat(rng):
    q = rng.standard_normal(4)
    return q / np.linalg.norm(q)


def _close(got, want, tol):
    for rows in (slice(0, 6), slice(6, 24)):
        for cols in (slice(0, 6), slice(6, 24)):
            scale = np.abs(want[rows, cols]).max()
            if scale == 0.0:   # orders of different parity do not couple at the centre
                scale = np.abs(want).max() * 1e-2
            if np.abs(got[rows, cols] - want[rows, cols]).max() > tol * scale:
                return False
    return True


def _general(he, quat, axes, nu0=0.3):
    g, e = np.zeros(576), np.zeros(576)
    short = he.he_self24(p(np.ascontiguousarray(quat)), p(np.ascontiguousarray(axes)), D(nu0), p(g), p(e))
    return g.reshape(24, 24), e.reshape(24, 24), short


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("nu0", [0.0, 0.3, 0.49])
def test_routes_agree(he, shape, nu0):
    rng = np.random.default_rng(3)
    for t in range(8):
        g, e, short = _general(he, _quat(rng) if t else np.array([1.0, 0, 0, 0]), 0.01 * np.array(shape, dtype=float), nu0)
        assert short == (min(shape) >= 0.2)
        if short:
            assert _close(e, g, 1e-12), t


@pytest.mark.gpu
@pytest.mark.parametrize("num", [1, 8, 33, 130])
def test_assembled_own_blocks(he, num):
    import torch

    import ibemproject_gb300 as g
    rng = np.random.default_rng(num)
    cen = rng.uniform(0, 0.05 * num ** (1 / 3), (num, 3))
    axes = 0.01 * np.array([SHAPES[k % len(SHAPES)] for k in range(num)], dtype=float)
    quats = np.array([_quat(rng) for _ in range(num)])
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    c, a, q = dev(cen), dev(axes), dev(quats)
    n = 24 * num
    A = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    m = g.material(70e9, 0.3, 400e9, 0.2)
    g.check(g.lib().ibem_e3d_ell_pair_blocks(c.data_ptr(), a.data_ptr(), q.data_ptr(), num, ctypes.byref(m), A.data_ptr(),
                                             n, 0, 0, None))
    got = A.cpu().numpy().T
    for s in range(num):
        want, _, _ = _general(he, quats[s], axes[s])
        own = got[24 * s:24 * s + 24, 24 * s:24 * s + 24]
        assert _close(own, want, 1e-11), (s, SHAPES[s % len(SHAPES)], np.abs(own - want).max() / np.abs(want).max())
