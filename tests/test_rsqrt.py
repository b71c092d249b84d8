"""The FP64 1/sqrt of the kernels bound by the FP64 pipe (fp64_math.cuh), on the device, over every
exponent of the normal numbers, against extended precision and CUDA's rsqrt; and what it gives
outside its range.

Bound: the iteration leaves 2^-58 of an estimate of 20 bits; the product x y under it is rounded
(2^-53), which enters by half, and the result too (2^-53): 1.54 2^-53 in all.  CUDA's own may
be off by one unit in the last place, 2 2^-53, so the two differ by 3.54 2^-53 at most.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
HG = os.path.join(ROOT, "tests", "hostgen")
SO = os.path.join(HG, "_build", "libdevrsqrt.so")


@pytest.fixture(scope="module")
def rsqrt():
    import torch

    from ibemproject_gb300 import build
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I",
                    os.path.join(ROOT, "ibemproject_gb300", "csrc"), "-o", SO, os.path.join(HG, "devrsqrt.cu")], check=True)
    f = ctypes.CDLL(SO).dr_rsqrt
    f.argtypes = [ctypes.c_int] + 3 * [ctypes.c_void_p]

    def call(x):
        t = torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).cuda()
        own, ref = torch.empty_like(t), torch.empty_like(t)
        torch.cuda.synchronize()
        assert f(t.numel(), t.data_ptr(), own.data_ptr(), ref.data_ptr()) == 0
        return own.cpu().numpy(), ref.cpu().numpy()
    return call


def test_every_exponent(rsqrt):
    rng = np.random.default_rng(1)
    m = np.concatenate([1 + rng.random(200), 1 + np.arange(4) * 2.0 ** -52, 2 - np.arange(1, 5) * 2.0 ** -52,
                        np.sqrt(2) + np.arange(-2, 3) * 2.0 ** -51])
    x = np.ldexp(m[None], np.arange(-1022, 1024)[:, None]).ravel()
    own, ref = rsqrt(x)
    # 1/sqrt on mantissas in [1, 4), where numpy's extended sqrt is exact to 2^-64
    f, e = np.frexp(x)
    odd = e % 2 != 0
    f, e = np.where(odd, 2 * f, 4 * f), np.where(odd, e - 1, e - 2)
    want = np.longdouble(1) / np.sqrt(f.astype(np.longdouble))
    scale = lambda v: np.ldexp(v, e // 2).astype(np.longdouble)
    err = np.abs(scale(own) - want) / want
    assert float(err.max()) <= 1.54 * 2.0 ** -53, (float(err.max()) * 2 ** 53, x[err.argmax()])
    assert np.abs(own / ref - 1).max() <= 3.54 * 2.0 ** -53 + 2.0 ** -52


def test_outside_the_range(rsqrt):
    own, _ = rsqrt([0.0, -0.0, 5e-324, 2.0 ** -1023, np.inf, -1.0, np.nan])
    assert not np.isfinite(own).any()
