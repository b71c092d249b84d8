"""The pivot search key of the FP64 panels (pivot_key.cuh), on the host: the order of |a| over the
whole range, 14 bits of the mantissa over the range of exponents that each number of rows leaves room
for (a factor 1 + 2^-14 is told apart everywhere there), the smaller row at equal size, never 0,
infinities and NaN the greatest."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HG = os.path.join(ROOT, "tests", "hostgen")
SO = os.path.join(HG, "_build", "libhostpivot.so")
RANGES = {7: (-1022, 1023), 8: (-896, 126), 9: (-384, 126), 10: (-128, 126)}


@pytest.fixture(scope="module")
def lib():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "ibemproject_gb300", "csrc"),
                    "-o", SO, os.path.join(HG, "hostpivot.cpp")], check=True)
    f = ctypes.CDLL(SO).hp_key64
    f.restype, f.argtypes = ctypes.c_uint, [ctypes.c_int, ctypes.c_uint, ctypes.c_int]
    return f


@pytest.fixture(params=sorted(RANGES))
def key(lib, request):
    f = lambda v, q=0: lib(request.param, int(np.float64(v).view(np.uint64)) >> 32, q)
    f.bits, f.rows, f.range = request.param, 1 << request.param, RANGES[request.param]
    return f


def test_order_over_the_whole_range(key):
    v = np.concatenate([[0.0], 2.0 ** np.linspace(-1074, 1023.999, 20001), [np.inf]])
    k = [key(x) for x in v]
    assert all(a <= b for a, b in zip(k, k[1:]))
    assert key(0.0, key.rows - 1) > 0
    assert key(np.nan) == k[-1] == key(-np.inf)
    assert [key(-x) for x in v[::100]] == [key(x) for x in v[::100]]


def test_resolution(key):
    for e in range(key.range[0], key.range[1] + 1):
        for m in (0, 1, 2 ** 13, 2 ** 14 - 1):
            a = np.ldexp(1 + m * 2.0 ** -14, e)
            with np.errstate(over="ignore"):
                b = np.ldexp(1 + (m + 1) * 2.0 ** -14, e)
            assert key(a, 0) < key(b, key.rows - 1), (e, m)


def test_smaller_row_at_equal_size(key):
    for v in (0.0, 1e-300, 0.75, 1.0, 1e300, np.inf, np.nan):
        k = [key(v, q) for q in range(key.rows)]
        assert all(a > b for a, b in zip(k, k[1:]))
