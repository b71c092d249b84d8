"""Sixteen nearest neighbours of microstructures whose coordinates lie at the ends of the FP32
range (the kernel's first pass bounds the distance in FP32, where the squares of lengths below
1e-19 lose their digits and those above 1e19 overflow), against a sort of the FP64 distances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-16, 1e-19, 1e-20, 1e-21, 1e-22, 1e-24, 1e17, 1e20])
@pytest.mark.parametrize("num", [17, 40, 300])
def test_neighbours(scale, num):
    from ibemproject_gb300 import batch as B, cases
    c = cases.farfield_case(num=num, r0=0.012, vf=0.12, grid=0, seed=num)
    rng = np.random.default_rng(num)
    c.centers = scale * rng.uniform(0, 1, (num, 3))
    c.radius = scale * np.full(num, 0.01)
    bt = B.DeviceBatch([c])
    got = B.prepare(bt)["nbr"].cpu().numpy().reshape(num, 16)
    u = c.centers / scale   # (distances in the order of the scaled ones, no underflow)
    d2 = ((u[:, None] - u[None]) ** 2).sum(-1)
    np.fill_diagonal(d2, np.inf)
    for p in range(num):
        want = np.lexsort((np.arange(num), d2[p]))[:16]
        assert set(got[p]) == set(want), (p, got[p], want)
