"""FP64 stress sums with the spheres in slices: few points and many spheres, sizes at the edges of
the point blocks (128), the sphere chunks (32) and the slices, points inside and outside spheres,
against the sum of single-sphere calls (one slice), which the linearity of the sum allows.

Tolerance: both are sums of the same terms in FP64, each with a few hundred roundings of 1.1e-16
of its intermediate results (up to ten times the term): 1e-12 of the sum of absolute terms.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nump,num", [(1, 64), (127, 63), (129, 130), (257, 97), (3000, 200)])
def test_slices_add_up(nump, num):
    import torch

    import ibemproject_gb300 as g
    rng = np.random.default_rng(nump)
    # disjoint spheres, one to a cell of a 6 x 6 x 6 lattice
    cell = rng.permutation(216)[:num]
    cen = (np.stack([cell % 6, cell // 6 % 6, cell // 36], axis=1) + 0.5 + rng.uniform(-0.15, 0.15, (num, 3))) / 6
    rad = rng.uniform(0.01, 0.05, num)
    pts = rng.uniform(0.0, 1.0, (nump, 3))
    pts[::3] = cen[rng.integers(0, num, len(pts[::3]))] + 0.003 * rng.standard_normal((len(pts[::3]), 3))
    E = rng.standard_normal((num, 24))
    E[:, 6:] /= rad[:, None]
    m = g.Material(70e9, 0.3, 400e9, 0.2)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    dp = up(pts)
    sig = np.zeros(6)

    def field(sel):
        dc, dr, de = up(cen[sel]), up(rad[sel]), up(E[sel])
        s = torch.zeros(nump, 6, dtype=torch.float64, device="cuda")
        g.check(g.lib().ibem_e3d_field_form(g.SOLVE_FP64, P(dp), nump, P(dc), P(dr), len(sel), ctypes.byref(m), 24, P(de),
                                            None, 0, None, 0, None, None, sig.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                            P(s), None))
        return s.cpu().numpy()

    got = field(np.arange(num))
    terms = np.stack([field(np.array([h])) for h in range(num)])
    scale = np.abs(terms).sum(axis=0).max()
    assert np.abs(got - terms.sum(axis=0)).max() <= 1e-12 * scale
