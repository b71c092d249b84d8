"""Layout-60 FP64 products of pairs whose target centre lies on the source's surface to within a
few roundings: the pair is taken once, as a whole, and on the side that the rounded operations
r2 = (x0 x0 + x1 x1) + x2 x2, x = (c_s - c_h) (1 / a_h) put it, whichever of the product's kernels
looks at it.

The potentials' second derivatives jump at the surface, so each side's product is known from
the pair a relative 1e-10 farther out or in, which moves it by less than 1e-8 of itself (ten
powers of the distance at most); 1e-7 is asked, where the two sides differ by more than 1e-3.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ORDERS = ((0, 6), (6, 24), (24, 60))


def _cases(rng, num):
    from ibemproject_gb300 import cases
    cs = []
    for k in range(num):
        c = cases.farfield_case(num=2, r0=0.01, vf=0.01, grid=0, seed=1)
        d = rng.standard_normal(3)
        a = 0.01 * (0.5 + rng.random())
        c.radius = np.array([a, 0.05 * a])
        c.centers = np.stack([np.zeros(3), d / np.linalg.norm(d)])   # source, then the offset's direction
        c.centers[0] = 0.01 * rng.uniform(-1, 1, 3) if k % 2 else 0.0
        cs.append(c)
    return cs


def _placed(cs, factors):
    import copy
    out = []
    for c, f in zip(cs, factors):
        q = copy.copy(c)
        q.centers = np.stack([c.centers[0], c.centers[0] + c.radius[0] * f * c.centers[1]])
        out.append(q)
    return out


@pytest.mark.parametrize("order", [0, 1, 2])
def test_pair_on_the_surface_is_taken_once(order):
    import torch

    from ibemproject_gb300 import batch as B
    rng = np.random.default_rng(40 + order)
    base = _cases(rng, 400)
    ulps = rng.integers(-3, 4, len(base)) * 2.0 ** -52
    sets = [_placed(base, 1 + ulps), _placed(base, np.full(len(base), 1 + 1e-10)), _placed(base, np.full(len(base), 1 - 1e-10))]
    e = rng.standard_normal(60)
    y = []
    for cs in sets:
        bt = B.DeviceBatch(cs, layout=60)
        dr, dc = bt.scalings()
        x = np.zeros((len(cs), 2, 60))
        x[:, 0, slice(*ORDERS[order])] = e[slice(*ORDERS[order])]
        xt = torch.from_numpy(x.ravel() * dc).cuda()
        y.append((B.matvec(bt, xt, 64).cpu().numpy() * dr).reshape(len(cs), 2, 60)[:, 1])
    got, outer, inner = y
    sides = []
    told = 0
    for k, c in enumerate(sets[0]):
        p = (c.centers[1] - c.centers[0]) * (1.0 / c.radius[0])
        outside = (p[0] * p[0] + p[1] * p[1]) + p[2] * p[2] > 1.0
        sides.append(outside)
        want = outer[k] if outside else inner[k]
        other = inner[k] if outside else outer[k]
        for a, b in ORDERS:
            scale = np.abs(want[a:b]).max()
            if np.abs(want - other)[a:b].max() <= 1e-3 * scale:
                continue
            told += 1
            assert np.abs(got[k] - want)[a:b].max() <= 1e-7 * scale, (k, a, bool(outside), got[k][a:b], want[a:b], other[a:b])
    assert 100 < sum(sides) < 300 and told > 300
