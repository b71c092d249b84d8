"""Launch shapes whose source slices are cut into pieces: the reported choice, and the products in
every tile shape and piece count against the assembled matrix, on a ragged batch (realisations of
1, 40 and 130 spheres: pieces without a source, and of one).

Tolerances as for the other products: FP64 and double-float 1e-12, FP32 2e-5, in the scaled norm.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cases(nums):
    from ibemproject_gb300 import cases
    return [cases.farfield_case(num=n, r0=0.012, vf=0.15, grid=0, seed=50 + k, E1=70e9 * (3 + 4 * k))
            for k, n in enumerate(nums)]


@pytest.mark.parametrize("shape", ["0,0,1,2", "0,0,3,4", "1,0,1,3", "1,0,5,4", "2,0,1,4", "2,0,2,2", "1,1,3,1"])
def test_products(shape, monkeypatch):
    import torch

    from ibemproject_gb300 import batch as B
    monkeypatch.setenv("IBEM_MF_F32_SHAPE", shape)
    cs = _cases([1, 40, 130])
    bt = B.DeviceBatch(cs)
    ts, pers, slices, pc = (int(v) for v in shape.split(","))
    assert B.tile_shape(bt) == (64 << ts, pers, min(slices, 5))
    f, w = B.pieces(bt)
    assert f == pc and 2 <= w <= 4   # three tiles, five slices: pieces until four CTAs per SM
    rng = np.random.default_rng(8)
    dr, dc = bt.scalings()
    x = torch.from_numpy(rng.standard_normal(bt.N) * dc).cuda()
    ys = {p: B.matvec(bt, x, p).cpu().numpy() for p in (32, 48, 64, 65)}
    for s, c in enumerate(cs):
        rows = bt.seg_rows(s)
        ref = dr[rows] * (B.dense_system(c).cpu().numpy().T @ x.cpu().numpy()[rows])
        for p, y in ys.items():
            err = np.linalg.norm(dr[rows] * y[rows] - ref) / np.linalg.norm(ref)
            assert err < (2e-5 if p == 32 else 1e-12), (p, s, err)


@pytest.mark.parametrize("shape", ["1,0,1,5", "1,0,1,0", "1,1,1,2", "1,0", "3,0,1,1"])
def test_refused(shape, monkeypatch):
    import ibemproject_gb300 as g
    from ibemproject_gb300 import batch as B
    monkeypatch.setenv("IBEM_MF_F32_SHAPE", shape)
    with pytest.raises(g.IbemError) as e:
        B.pieces(B.DeviceBatch(_cases([5])))
    assert e.value.status == g.IBEM_ERR_ARG


def test_reported_choice():
    from ibemproject_gb300 import batch as B
    bt = B.DeviceBatch(_cases([64]))
    got = B.pieces(bt)
    assert all(1 <= v <= 4 for v in got) and B.pieces(bt) == got
    if B.tile_shape(bt)[1]:
        assert got[0] == 1
