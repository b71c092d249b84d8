"""Device memory that the library keeps between calls: bounded, reported, and given back on
request, so that an allocator beside it can have it."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
GIB = 1 << 30


def _solve(n):
    import torch

    import ibemproject_gb300 as g
    A = torch.randn(n, n, dtype=torch.float64, device="cuda") + 2 * n ** 0.5 * torch.eye(n, dtype=torch.float64, device="cuda")
    b = torch.randn(n, dtype=torch.float64, device="cuda")
    x = torch.empty_like(b)
    rep = g.SolveReport()
    g.check(g.lib().ibem_e3d_solve(g.SOLVE_FP64, n, A.data_ptr(), n, b.data_ptr(), x.data_ptr(), 1e-12, ctypes.byref(rep),
                                   None))


@pytest.mark.parametrize("n", [300, 4000, 16000])   # the last one's matrix alone is 2 GiB
def test_kept_memory_is_bounded_and_goes_back(n):
    import torch

    import ibemproject_gb300 as g
    _solve(n)
    torch.cuda.synchronize()
    kept = g.memory_kept()
    assert 0 < kept <= GIB + (64 << 20)   # whole blocks of the driver's, at most two of 32 MiB more
    free = torch.cuda.mem_get_info()[0]
    g.memory_trim()
    assert g.memory_kept() == 0
    assert torch.cuda.mem_get_info()[0] - free >= kept // 2
    _solve(300)   # and the pool goes on
