"""Memory of the host-buffer pipelines goes back to the library's pool as unused: what the pool
reports as kept after them is what trimming gives back, call after call."""
import pytest

pytestmark = pytest.mark.gpu


def _run(which):
    import ibemproject_gb300 as g
    from ibemproject_gb300 import cases
    if which == "cube":
        g.run_host(cases.bounded_cube_case(n_face=8, num=8, grid=4), layout=24, form=g.SOLVE_FP64)
    elif which == "farfield":
        g.run_host(cases.farfield_case(num=60, r0=0.012, vf=0.1, grid=6, seed=2), layout=24, form=g.SOLVE_MIXED_IR)
    else:
        g.run_host_mf(cases.farfield_case(num=60, r0=0.012, vf=0.1, grid=6, seed=2), g.PRECOND_NEUMANN)


@pytest.mark.parametrize("which", ["cube", "farfield", "mf"])
def test_kept_after_host_pipelines(which):
    import torch

    import ibemproject_gb300 as g
    _run(which)   # what the first call loads stays out of it
    for _ in range(3):
        g.memory_trim()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        _run(which)
        torch.cuda.synchronize()
        kept = g.memory_kept()
        held = before - torch.cuda.mem_get_info()[0]
        assert held - (32 << 20) <= kept <= held + (32 << 20) and held > 0, (held, kept)   # a block of the driver's
