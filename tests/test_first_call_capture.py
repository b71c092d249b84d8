"""Stress sums captured into a CUDA graph, replayed on changed inputs, against the same call without a
graph; in a process of its own, so that the library's first device work is the captured call
(what it sets up on first use may not disturb the capture)."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes
import sys
import numpy as np
import torch
import ibemproject_gb300 as g
from ibemproject_gb300 import cases

form, nump = (int(v) for v in sys.argv[1:])
c = cases.farfield_case(num=200, r0=0.012, vf=0.1, grid=0, seed=3)
rng = np.random.default_rng(2)
dev = lambda v: torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64)).cuda()
cen, rad, E = dev(c.centers), dev(c.radius), dev(rng.standard_normal(24 * c.num) * 1e-3)
pts, out = dev(rng.uniform(0, 1, (nump, 3)) * c.centers.max()), torch.zeros(nump, 6, dtype=torch.float64, device="cuda")
sig = np.ascontiguousarray(c.sig_inf).ctypes.data_as(ctypes.POINTER(ctypes.c_double))
m = g.material(c.E0, c.nu0, c.E1, c.nu1)
st = torch.cuda.Stream()


def call():
    g.check(g.lib().ibem_e3d_field_form(form, pts.data_ptr(), nump, cen.data_ptr(), rad.data_ptr(), c.num,
                                        ctypes.byref(m), 24, E.data_ptr(), None, 0, None, 0, None, None, sig,
                                        out.data_ptr(), ctypes.c_void_p(st.cuda_stream)))


torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=st):
    call()
last = None
for k in range(3):
    E.mul_(1.5)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    got = out.clone()
    torch.cuda.synchronize()
    call()
    torch.cuda.synchronize()
    assert torch.equal(got, out), (got - out).abs().max()
    assert last is None or not torch.equal(got, last)
    last = got
print("captured")
"""


@pytest.mark.parametrize("form", [0, 1])   # FP64, mixed
@pytest.mark.parametrize("nump", [100, 5000])
def test_first_call_in_a_capture(form, nump):
    r = subprocess.run([sys.executable, "-c", CHILD, str(form), str(nump)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
