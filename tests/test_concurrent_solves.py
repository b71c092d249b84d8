"""Matrix-free solves from several host threads at once, each on a stream of its own: every thread's
Arnoldi steps report through a slot of pinned memory of their own, are launched ahead and chained,
and the buffers come from one pool.  More threads than slots: those without one go step by step.

Each solution against the same solve alone: both are refined to a residual of 1e-11, and the
systems' condition is below 100, so they agree to 1e-8 of the largest entry (as in the other
tests of these solves).
"""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(seed, num, layout):
    from ibemproject_gb300 import batch as B, cases
    bt = B.DeviceBatch([cases.farfield_case(num=n, r0=0.012, vf=0.12, grid=0, seed=100 * seed + n) for n in num],
                       layout=layout)
    return bt, B.farfield_rhs(bt, np.array([0.3, 0.1, 0.0, -0.2, 0.05, 1.0]))


def _solve(bt, b, stream):
    """B.solve on a stream given."""
    import torch

    import ibemproject_gb300 as g
    from ibemproject_gb300 import batch as B
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    reps = (g.MfReport * bt.nseg)()
    opt = g.MfOptions(8, 0, 0, 1e-11, 0.0, 0)   # restarts after 8 steps: several cycles a solve
    g.check(g.lib().ibem_e3d_mf_solve_layout(bt.ref(), bt.layout, b.data_ptr(), x.data_ptr(), B.PRECOND_BLOCK_JACOBI, None,
                                             ctypes.byref(opt), reps, ctypes.c_void_p(stream.cuda_stream)))
    stream.synchronize()
    assert all(r.rel_residual <= 1e-11 for r in reps)
    return x.cpu().numpy()


@pytest.mark.parametrize("layout", [24, 60])
@pytest.mark.parametrize("threads,repeats", [(2, 6), (8, 4), (80, 1)])
def test_threads(layout, threads, repeats):
    import torch
    sets = [_problem(k, [(1, 9, 30), (40,), (3, 17)][k % 3], layout) for k in range(4)]
    main = torch.cuda.Stream()
    want = [_solve(bt, b, main) for bt, b in sets]
    start, errors = threading.Barrier(threads), []

    def work(t):
        try:
            stream = torch.cuda.Stream()
            start.wait(60)
            for r in range(repeats):
                k = (t + r) % len(sets)
                x = _solve(*sets[k], stream)
                err = np.abs(x - want[k]).max() / np.abs(want[k]).max()
                assert err < 1e-8, (t, r, k, err)
        except BaseException as e:   # noqa: BLE001 - reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors[:3]
