"""The kernel launches per factorization that a handle reports are those that run: multifrontal and
left-looking FP64, before and after a mixed factorization with tile-owner updates."""
import ctypes

import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W

pytestmark = pytest.mark.gpu


def reported(h):
    sizes = (ctypes.c_longlong * 6)()
    assert swc.lib().swc_sizes(h._h, sizes) == swc.SWC_OK
    return int(sizes[3])


def counted(h, x):
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        assert h.factor(x) == 0
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    if not names:
        pytest.skip("no device events from the profiler")
    return sum(not n.startswith("Mem") for n in names)


@pytest.mark.parametrize("left", [False, True])
@pytest.mark.parametrize("plan", [0, 2, 4, 6])
def test_reported_launches_are_those_that_run(cuda_ok, plan, left):
    import torch
    P = W.assemble_own(M.stencil27_3dof(9, shift=0.5, seed=4), M.nested_dissection((9, 9, 9), dof=3))
    pp, ps = P.prunePtr.copy(), P.pruneSet.copy()
    if left:      # without its first descendant the root's prune set is not complete
        last = P.super.size - 2
        keep = np.ones(ps.size, bool)
        keep[pp[last]] = False
        pp[last + 1:] -= 1
        ps = np.ascontiguousarray(ps[keep])
    h = swc.Handle(0)
    h.set_plan(plan)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, pp, ps)
    x = torch.from_numpy(P.A2x).cuda()
    n = reported(h)
    for _ in range(3):        # directly, then as a graph
        assert counted(h, x) == n
    assert h.factor(x, mode=swc.SWC_MODE_MIXED_TF32X3) == 0
    assert reported(h) == n
    assert counted(h, x) == n
