"""swc_solve_noalloc gives the same result as swc_solve, bit for bit, at every number of right-hand
sides it takes: counts around the groups of eight, and structures whose eight vectors and
contributions fit its scratch interleaved and others of which it takes four, two or one at a time."""
import ctypes

import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W

pytestmark = pytest.mark.gpu
SCRATCH = 1048576


def structures():
    yield "plate", M.weighted_grid_2d(61, 47, shift=0.1, seed=1), M.nested_dissection((61, 47)), 1 << 30
    yield "plate_wide", M.weighted_grid_2d(201, 189, shift=0.1, seed=2), M.nested_dissection((201, 189)), 1 << 30
    yield "plate_crowded", M.weighted_grid_2d(330, 301, shift=0.1, seed=2), M.nested_dissection((330, 301)), 1 << 30
    yield "plate_largest", M.weighted_grid_2d(410, 400, shift=0.1, seed=2), M.nested_dissection((410, 400)), 1 << 30
    yield "brick", M.laplacian_3d(20, 1e-2), M.nested_dissection((20, 20, 20)), 1 << 30
    yield "brick_large", M.laplacian_3d(31, 1e-2), M.nested_dissection((31, 31, 31)), 1 << 30
    yield "brick_capped", M.laplacian_3d(15, 1e-2), M.nested_dissection((15, 15, 15)), 70
    A = M.stencil27_3dof(9, shift=0.5, seed=4)
    yield "elastic", A, M.nested_dissection((9, 9, 9), dof=3), 1 << 30
    yield "single", M.laplacian_2d(1), np.arange(1), 1 << 30


@pytest.mark.parametrize("case", list(structures()), ids=lambda c: c[0])
def test_same_result_as_solve(cuda_ok, case):
    import torch
    _, A, perm, max_width = case
    P = W.assemble_own(A, perm, max_width=max_width)
    h = swc.Handle(0)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    assert h.factor(P.A2x) == 0
    rows = max(int(P.Li_ptr[-1]) - P.n, 1)
    b = torch.from_numpy(np.random.default_rng(8).standard_normal((17, P.n))).cuda()
    done = 0
    for nrhs in (1, 2, 3, 7, 8, 9, 17):
        if rows * nrhs > SCRATCH:
            continue
        done += 1
        x = torch.full((nrhs, P.n), float("nan"), dtype=torch.float64, device="cuda")
        y = torch.empty_like(x)
        torch.cuda.synchronize()
        for fn, out, tail in (("swc_solve_noalloc", x, ()), ("swc_solve", y, (1,))):
            rc = getattr(swc.lib(), fn)(h._h, ctypes.c_void_p(b.data_ptr()), ctypes.c_void_p(out.data_ptr()), nrhs, *tail)
            assert rc == swc.SWC_OK, swc.lib().swc_last_error().decode()
        torch.cuda.synchronize()
        assert torch.equal(x, y), nrhs
    assert done >= 2
