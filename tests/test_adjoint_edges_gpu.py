"""d log det A on structures around the sweep's edges (warp, CTA and wide fronts, partial
column blocks, forests, fronts whose two panels exceed shared memory) against the dense FP64
inverse.  Bound 1e-10 of max |gradient|: condition numbers up to about 1e4, so
2^-53 * 1e4 with two decimal digits to spare."""
import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W

pytestmark = pytest.mark.gpu


def structures():
    yield "tiny", M.weighted_grid_2d(7, 5, shift=0.1, seed=3), M.nested_dissection((7, 5)), 1 << 30, 0
    yield "plate", M.weighted_grid_2d(70, 61, shift=0.1, seed=1), M.nested_dissection((70, 61)), 1 << 30, 0
    yield "plate_capped", M.weighted_grid_2d(50, 45, shift=0.1, seed=2), M.nested_dissection((50, 45)), 9, 0
    yield "brick", M.laplacian_3d(16, 1e-2), M.nested_dissection((16, 16, 16)), 1 << 30, 0
    yield "brick_capped", M.laplacian_3d(15, 1e-2), M.nested_dissection((15, 15, 15)), 65, 0
    yield "brick_larger_small", M.laplacian_3d(16, 1e-2), M.nested_dissection((16, 16, 16)), 12, 3
    A = M.stencil27_3dof(8, shift=0.5, seed=4)
    yield "elastic", A, M.nested_dissection((8, 8, 8), dof=3), 1 << 30, 0
    B = M.stencil27_3dof(11, shift=0.5, seed=5)     # 2,000-row fronts of a few columns
    yield "elastic_narrow", B, M.nested_dissection((11, 11, 11), dof=3), 6, 3
    yield "crowded", M.random_geometric(4500, dim=2, degree=4.0, seed=6, shift=0.1), None, 1 << 30, 0


@pytest.mark.parametrize("case", list(structures()), ids=lambda c: c[0])
@pytest.mark.parametrize("mode", [swc.SWC_MODE_FP64, swc.SWC_MODE_MIXED_TF32X3])
def test_logdet_grad_matches_dense(cuda_ok, case, mode):
    _, A, perm, max_width, plan = case
    if perm is None:
        perm = swc.order_nd(A.n, A.indptr, A.indices)
    P = W.assemble_own(A, perm, max_width=max_width)
    h = swc.Handle(0)
    h.set_plan(plan)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    assert h.factor(P.A2x, mode) == 0
    import torch
    cols = np.repeat(np.arange(P.n), np.diff(P.A2p))
    D = torch.zeros(P.n, P.n, dtype=torch.float64, device="cuda")
    r, c = torch.from_numpy(P.A2i.astype(np.int64)).cuda(), torch.from_numpy(cols).cuda()
    D[r, c] = torch.from_numpy(P.A2x).cuda()
    D[c, r] = D[r, c]
    Z = torch.linalg.inv(D)
    ref = (Z[r, c] * ((r != c).double() + 1.0)).cpu().numpy()
    g = h.logdet_grad()
    bound = 1e-10 if mode == swc.SWC_MODE_FP64 else 1e-3
    assert np.abs(g - ref).max() <= bound * np.abs(ref).max()
    assert np.array_equal(h.logdet_grad(), g)
    assert h.logdet() == pytest.approx(float(torch.linalg.slogdet(D)[1]), rel=1e-10 if mode == 0 else 1e-4)
