"""Several right-hand sides at a time (interleaved by eight, tensor-core products) against the
solve of each one alone, at counts around the groups of eight and on structures with warp, CTA
and chained supernodes of partial blocks.  Both are backward stable FP64 solves of the same
factor: they differ by rounding, bounded here by 1e-10 of max |x| for condition numbers up to
about 1e4 (2^-53 * 1e4 with three decimal digits to spare)."""
import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W

pytestmark = pytest.mark.gpu


def structures():
    yield "plate", M.weighted_grid_2d(61, 47, shift=0.1, seed=1), M.nested_dissection((61, 47)), 1 << 30
    yield "plate_wide", M.weighted_grid_2d(260, 251, shift=0.1, seed=2), M.nested_dissection((260, 251)), 1 << 30
    yield "brick", M.laplacian_3d(20, 1e-2), M.nested_dissection((20, 20, 20)), 1 << 30
    yield "brick_capped", M.laplacian_3d(15, 1e-2), M.nested_dissection((15, 15, 15)), 70
    A = M.stencil27_3dof(9, shift=0.5, seed=4)
    yield "elastic", A, M.nested_dissection((9, 9, 9), dof=3), 1 << 30
    yield "single", M.laplacian_2d(1), np.arange(1), 1 << 30


@pytest.mark.parametrize("case", list(structures()), ids=lambda c: c[0])
def test_matches_single_solves(cuda_ok, case):
    _, A, perm, max_width = case
    P = W.assemble_own(A, perm, max_width=max_width)
    h = swc.Handle(0)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    assert h.factor(P.A2x) == 0
    rng = np.random.default_rng(8)
    B = rng.standard_normal((P.n, 17))
    X1 = np.stack([h.solve(B[:, k]) for k in range(17)], axis=1)
    for nrhs in (2, 7, 8, 9, 17):
        X = h.solve(B[:, :nrhs])
        assert np.abs(X - X1[:, :nrhs]).max() <= 1e-10 * np.abs(X1).max(), nrhs
        Y = h.solve(B[:, :nrhs])
        assert np.array_equal(X, Y)
    X, berr, _, _ = h.refine(B[:, :9], tol=1e-14)
    assert berr.max() <= 1e-14
    assert np.abs(X - X1[:, :9]).max() <= 1e-10 * np.abs(X1).max()


def test_timeout_in_any_group_is_reported(cuda_ok):
    P = W.assemble_own(M.laplacian_3d(20, 1e-2), M.nested_dissection((20, 20, 20)))
    h = swc.Handle(0)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    assert h.factor(P.A2x) == 0
    B = np.random.default_rng(9).standard_normal((P.n, 16))
    X = h.solve(B)
    h.set_wait_budget(0)
    timeouts = 0
    for _ in range(3):
        try:
            h.solve(B)
        except swc.SWCError as e:
            assert e.code == swc.SWC_TIMEOUT, str(e)
            timeouts += 1
    assert timeouts > 0
    h.set_wait_budget(-1)
    assert np.abs(h.solve(B) - X).max() <= 1e-12 * np.abs(X).max()
