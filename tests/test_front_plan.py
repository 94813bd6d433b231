"""The multifrontal FP64 factorization: its plan (row maps of the children, walks, tiles,
placement of the contribution blocks) is checked by swc_plan_stats on the CPU, which raises on
the first violation; on the GPU its factor is compared with the oracle's at sizes around the
kernels' edges (1e-12 of max |L|: the bound the factor tests use)."""
import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W
from oracle import oracle as O


def grid(kind, dims, max_width):
    if kind == "plate":
        A, perm = M.weighted_grid_2d(*dims, seed=3), M.nested_dissection(dims)
    elif kind == "star":      # one wide supernode with many children: several batches of maps
        A = M.random_geometric(dims[0], dim=2, degree=6.0, seed=5)
        perm = swc.order_nd(A.n, A.indptr, A.indices)
    else:
        A, perm = M.stencil27_3dof(dims[0], shift=0.05, seed=2), M.nested_dissection(dims, dof=3)
    return W.assemble_own(A, perm, max_width=max_width)


def arrow(n, k):
    """n - k independent columns, each coupled to the last k: a root with n - k children."""
    import scipy.sparse as sp
    rng = np.random.default_rng(7)
    B = rng.uniform(-1.0, 1.0, (k, n - k))
    A = sp.bmat([[sp.identity(n - k) * (4.0 * k), None], [sp.csc_matrix(B), sp.identity(k) * (4.0 * n)]])
    return W.assemble_own(M.LowerCSC.from_scipy(sp.csc_matrix(A)), np.arange(n), nrelax=[0, 0, 0],
                          zrelax=[0.0, 0.0, 0.0])


CASES = [("plate", (7, 5), 1 << 30), ("plate", (23, 31), 1 << 30), ("plate", (64, 61), 9),
         ("plate", (90, 77), 1 << 30), ("star", (700,), 1 << 30), ("elastic", (6, 6, 6), 65),
         ("elastic", (8, 8, 8), 1 << 30), ("elastic", (9, 9, 9), 40), ("arrow", (400, 5), 0),
         ("arrow", (90, 70), 0)]


def problem(kind, dims, max_width):
    return arrow(*dims) if kind == "arrow" else grid(kind, dims, max_width)


@pytest.mark.parametrize("plan", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("kind,dims,max_width", CASES)
def test_plan_holds(kind, dims, max_width, plan):
    P = problem(kind, dims, max_width)
    st = swc.plan_stats(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet,
                        plan=plan)      # raises on a violation
    assert st["launches"] > 0


@pytest.mark.gpu
@pytest.mark.parametrize("plan", [0, 2, 3])
@pytest.mark.parametrize("kind,dims,max_width", CASES)
def test_factor_matches_oracle(cuda_ok, kind, dims, max_width, plan):
    P = problem(kind, dims, max_width)
    Lo, ok, _ = O.oracle_factor(P.n, P.A2p, P.A2i, P.A2x, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr,
                                P.pruneSet, P.levelPtr, P.parPtr, P.partition, P.xsize)
    assert ok == 1
    h = swc.Handle(0)
    h.set_plan(plan)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    assert h.factor(P.A2x) == 0
    L = h.get_L()
    assert np.abs(L - Lo).max() <= 1e-12 * np.abs(Lo).max()
    assert np.all(L[Lo == 0.0] == 0.0)
    assert h.factor(P.A2x) == 0
    assert np.array_equal(h.get_L(), L)


@pytest.mark.gpu
def test_incomplete_prune_sets_keep_left_looking(cuda_ok):
    """Prune sets that leave a descendant out are taken as they are (the update is not
    applied), as the oracle does."""
    P = grid("plate", (40, 37), 1 << 30)
    pp, ps = P.prunePtr.copy(), P.pruneSet.copy()
    last = P.super.size - 2
    keep = np.ones(ps.size, bool)
    keep[pp[last]] = False               # the root's first descendant
    pp[last + 1:] -= 1
    ps = np.ascontiguousarray(ps[keep])
    Lo, ok, _ = O.oracle_factor(P.n, P.A2p, P.A2i, P.A2x, P.lC, P.Ls, P.Li_ptr, P.super, pp, ps,
                                P.levelPtr, P.parPtr, P.partition, P.xsize)
    assert ok == 1
    h = swc.Handle(0)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, pp, ps)
    assert h.factor(P.A2x) == 0
    assert np.abs(h.get_L() - Lo).max() <= 1e-12 * np.abs(Lo).max()
