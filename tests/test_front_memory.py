"""Device memory of structures with a wide border: many narrow supernodes that all reach the same
last columns.  Every front's contribution block there is as large as the border squared, whatever
the front's width, and so is its front in the gradient's reverse sweep; the library's plan check
bounds the blocks alive together by a multiple of L, and checks the sweep's order and places."""
import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W


def bordered(nb, w, k, leaf=0):
    """nb chains of w columns, each coupled to all of k border columns; `leaf` more columns hang
    below each chain (they reach its columns only)."""
    rng = np.random.default_rng(3)
    m = leaf + w
    n = nb * m + k
    o = np.arange(nb)[:, None] * m
    rows, cols = [], []

    def add(r, c):
        r, c = np.broadcast_arrays(r, c)
        rows.append(r.ravel())
        cols.append(c.ravel())

    for t in range(w):
        add(nb * m + np.arange(k)[None, :], o + leaf + t)
        for u in range(t):
            add(o + leaf + t, o + leaf + u)
        for u in range(leaf):
            add(o + leaf + t, o + u)
    import scipy.sparse as sp
    r, c = np.concatenate(rows), np.concatenate(cols)
    A = sp.coo_matrix((rng.uniform(-1.0, 1.0, r.size), (r, c)), shape=(n, n)).tocsc()
    d = np.asarray(abs(A).sum(0)).ravel() + np.asarray(abs(A).sum(1)).ravel() + 1.0
    return W.assemble_own(M.LowerCSC.from_scipy(sp.csc_matrix(A + sp.diags(d))), np.arange(n))


def arrays(P):
    return P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet


@pytest.mark.parametrize("nb,w,k,leaf", [(5000, 1, 100, 0), (8000, 1, 250, 0), (600, 4, 300, 4),
                                          (200, 80, 400, 4)])
def test_contribution_blocks_are_bounded(nb, w, k, leaf):
    P = bordered(nb, w, k, leaf)
    for plan in (0, 3):
        assert swc.plan_stats(*arrays(P), plan=plan)["launches"] > 0      # raises on a violation


@pytest.mark.gpu
def test_factor_of_a_bordered_matrix_stays_within_the_bound(cuda_ok):
    import torch
    P = bordered(8000, 1, 250)
    h = swc.Handle(0)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    h.analyze(*arrays(P))
    assert h.factor(P.A2x) == 0
    used = free - torch.cuda.mem_get_info()[0]
    assert used <= 4 * 8 * P.xsize + (256 << 20) + (256 << 20)     # L and blocks; tables
    b = np.random.default_rng(1).standard_normal(P.n)
    x = h.solve(b)
    import scipy.sparse as sp
    A = sp.csc_matrix((P.A2x, P.A2i, P.A2p), shape=(P.n, P.n))
    A = A + sp.tril(A, -1).T
    r = np.abs(A @ x - b).max() / (abs(A).sum(1).max() * np.abs(x).max())
    assert r <= 1e-14


@pytest.mark.gpu
@pytest.mark.parametrize("nb,w,k,leaf", [(600, 4, 300, 4), (200, 80, 400, 4)])
def test_gradient_in_groups_matches_dense(cuda_ok, nb, w, k, leaf):
    """The sweep's fronts are too many to be held together: groups, small or wide supernodes.  Bound
    as for the other structures (tests/test_adjoint_edges_gpu.py): 1e-10 of max |gradient|."""
    import torch
    P = bordered(nb, w, k, leaf)
    h = swc.Handle(0)
    h.analyze(*arrays(P))
    assert h.factor(P.A2x) == 0
    r = torch.from_numpy(P.A2i.astype(np.int64)).cuda()
    c = torch.from_numpy(np.repeat(np.arange(P.n), np.diff(P.A2p))).cuda()
    D = torch.zeros(P.n, P.n, dtype=torch.float64, device="cuda")
    D[r, c] = torch.from_numpy(P.A2x).cuda()
    D[c, r] = D[r, c]
    Z = torch.linalg.inv(D)
    ref = (Z[r, c] * ((r != c).double() + 1.0)).cpu().numpy()
    g = h.logdet_grad()
    assert np.abs(g - ref).max() <= 1e-10 * np.abs(ref).max()
    for _ in range(2):      # as a graph
        assert np.array_equal(h.logdet_grad(), g)


@pytest.mark.gpu
def test_gradient_of_a_bordered_matrix_stays_within_the_bound(cuda_ok):
    """2,000 fronts of 504 x 504 (4 GB) over an L of 33 MB."""
    import torch
    P = bordered(2000, 4, 500, 4)
    h = swc.Handle(0)
    h.analyze(*arrays(P))
    assert h.factor(P.A2x) == 0
    g = torch.empty(P.A2x.size, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    h.logdet_grad(out=g)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= (256 << 20) + (128 << 20)      # fronts; tables
    assert bool(torch.isfinite(g).all())
