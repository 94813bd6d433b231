"""Device memory of structures with a wide border: many narrow supernodes that all reach the same
last columns.  Every front's contribution block there is as large as the border squared, whatever
the front's width; the library's plan check bounds the blocks alive together by a multiple of L."""
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


@pytest.mark.parametrize("nb,w,k,leaf", [(5000, 1, 100, 0), (8000, 1, 250, 0), (600, 4, 300, 4)])
def test_contribution_blocks_are_bounded(nb, w, k, leaf):
    P = bordered(nb, w, k, leaf)
    assert swc.plan_stats(*arrays(P))["launches"] > 0      # raises on a violation


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
