"""Single right-hand side solves of structures made of small supernodes (one CTA each), at widths
around the solving warp's 32 rows and the class's limit of 64 columns, at the largest panel height
of the class (2048 rows), and without rows below.  Against a dense FP64 solve: both are backward
stable, so they differ by at most a small multiple of n * 2^-53 * cond(A) (n <= 2053,
cond <= 1e2 here: 2.3e-11 times max |x|; 1e-10 is allowed)."""
import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W

pytestmark = pytest.mark.gpu


def dense_spd(n, seed):
    """Full lower triangle, diagonally dominant by two."""
    rng = np.random.default_rng(seed)
    T = np.tril(rng.uniform(-1, 1, (n, n)), -1)
    off = np.abs(T).sum(0) + np.abs(T).sum(1)
    D = T + np.diag(2 * off + 1)
    counts = np.arange(n, 0, -1)
    indptr = np.concatenate([[0], np.cumsum(counts)])
    indices = np.concatenate([np.arange(j, n) for j in range(n)])
    return M.LowerCSC(n=n, indptr=indptr.astype(np.int32), indices=indices.astype(np.int32),
                      data=np.concatenate([D[j:, j] for j in range(n)]))


def solve_both(A, perm, max_width):
    P = W.assemble_own(A, perm, max_width=max_width)
    h = swc.Handle(0)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    assert h.factor(P.A2x) == 0
    D = np.zeros((P.n, P.n))
    cols = np.repeat(np.arange(P.n), np.diff(P.A2p))
    D[P.A2i, cols] = P.A2x
    D[cols, P.A2i] = P.A2x
    b = np.random.default_rng(5).standard_normal(P.n)
    ref = np.linalg.solve(D, b)
    for _ in range(3):   # launched one by one, then as a graph
        assert np.abs(h.solve(b) - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("max_width", [1, 31, 32, 33, 63, 64])
def test_widths(cuda_ok, max_width):
    solve_both(M.laplacian_3d(11, 0.5), M.nested_dissection((11, 11, 11)), max_width)


@pytest.mark.parametrize("n,max_width", [(1, 1), (33, 33), (64, 64), (65, 64), (190, 64), (2053, 5)])
def test_dense(cuda_ok, n, max_width):
    solve_both(dense_spd(n, n), np.arange(n), max_width)


@pytest.mark.parametrize("nrhs", [1, 2, 4, 5, 8, 9])
@pytest.mark.parametrize("dense", [False, True])
def test_residuals(cuda_ok, dense, nrhs):
    """The backward errors that a refinement reports (its residuals take one, four or eight vectors
    per pass, rows of 4 to 190 entries, a row count that no block divides) against the same norms in
    numpy: each residual entry is a sum of at most n + 1 terms, so both are within (n + 2) 2^-53 of
    the exact value, relative to max |A| row sum times max |x|."""
    A, perm = (dense_spd(190, 3), np.arange(190)) if dense else (M.laplacian_2d(29), M.nested_dissection((29, 29)))
    P = W.assemble_own(A, perm)
    h = swc.Handle(0)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    assert h.factor(P.A2x) == 0
    D = np.zeros((P.n, P.n))
    cols = np.repeat(np.arange(P.n), np.diff(P.A2p))
    D[P.A2i, cols] = P.A2x
    D[cols, P.A2i] = P.A2x
    B = np.random.default_rng(7).standard_normal((P.n, nrhs))
    X, berr, _, _ = h.refine(B if nrhs > 1 else B[:, 0], tol=1e-14)
    X = np.asarray(X).reshape(P.n, -1)
    want = np.abs(B - D @ X).max(0) / (np.abs(D).sum(1).max() * np.abs(X).max(0))
    assert np.abs(np.asarray(berr) - want).max() <= 2 * (P.n + 2) * 2.0 ** -53
