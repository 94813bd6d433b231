"""Plans of many small independent structures (a batch): the places of the fronts and blocks, tens of
thousands of them freed and taken level by level, are found in logarithmic time."""
import time

import numpy as np

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W


def test_placing_half_a_million_fronts_is_quick():
    """1,500 copies of twelve grids, 549,000 supernodes of uneven size.  A search through the free
    places in order took 23 s here, the whole plan and its checks now 1.0; the bound lies between."""
    parts = []
    for nx in range(10, 22):
        A = M.permute_lower(M.weighted_grid_2d(nx, nx, seed=1), M.nested_dissection((nx, nx)))
        parts.append((A.n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data))
    n0 = sum(p[0] for p in parts)
    ptr, idx, val, at = [np.zeros(1, np.int64)], [], [], 0
    for n, p, i, v in parts:
        ptr.append(p[1:] + ptr[-1][-1])
        idx.append(i + at)
        val.append(v)
        at += n
    ptr, idx, val = np.concatenate(ptr), np.concatenate(idx), np.concatenate(val)
    copies = 1500
    k = np.arange(copies)[:, None]
    indptr = np.concatenate([np.zeros(1, np.int64), (ptr[1:] + k * ptr[-1]).ravel()])
    indices = (idx + k * n0).ravel()
    A = M.LowerCSC(copies * n0, indptr.astype(np.int32), indices.astype(np.int32), np.tile(val, copies))
    P = W.assemble_own(A, np.arange(A.n))
    t = time.perf_counter()
    swc.plan_stats(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    assert time.perf_counter() - t < 12.0
