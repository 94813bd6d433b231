"""The work reported per kernel class of an FP64 factorization is the multifrontal kernels' own:
counted here from the supernodes' sizes."""
import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W


def plate(nx, ny):
    return W.assemble_own(M.weighted_grid_2d(nx, ny, seed=3), M.nested_dissection((nx, ny)))


def elastic(k):
    return W.assemble_own(M.stencil27_3dof(k, shift=0.05, seed=2), M.nested_dissection((k, k, k), dof=3))


def stats(P):
    return swc.plan_stats(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)


def sizes(P):
    w = np.diff(P.super).astype(float)
    m = (P.Li_ptr[P.super[1:]].astype(np.int64) - P.Li_ptr[P.super[:-1]].astype(np.int64)).astype(float)
    return w, m - w


@pytest.mark.parametrize("P", [plate(20, 20), plate(64, 61), elastic(6), elastic(9)],
                         ids=["plate_20", "plate_64", "elastic_6", "elastic_9"])
def test_products_are_counted_once(P):
    """Small fronts factored whole, and every front's contribution block."""
    w, r = sizes(P)
    small = (w <= 64) & (w + r <= 1024) & (w * (w + r) <= 4096)
    st = stats(P)
    assert st["small"] + st["tiled"] <= w.size and st["tiled"] == int((~small).sum())
    want = (w ** 3 / 3 + r * w * w)[small].sum() + (r * (r + 1) * w).sum()
    got = st["flops"]["small"] + st["flops"]["update"]
    assert got == pytest.approx(want, rel=1e-12)


def test_bytes_of_small_fronts():
    """All fronts small: L and the blocks written, A, the children's blocks and row maps read."""
    P = plate(20, 20)
    w, r = sizes(P)
    st = stats(P)
    assert st["tiled"] == 0
    blocks = (r * (r + 1) / 2).sum()
    want = 8 * ((w + r) * w).sum() + 12.0 * P.A2i.size + 2 * 8 * blocks + 4 * r.sum()
    assert st["flops"]["update"] == 0.0 and st["bytes"]["update"] == 0.0
    assert st["bytes"]["small"] == pytest.approx(want, rel=1e-12)


@pytest.mark.gpu
def test_profile_times_the_extend_add_with_the_updates(cuda_ok):
    P = elastic(9)
    h = swc.Handle(0)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    prof = h.profile(P.A2x)
    st = stats(P)
    assert prof["assemble"][0] == 1
    assert prof["update"][0] > 1
    for k in ("small", "assemble", "update", "panel", "syrk"):
        assert prof[k][2] == st["flops"][k] and prof[k][3] == st["bytes"][k]
    # the mixed modes' updates keep their own count
    mixed = h.profile(P.A2x, mode=swc.SWC_MODE_MIXED_TF32X3)
    assert mixed["update"][2] > 0 and mixed["small"][2] > 0
