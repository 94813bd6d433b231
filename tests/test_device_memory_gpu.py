"""What a handle does when device memory is short: the contribution blocks of the FP64 factorization
are the one thing it can do without, so they make room for whatever else a call needs (the mixed
modes' mirror, the solves' workspace, the gradient's fronts), as they would not be there at all
with the left-looking kernels."""
import numpy as np
import pytest

import swcholesky_b200 as swc
from swcholesky_b200 import matrices as M
from swcholesky_b200 import workloads as W

pytestmark = pytest.mark.gpu

MB = 1 << 20


def plate(nx, ny):
    return W.assemble_own(M.weighted_grid_2d(nx, ny, seed=3), M.nested_dissection((nx, ny)))


def analyzed(P):
    h = swc.Handle(0)
    h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
    return h


def free_bytes():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()     # torch's own idle memory is not the library's
    return torch.cuda.mem_get_info()[0]


def fill(leave):
    """Device memory taken until `leave` bytes are free."""
    import torch
    return torch.empty(free_bytes() - leave, dtype=torch.uint8, device="cuda")


@pytest.fixture(scope="module")
def problem():
    return plate(500, 500)     # L 121 MB, blocks 191 MB, mirror 396 MB


@pytest.mark.parametrize("op", ["mixed", "solve", "refine", "gradient"])
def test_blocks_make_room(cuda_ok, problem, op):
    import torch
    P = problem
    rng = np.random.default_rng(5)
    b = torch.from_numpy(rng.standard_normal((8, P.n))).cuda()
    x = torch.empty_like(b)
    values = torch.from_numpy(P.A2x).cuda()
    g = torch.empty(P.A2x.size, dtype=torch.float64, device="cuda")

    def call(h):
        if op == "mixed":
            return h.factor(values, mode=swc.SWC_MODE_MIXED_TF32X3)
        if op == "solve":
            return h.solve(b, out=x)
        if op == "refine":
            return h.refine(b, out=x)
        return h.logdet_grad(out=g)

    h = analyzed(P)
    assert h.factor(values) == 0
    assert h.factor(values) == 0           # its graph
    L = h.get_L()
    before = free_bytes()
    call(h)
    need = before - free_bytes()           # what the call takes (and keeps)
    want = [t.clone() for t in (x, g)]
    del h
    h = analyzed(P)
    assert h.factor(values) == 0
    assert h.factor(values) == 0
    x.zero_()
    g.zero_()
    taken = fill(need - min(need // 2, 60 * MB))
    try:
        call(h)                            # would fail beside the blocks
    finally:
        del taken
        torch.cuda.empty_cache()
    if op in ("solve", "refine"):
        assert torch.equal(x, want[0])
    if op == "gradient":
        assert torch.equal(g, want[1])
    # the next FP64 factorizations: left-looking, directly and as a graph
    for _ in range(3):
        assert h.factor(values) == 0
        assert np.abs(h.get_L() - L).max() <= 1e-12 * np.abs(L).max()


def test_mixed_handles_take_no_blocks(cuda_ok, problem):
    """An analysis takes L and tables; the blocks come with the first FP64 factorization."""
    P = problem
    before = free_bytes()
    h = analyzed(P)
    after = free_bytes()
    assert before - after <= 8 * P.xsize + 100 * MB
    assert h.factor(P.A2x) == 0
    assert after - free_bytes() >= 150 * MB


def test_a_large_structures_memory_is_given_back(cuda_ok, problem):
    """A handle that goes on to a small structure holds no more than a small multiple of it."""
    small = plate(20, 20)
    values = (problem.A2x, small.A2x)
    h = swc.Handle(0)
    before = free_bytes()

    def step(P, x):
        h.analyze(P.n, P.A2p, P.A2i, P.lC, P.Ls, P.Li_ptr, P.super, P.prunePtr, P.pruneSet)
        after = free_bytes()
        assert h.factor(x) == 0
        assert h.factor(x) == 0
        return after

    step(problem, values[0])
    assert before - free_bytes() >= 8 * problem.xsize
    assert before - step(small, values[1]) <= 100 * MB
    assert before - free_bytes() <= 40 * MB      # a few tables, the two graphs


def test_growing_numbers_of_right_hand_sides_keep_one_workspace(cuda_ok, problem):
    import torch
    P = problem
    b = torch.randn(48, P.n, dtype=torch.float64, device="cuda")
    used = []
    for counts in ([48], [1, 2, 3, 5, 8, 13, 21, 34, 48]):
        h = analyzed(P)
        assert h.factor(P.A2x) == 0
        before = free_bytes()
        for k in counts:
            h.solve(b[:k].contiguous() if k > 1 else b[0].contiguous())
        used.append(before - free_bytes())
        del h
    assert used[1] <= used[0] + 32 * MB
