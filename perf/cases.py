"""The work that programs have this library do, as cases that can be timed.

A case is a dict of plain values: what is called (`op`), the operator (`grid`: "plate" a
weighted 5-point grid, "brick" a weighted 7-point grid, "elastic" a 27-point grid with three
unknowns per node), its sizes, and the options of the call.  The matrices are seeded graph
operators in a geometric nested-dissection order with the library's own supernode partition;
the structure depends on the sizes alone, the values on the seed.

ops:
  factor      Handle.factor with device values; the result is L (the reference's layout).
  refine      Handle.factor, then Handle.refine of nrhs right-hand sides (default tolerance).
  solve       Handle.solve of nrhs right-hand sides with a factor made beforehand.
  batch       Handle.factor and Handle.refine of a block-diagonal batch of plates.
  likelihood  one step of a Gaussian likelihood: factor, log det, solve, and the gradients of
              the log determinant and of the quadratic form with respect to the values.
  dropin      sw_cholesky_left_par_05 on host arrays, analysis and transfers included.
"""
import math

import numpy as np
import torch

import swcholesky_b200 as swc
from swcholesky_b200 import matrices

MODES = {"fp64": swc.SWC_MODE_FP64, "tf32x3": swc.SWC_MODE_MIXED_TF32X3,
         "bf16x3": swc.SWC_MODE_MIXED_BF16X3}
DENSE_MAX = 20000      # unknowns up to which exact() forms dense matrices


def listed():
    return [
        # a small plate refactored in a time-stepping or Newton loop: launches and latency
        dict(name="factor_plate_20", op="factor", grid="plate", nx=20, ny=20, nz=1, mode="fp64", nrhs=0),
        # a 2D mesh of the size most direct solvers are called with
        dict(name="factor_plate_100", op="factor", grid="plate", nx=100, ny=100, nz=1, mode="fp64", nrhs=0),
        # an ordinary 3D scalar problem with uneven sides
        dict(name="factor_brick_41", op="factor", grid="brick", nx=41, ny=37, nz=43, mode="fp64", nrhs=0),
        # the large 3D factorization in double precision
        dict(name="factor_brick_60", op="factor", grid="brick", nx=60, ny=60, nz=60, mode="fp64", nrhs=0),
        # vector unknowns, 81 entries a row: wide supernodes early in the tree
        dict(name="factor_elastic_24", op="factor", grid="elastic", nx=24, ny=23, nz=22, mode="fp64", nrhs=0),
        # the large 3D solve with tensor-core updates, refined to double precision
        dict(name="refine_tf32_brick_60", op="refine", grid="brick", nx=60, ny=60, nz=60, mode="tf32x3", nrhs=1),
        # several load cases of an ill-conditioned structure, refined
        dict(name="refine_bf16_elastic_36", op="refine", grid="elastic", nx=36, ny=35, nz=33, mode="bf16x3", nrhs=8),
        # one more right-hand side with a factor that is kept (the inner solve of an iteration)
        dict(name="solve_brick_60", op="solve", grid="brick", nx=60, ny=60, nz=60, mode="fp64", nrhs=1),
        # several right-hand sides of a 2D problem with a factor that is kept
        dict(name="solve_plate_301_rhs8", op="solve", grid="plate", nx=301, ny=287, nz=1, mode="fp64", nrhs=8),
        # many independent small systems of uneven size in one call
        dict(name="batch_48", op="batch", grid="plate", nx=30, ny=130, nz=48, mode="fp64", nrhs=1),
        # parameter fitting of a Gaussian Markov random field: value and gradients
        dict(name="likelihood_plate_320", op="likelihood", grid="plate", nx=320, ny=310, nz=1, mode="fp64", nrhs=1),
        # a program of the reference with its one call replaced: host arrays in and out
        dict(name="dropin_brick_24", op="dropin", grid="brick", nx=25, ny=24, nz=23, mode="fp64", nrhs=0),
    ]


def _sides(rng, grid, n):
    """Uneven sides of a grid of about n unknowns."""
    dim = 2 if grid == "plate" else 3
    side = (n / (3 if grid == "elastic" else 1)) ** (1.0 / dim)
    d = [max(3, round(side * rng.uniform(0.8, 1.25))) for _ in range(dim)]
    return dict(nx=d[0], ny=d[1], nz=d[2] if dim == 3 else 1)


def draw(rng):
    op = rng.choice(["factor", "factor", "refine", "refine", "solve", "solve", "batch", "likelihood", "dropin"])
    grid = "plate" if op in ("batch", "likelihood") else rng.choice(["plate", "brick", "elastic"])
    most = {"factor": 60000, "refine": 60000, "solve": 60000, "likelihood": 60000, "dropin": 15000}.get(op, 0)
    mode = rng.choice(list(MODES)) if op == "refine" else "fp64"
    nrhs = {"refine": rng.choice([1, 1, 2, 3, 5, 8]), "solve": rng.choice([1, 1, 2, 4, 7, 12]),
            "batch": 1, "likelihood": 1}.get(op, 0)
    if op == "batch":      # sides from nx to ny, nz matrices
        lo = rng.randint(12, 40)
        return dict(op=op, grid=grid, nx=lo, ny=lo + rng.randint(5, 80), nz=rng.randint(5, 40), mode=mode, nrhs=nrhs)
    n = math.exp(rng.uniform(math.log(400), math.log(most)))
    return dict(op=op, grid=grid, **_sides(rng, grid, n), mode=mode, nrhs=nrhs)


# ---- matrices ------------------------------------------------------------------------------

def _dims(case):
    return (case["nx"], case["ny"]) if case["grid"] == "plate" else (case["nx"], case["ny"], case["nz"])


def _structure(grid, dims, device):
    """Grid nodes and edges: (nodes, per offset of the stencil the edges' lower and upper ends);
    within one offset every node is the lower (and the upper) end of at most one edge."""
    dim = len(dims)
    if grid == "elastic":
        offs = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (a, b, c) > (0, 0, 0)]
    else:
        offs = [tuple(int(i == k) for i in range(dim)) for k in range(dim)]
    nodes = math.prod(dims)
    idx = torch.arange(nodes, device=device).reshape(dims[::-1]).permute(*range(dim - 1, -1, -1))
    us, vs = [], []
    for off in offs:
        a = tuple(slice(max(0, -o), d - max(0, o)) for o, d in zip(off, dims))
        b = tuple(slice(max(0, o), d - max(0, -o)) for o, d in zip(off, dims))
        us.append(idx[a].reshape(-1))
        vs.append(idx[b].reshape(-1))
    return nodes, us, vs


def _incident(nodes, us, vs, w):
    """Per node the sum of its edges' weights, in a fixed order."""
    out = torch.zeros((nodes,) + w.shape[1:], dtype=w.dtype, device=w.device)
    at = 0
    for u, v in zip(us, vs):
        out[u] += w[at:at + u.numel()]
        out[v] += w[at:at + u.numel()]
        at += u.numel()
    return out


def _matrix(grid, dims, seed, device):
    """Lower CSC of the ordered operator (int32 columns and rows on the host, values on the
    device): a weighted graph Laplacian (log-normal weights) plus a diagonal shift; "elastic"
    has a symmetric positive definite 3 x 3 coupling per edge and a condition number of about
    1e6, "brick" of about 1e4, "plate" of about 1e2."""
    g = torch.Generator(device=device).manual_seed(int(seed))
    nodes, us, vs = _structure(grid, dims, device)
    u, v = torch.cat(us), torch.cat(vs)
    dof = 3 if grid == "elastic" else 1
    n = nodes * dof
    perm = torch.from_numpy(matrices.nested_dissection(dims, dof=dof)).to(device)
    place = torch.empty(n, dtype=torch.int64, device=device)
    place[perm] = torch.arange(n, device=device)
    sigma = {"plate": 0.7, "brick": 0.5, "elastic": 1.0}[grid]
    w = torch.exp(sigma * torch.randn(u.numel(), generator=g, device=device, dtype=torch.float64))
    if dof == 1:
        diag = _incident(nodes, us, vs, w)
        diag += 0.1 if grid == "plate" else 2e-3
        rows = torch.cat([torch.arange(n, device=device), u])
        cols = torch.cat([torch.arange(n, device=device), v])
        vals = torch.cat([diag, -w])
    else:
        d = torch.randn(u.numel(), 3, generator=g, device=device, dtype=torch.float64)
        d = d / d.norm(dim=1, keepdim=True)
        eye = torch.eye(3, device=device, dtype=torch.float64)
        blk = w[:, None, None] * (eye + d[:, :, None] * d[:, None, :])
        diag = _incident(nodes, us, vs, blk)
        shift = 2.0 * float(diag.diagonal(dim1=1, dim2=2).max()) / 1e6
        diag += shift * eye
        k = torch.arange(3, device=device)
        low = torch.tril_indices(3, 3, device=device)
        at = 3 * torch.arange(nodes, device=device)
        rows = torch.cat([(at[:, None] + low[0]).reshape(-1), (3 * u[:, None, None] + k[:, None]).expand(-1, 3, 3).reshape(-1)])
        cols = torch.cat([(at[:, None] + low[1]).reshape(-1), (3 * v[:, None, None] + k).expand(-1, 3, 3).reshape(-1)])
        vals = torch.cat([diag[:, low[0], low[1]].reshape(-1), -blk.reshape(-1)])
    rows, cols = place[rows], place[cols]
    lo, hi = torch.minimum(rows, cols), torch.maximum(rows, cols)
    key, order = torch.sort(lo * n + hi)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=device)
    indptr[1:] = torch.cumsum(torch.bincount(lo, minlength=n), 0)
    return n, indptr.to(torch.int32).cpu().numpy(), (key % n).to(torch.int32).cpu().numpy(), vals[order].contiguous()


def _batch_sides(case):
    """The matrices' sides: spread over [nx, ny], in a fixed mixed order."""
    return [case["nx"] + (37 * k * k + 11 * k) % (case["ny"] - case["nx"] + 1) for k in range(case["nz"])]


class _Mat:
    """One ordered matrix of a batch (n, indptr, indices), as Handle.batch_analyze takes it."""

    def __init__(self, n, indptr, indices):
        self.n, self.indptr, self.indices = n, indptr, indices


def _batch(case, seed, device):
    mats, vals = [], []
    for k, s in enumerate(_batch_sides(case)):
        n, c, r, x = _matrix("plate", (s, s), 1000 * int(seed) + k, device)
        mats.append(_Mat(n, c, r))
        vals.append(x)
    return mats, vals


def _rhs(n, nrhs, seed, device):
    g = torch.Generator(device=device).manual_seed(int(seed) + 77)
    b = torch.randn(max(nrhs, 1), n, generator=g, device=device, dtype=torch.float64)
    return b[0].contiguous() if nrhs <= 1 else b


# ---- states and passes ---------------------------------------------------------------------

class _DeviceL:
    """L of a handle where it is, for torch.as_tensor."""

    def __init__(self, handle):
        self.handle = handle     # alive as long as the tensor
        self.__cuda_array_interface__ = dict(shape=(handle.xsize,), typestr="<f8", version=2,
                                             data=(handle.device_L_ptr(), False))


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    op = case["op"]
    if op == "batch":
        mats, vals = _batch(case, seed, device)
        h = swc.Handle(device.index)
        h.batch_analyze(mats)
        b = _rhs(h.n, 1, seed, device)
        return dict(case=case, h=h, values=torch.cat(vals), b=b, x=torch.empty_like(b))
    n, c, r, x = _matrix(case["grid"], _dims(case), seed, device)
    bs = swc.supernodes(n, c, r)
    lay = swc.layout(n, c, r, bs)
    if op == "dropin":
        return dict(case=case, n=n, c=c, r=r, values=x.cpu().numpy(), bs=bs, lay=lay,
                    L=np.zeros(lay["xsize"], np.float64))
    h = swc.Handle(device.index)
    h.analyze(n, c, r, lay["lC"], lay["Ls"], lay["Li_ptr"], bs, lay["prunePtr"], lay["pruneSet"])
    b = _rhs(n, case["nrhs"], seed, device)
    s = dict(case=case, h=h, values=x, b=b, x=torch.empty_like(b))
    if op == "solve":
        torch.cuda.synchronize()
        h.factor(x, MODES[case["mode"]])
    if op == "likelihood":
        s["g_logdet"], s["g_quad"] = torch.empty_like(x), torch.empty_like(x)
    if op == "factor":
        s["L"] = torch.as_tensor(_DeviceL(h), device=device)
    return s


def run(s):
    case, op = s["case"], s["case"]["op"]
    if op == "dropin":
        lay = s["lay"]
        s["L"].fill(0.0)
        ok = swc.sw_cholesky_left_par_05(
            s["n"], s["c"], s["r"], s["values"], lay["lC"], lay["Ls"], lay["Li_ptr"], s["L"], s["bs"],
            s["bs"].size - 1, None, lay["prunePtr"], lay["pruneSet"], lay["levelPtr"].size - 1,
            lay["levelPtr"], None, 0, lay["parPtr"], lay["partition"], 0, 1, 0, 0, None)
        return dict(ok=int(ok), L=s["L"])
    h = s["h"]
    if op == "solve":
        return dict(x=h.solve(s["b"], out=s["x"]))
    info = h.factor(s["values"], MODES[case["mode"]])
    if op == "factor":
        return dict(info=info, L=s["L"])
    if op == "likelihood":
        logdet = h.logdet()
        x = h.solve(s["b"], out=s["x"])
        h.logdet_grad(s["g_logdet"])
        h.solve_grad(x, x, s["g_quad"])
        return dict(info=info, logdet=logdet, x=x, g_logdet=s["g_logdet"], g_quad=s["g_quad"])
    x = h.refine(s["b"], out=s["x"])[0]
    return dict(info=info, x=x)


# ---- what a pass cannot do without -----------------------------------------------------------

def _counts(grid, dims):
    """(unknowns, entries of A's lower triangle, entries of L, sum of squared column counts)."""
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    n, c, r, _ = _matrix(grid, dims, 0, device)
    bs = swc.supernodes(n, c, r, nrelax=[0, 0, 0], zrelax=[0.0, 0.0, 0.0])
    lip = swc.layout(n, c, r, bs)["Li_ptr"].astype(np.int64)
    col = lip[bs[1:]] - lip[bs[:-1]]                 # rows of each supernode
    width = np.diff(bs)
    cj = (np.repeat(col, width) - (np.arange(n) - np.repeat(bs[:-1], width))).astype(np.float64)
    return n, int(c[n]), float(cj.sum()), float((cj * cj).sum())


def work(case):
    op = case["op"]
    if op == "batch":
        each = [_counts("plate", (s, s)) for s in _batch_sides(case)]
        n, nnz, nl, fl = (sum(e[i] for e in each) for i in range(4))
    else:
        n, nnz, nl, fl = _counts(case["grid"], _dims(case))
    k = max(case["nrhs"], 1)
    factor = dict(bytes=8.0 * (nnz + nl), flops=fl)
    solve = dict(bytes=8.0 * (nl + 2.0 * n * k), flops=4.0 * nl * k)
    if op in ("factor", "dropin"):
        return factor
    if op == "solve":
        return solve
    if op == "likelihood":     # the selected inverse costs about twice the factorization
        return dict(bytes=factor["bytes"] + 16.0 * n + 16.0 * nnz, flops=3.0 * fl + 4.0 * nl + 4.0 * nnz)
    # factor, one solve and one residual
    return dict(bytes=factor["bytes"] + 16.0 * n * k, flops=fl + 4.0 * nl * k + 4.0 * nnz * k)


# ---- the same results in plain 64 bits ---------------------------------------------------------

def _dense(n, c, r, x):
    cols = torch.from_numpy(np.repeat(np.arange(n), np.diff(c))).to(x.device)
    rows = torch.from_numpy(r.astype(np.int64)).to(x.device)
    A = torch.zeros(n, n, dtype=torch.float64, device=x.device)
    A[rows, cols] = x
    A[cols, rows] = x
    return A, rows, cols


def _solve_dense(A, b):
    """x = A^{-1} b by a dense factorization and two steps of refinement; b (n,) or (k, n)."""
    L = torch.linalg.cholesky(A)
    B = b.reshape(-1, A.shape[0]).T
    X = torch.cholesky_solve(B, L)
    for _ in range(2):
        X = X + torch.cholesky_solve(B - A @ X, L)
    return X.T.reshape(b.shape).contiguous(), L


def exact(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    op = case["op"]
    if op == "batch":
        mats, vals = _batch(case, seed, device)
        if max(m.n for m in mats) > DENSE_MAX:
            return None
        b = _rhs(sum(m.n for m in mats), 1, seed, device)
        xs, at = [], 0
        for m, v in zip(mats, vals):
            A = _dense(m.n, m.indptr, m.indices, v)[0]
            xs.append(_solve_dense(A, b[at:at + m.n])[0])
            at += m.n
        return dict(info=None, x=torch.cat(xs))
    dof = 3 if case["grid"] == "elastic" else 1
    if math.prod(_dims(case)) * dof > DENSE_MAX:
        return None
    n, c, r, v = _matrix(case["grid"], _dims(case), seed, device)
    A, rows, cols = _dense(n, c, r, v)
    b = _rhs(n, case["nrhs"], seed, device)
    if op in ("refine", "solve"):
        x = _solve_dense(A, b)[0]
        return dict(x=x) if op == "solve" else dict(info=None, x=x)
    if op == "likelihood":
        x, L = _solve_dense(A, b)
        Z = torch.cholesky_inverse(L)
        off = (rows != cols).to(torch.float64) + 1.0
        return dict(info=None, logdet=float(2.0 * torch.log(L.diagonal()).sum()), x=x,
                    g_logdet=Z[rows, cols] * off, g_quad=-x[rows] * x[cols] * off)
    # L where the layout (an input of the call) has its entries
    L = torch.linalg.cholesky(A).cpu().numpy()
    bs = swc.supernodes(n, c, r)
    lay = swc.layout(n, c, r, bs)
    lip, ls = lay["Li_ptr"].astype(np.int64), lay["Ls"]
    out = [L[ls[lip[bs[s]]:lip[bs[s + 1]]]][:, bs[s]:bs[s + 1]].T.reshape(-1) for s in range(bs.size - 1)]
    out = np.concatenate(out)
    if op == "dropin":
        return dict(ok=None, L=out)
    return dict(info=None, L=torch.from_numpy(out))
