// Adjoint of the supernodal factorization: gradients with respect to the stored nonzeros of
// A (the lower triangle of P A P^T, symmetric storage: a stored off-diagonal value stands
// for both A_ij and A_ji).
//
// log det A.  d log det A = tr(A^{-1} dA), so the gradient is A^{-1} on the pattern of A,
// times 2 off the diagonal.  A^{-1} is computed on the whole pattern of L (the selected
// inverse) by a reverse sweep over the elimination tree, root to leaves, that retraces the
// factorization's POTRF / TRSM / SYRK steps backwards.  Per column block K (a small supernode,
// or 64 columns of a wide one) with the rows R of L below it:
//     U    = L_RK L_KK^{-1}
//     Z_RK = -Z_RR U
//     Z_KK = L_KK^{-T} L_KK^{-1} - U^T Z_RK
// (Takahashi, Fagan and Chin, 1973; the supernodal form of the reverse-mode Cholesky of
// Murray, "Differentiation of the Cholesky decomposition", 2016).
//
// The sweep is multifrontal: every supernode with children holds A^{-1} on its whole front (all
// rows of its panel squared, both triangles, column-major, leading dimension m), whose block
// over the off-diagonal rows is copied from the parent's front through the child's row map
// (rows are contained in the parent's).  Z_RR is then contiguous, so every product is a dense
// one; a front lives until its children are done, in an arena placed at analysis.  Supernodes
// without children keep only their panel.  Small supernodes take one kernel per level (a warp
// or a CTA each, everything in shared memory but Z_RR, which is read once from the parent's
// front); wide ones 64-column steps of three launches with 64x64 DMMA tiles.  Bound: the chain of
// steps from the root (22 of them for a 320 x 310 5-point grid, about 45 us each), then the
// small fronts' latency.  Against a sweep of 64-row FMA tiles per column block with Z_RR
// gathered entry by entry from all ancestors, that grid's gradient takes 1.3 ms, not 4.4 (B200).
//
// Functions of x = A^{-1} b.  With lam = A^{-1} (df/dx):
//     df/dA_ij = -(lam_i x_j + lam_j x_i)  (i != j),   -lam_i x_i  (i == j).
//
// The reference has no adjoint; this is a new capability of the library.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <map>
#include <string>
#include <vector>

#include "swc_engine.h"
#include "swc_front.h"
#include "swc_tile.h"

namespace swc {

namespace {

struct AdjDev {
  const int *parent, *rel, *apos;   // the tree (swc_front.h)
  const int64_t *zoff;              // per supernode: its front (or panel) in Z
  const char *kids;                 // per supernode: has children (a whole front is kept)
  double *Z;
  double *UT;                       // per task of the current step: U^T, 64 x rows, see utoff
  double *P;                        // per task: U(X,:)^T (Z_RR U)(X,:), 64 x 64
  double *grad;                     // per entry of A
};

__device__ __forceinline__ int nrows_of(const DevSym &S, int s) {
  return (int)(S.rowptr[s + 1] - S.rowptr[s]);
}

// ---- small supernodes: NW warps each.  In shared memory: the padded panel (front layout, see
// front_ld), in which U replaces L_RK; Y = Z_RR U; T = L_KK^{-1}.  y_global: the two panels do
// not fit, Y is read back from Z_RK = -Y (its scratch of 64 doubles per warp stays).
constexpr int ZW_W = 16, ZW_WARPS = 2;            // warp variant: width limit, warps per CTA
constexpr int ZW_SLICE = (2 * FRONT_WARP_ELEMS + ZW_W * (ZW_W + 4)) * 8 + FRONT_WARP_M * 4;
constexpr int ZC_T = 256, ZC_W = ZC_T / 32;
constexpr int ADJ_SMEM_MAX = 220 * 1024;

template <int NW>
__device__ __forceinline__ void zsync() {
  if (NW == 1) __syncwarp(); else __syncthreads();
}

template <int NW>
__device__ void adj_small_body(const DevSym &S, const AdjDev &A, int s, double *Pm, double *Y, double *T,
                               int *rel, bool y_global) {
  constexpr int NTH = 32 * NW;
  const int t = NW == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  const int lane = t & 31, warp = t >> 5, g = lane >> 2, kq = lane & 3;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int m = nrows_of(S, s), r = m - w;
  const int wp = front_wp(w), ld = front_ld(w, m), pad = wp - w, nk = wp >> 3, nr8 = (r + 7) >> 3;
  const int ldt = adj_ldt(w);
  const double *Ls = S.L + S.xptr[s];
  double *Z = A.Z + A.zoff[s];
  const bool front = A.kids[s] != 0;
  // the panel (upper triangle, padding: zeros; padded diagonal: ones) and the row map
#pragma unroll 8
  for (int e = t; e < wp * ld; e += NTH) {
    const int j = e / ld, i = e - j * ld;
    const int row = i < wp ? i : i - pad;
    const double v = ld_if(Ls + (size_t)j * m + row, j < w && (i < wp ? i < w && i >= j : row < m));
    Pm[e] = i == j && j >= w ? 1.0 : v;
  }
  for (int e = t; e < wp * ldt; e += NTH) T[e] = 0.0;
  const int *grel = A.rel + (S.rowptr[s] - f);
  for (int i = t; i < r; i += NTH) rel[i] = grel[i];
  zsync<NW>();
  // inverses of the 8x8 diagonal blocks: lane j of eight forms column j by forward substitution
  for (int c = t; c < wp; c += NTH) {
    const int b0 = c & ~7, j = c & 7;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      double acc = i == j ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < i; ++k)
        if (k >= j) acc = fma(-Pm[(b0 + k) * ld + b0 + i], x[k], acc);
      x[i] = i >= j ? acc / Pm[(b0 + i) * ld + b0 + i] : 0.0;
      T[c * ldt + b0 + i] = x[i];
    }
  }
  zsync<NW>();
  // T_ik = -T_ii sum_{k <= j < i} L_ij T_jk, a block column per warp (scratch: 64 doubles of Y)
  double *Ww = Y + warp * 64;
  for (int k = warp; k < nk; k += NW)
    for (int i = k + 1; i < nk; ++i) {
      double a[2] = {0.0, 0.0};
      for (int j = k; j < i; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          dmma(a, Pm[(8 * j + 4 * h + kq) * ld + 8 * i + g], T[(8 * k + g) * ldt + 8 * j + 4 * h + kq]);
      Ww[(2 * kq) * 8 + g] = a[0];
      Ww[(2 * kq + 1) * 8 + g] = a[1];
      __syncwarp();
      double c[2] = {0.0, 0.0};
#pragma unroll
      for (int h = 0; h < 2; ++h)
        dmma(c, neg(T[(8 * i + 4 * h + kq) * ldt + 8 * i + g]), Ww[g * 8 + 4 * h + kq]);
      T[(8 * k + 2 * kq) * ldt + 8 * i + g] = c[0];
      T[(8 * k + 2 * kq + 1) * ldt + 8 * i + g] = c[1];
      __syncwarp();
    }
  zsync<NW>();
  // U = L_RK T in place (a block row per warp; output block columns in increasing order only
  // read input block columns at or after them)
  for (int ib = warp; ib < nr8; ib += NW) {
    double *row = Pm + wp + 8 * ib;
    for (int n = 0; n < nk; ++n) {
      double c[2] = {0.0, 0.0};
      for (int k = 8 * n; k < wp; k += 4) dmma(c, row[(k + kq) * ld + g], T[(8 * n + g) * ldt + k + kq]);
      __syncwarp();
      row[(8 * n + 2 * kq) * ld + g] = c[0];
      row[(8 * n + 2 * kq + 1) * ld + g] = c[1];
      __syncwarp();
    }
  }
  zsync<NW>();
  pdl_wait();   // so far from L alone
  // Y = Z_RR U, Z_RR read from the parent's front and, for a front of its own, written to it
  if (r > 0) {
    const int p = A.parent[s], mp = nrows_of(S, p);
    const double *Zp = A.Z + A.zoff[p];
    for (int ib = warp; ib < nr8; ib += NW) {
      const int i = 8 * ib + g;
      const bool iin = i < r;
      const double *zrow = Zp + (iin ? rel[i] : 0);
      double *own = Z + (size_t)w * m + w + i;
      for (int n0 = 0; n0 < nk; n0 += 4) {
        double c[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q][0] = c[q][1] = 0.0;
        for (int k0 = 0; k0 < r; k0 += 16) {
          double a[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int k = k0 + 4 * u + kq;
            a[u] = ld_if(zrow + (size_t)rel[k < r ? k : 0] * mp, iin && k < r);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int k = k0 + 4 * u + kq;
            if (front && n0 == 0 && iin && k < r) own[(size_t)k * m] = a[u];
            if (k0 + 4 * u < r)
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (n0 + q < nk)
                  dmma(c[q], a[u], Pm[(8 * (n0 + q) + g) * ld + wp + min(k, 8 * nr8 - 1)]);
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (n0 + q < nk) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int col = 8 * (n0 + q) + 2 * kq + e;
              if (!y_global) Y[col * ld + wp + 8 * ib + g] = c[q][e];
              if (iin && col < w) {   // Z_RK = -Y
                Z[(size_t)col * m + w + i] = -c[q][e];
                if (front) Z[(size_t)(w + i) * m + col] = -c[q][e];
              }
            }
          }
      }
    }
  }
  zsync<NW>();
  // Z_KK = T^T T + U^T Y, lower 8x8 blocks
  int blk = 0;
  for (int a = 0; a < nk; ++a)
    for (int b = 0; b <= a; ++b, ++blk) {
      if (blk % NW != warp) continue;
      double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      for (int k = 8 * a; k < wp; k += 4)
        dmma(c[0], T[(8 * a + g) * ldt + k + kq], T[(8 * b + g) * ldt + k + kq]);
      for (int k = 0; k < 8 * nr8; k += 8)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = k + 4 * h + kq, col = 8 * b + g;
          const double y = !y_global ? Y[col * ld + wp + row]
                           : (row < r && col < w) ? -Z[(size_t)col * m + w + row] : 0.0;
          dmma(c[h], Pm[(8 * a + g) * ld + wp + row], y);
        }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = 8 * a + g, j = 8 * b + 2 * kq + e;
        if (i < w && j <= i) {
          const double v = c[0][e] + c[1][e];
          Z[(size_t)j * m + i] = v;
          Z[(size_t)i * m + j] = v;
        }
      }
    }
  zsync<NW>();
  // gradient of the entries of A in the supernode's columns
  for (int j = warp; j < w; j += NW)
    for (int p = S.Ap[f + j] + lane; p < S.Ap[f + j + 1]; p += 32) {
      const int pos = A.apos[p];
      if (pos < 0) { atomicExch(&S.status[1], 1); A.grad[p] = 0.0; continue; }
      A.grad[p] = Z[(size_t)j * m + pos] * (pos == j ? 1.0 : 2.0);
    }
  zsync<NW>();
}

__global__ void __launch_bounds__(ZC_T) k_adj_small(DevSym S, AdjDev A, const int *list) {
  extern __shared__ double zsm[];
  pdl_trigger();
  const int e = list[blockIdx.x], s = e < 0 ? ~e : e;   // ~s: y_global
  const int w = S.super[s + 1] - S.super[s], m = nrows_of(S, s);
  const int pe = front_wp(w) * front_ld(w, m);
  const int ye = e < 0 ? ZC_W * 64 : max(pe, ZC_W * 64);
  adj_small_body<ZC_W>(S, A, s, zsm, zsm + pe, zsm + pe + ye,
                       reinterpret_cast<int *>(zsm + pe + ye + front_wp(w) * adj_ldt(w)), e < 0);
}

__global__ void __launch_bounds__(ZW_WARPS * 32) k_adj_warp(DevSym S, AdjDev A, const int *list, int count) {
  extern __shared__ double zsm[];
  pdl_trigger();
  const int q = blockIdx.x * ZW_WARPS + (threadIdx.x >> 5);
  if (q >= count) return;
  double *P = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(zsm) +
                                         (size_t)(threadIdx.x >> 5) * ZW_SLICE);
  double *Y = P + FRONT_WARP_ELEMS, *T = Y + FRONT_WARP_ELEMS;
  adj_small_body<1>(S, A, list[q], P, Y, T, reinterpret_cast<int *>(T + ZW_W * (ZW_W + 4)), false);
}

// ---- wide supernodes ----------------------------------------------------------------------

// The block over the off-diagonal rows, from the parent's front: task = (s, i0, j0).
__global__ void __launch_bounds__(256) k_adj_copy(DevSym S, AdjDev A, const int4 *tasks) {
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, w = S.super[s + 1] - S.super[s], m = nrows_of(S, s), r = m - w;
  const int p = A.parent[s], mp = nrows_of(S, p);
  const int *rel = A.rel + (S.rowptr[s] - S.super[s]);
  const int i = tk.y + (threadIdx.x & 63);
  pdl_trigger();
  pdl_wait();
  if (i >= r) return;
  const double *src = A.Z + A.zoff[p] + rel[i];
  double *dst = A.Z + A.zoff[s] + (size_t)w * m + w + i;
#pragma unroll 4
  for (int j = tk.z + (threadIdx.x >> 6); j < min(r, tk.z + TB); j += 4)
    dst[(size_t)j * m] = src[(size_t)rel[j] * mp];
}

// task = (s, column block b, first row x0 of R, task index of x0 = 0): rows x0 .. x0 + 63 of
// U = L_RK T with T the inverse of the diagonal block the factorization stored; U^T at
// UT + 4096 * (first task) + row * 64.
// T(k, c) of the diagonal block at ti (column-major as the factorization stored it), as [k][c].
__device__ __forceinline__ void load_tinv(double *Ts, const double *ti, int w) {
#pragma unroll 8
  for (int e = threadIdx.x; e < TB * TB; e += MT) {
    const int c = e >> 6, k = e & (TB - 1);
    Ts[k * LDS + c] = ld_if(ti + e, k < w && c < w);
  }
}

constexpr int TT_SMEM = 2 * TB * LDS * 8;   // two 64x64 operands
static_assert(2 * TB * LDS >= 2 * STAGE, "the product's stages fit");
__global__ void __launch_bounds__(MT) k_adj_u(DevSym S, AdjDev A, const int4 *tasks) {
  extern __shared__ double zsm[];
  double *Ts = zsm, *Lx = zsm + TB * LDS;   // [k][column], [k][row]
  pdl_trigger();
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, c0 = tk.y * TB, x0 = tk.z;
  const int m = nrows_of(S, s), w = min(TB, S.super[s + 1] - S.super[s] - c0), off = c0 + w;
  const int nrow = min(TB, m - off - x0);
  const double *Lb = S.L + S.xptr[s] + (size_t)c0 * m + off + x0;
  load_tinv(Ts, S.dinv + ((size_t)S.dinv_off[s] + tk.y) * (TB * TB), w);
#pragma unroll 8
  for (int e = threadIdx.x; e < TB * TB; e += MT) {
    const int k = e >> 6, q = e & (TB - 1);
    Lx[k * LDS + q] = ld_if(Lb + (size_t)k * m + q, q < nrow && k < w);
  }
  __syncthreads();
  TileAcc acc;   // U^T: rows are columns of the block
  acc.zero();
  dmma_tile_smem(Ts, Lx, TB, acc);
  pdl_wait();   // UT may be read until the kernel ahead ends
  double *UT = A.UT + (size_t)tk.w * (TB * TB) + (size_t)x0 * TB;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (acc_col(j, e) < nrow) UT[(size_t)acc_col(j, e) * TB + acc_row(i)] = acc.v[i][j][e];
}

// The same rows of Z_RK = -Z_RR U (DMMA, K = all rows of R) and their share of U^T Z_RR U.
__global__ void __launch_bounds__(MT, 3) k_adj_zrk(DevSym S, AdjDev A, const int4 *tasks) {
  extern __shared__ double zsm[];
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, c0 = tk.y * TB, x0 = tk.z;
  const int m = nrows_of(S, s), w = min(TB, S.super[s + 1] - S.super[s] - c0), off = c0 + w;
  pdl_trigger();
  pdl_wait();
  const int mr = m - off, nrow = min(TB, mr - x0);
  double *Z = A.Z + A.zoff[s];
  const double *UT = A.UT + (size_t)tk.w * (TB * TB);
  TileAcc acc;
  acc.zero();
  dmma_tile_product(Z + (size_t)off * m + off + x0, m, nrow, UT, TB, w, mr, zsm, acc);
  __syncthreads();
  double *ys = zsm, *ux = zsm + TB * LDS;   // [row][column]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = acc_row(i), c = acc_col(j, e);
        ys[r * LDS + c] = (r < nrow && c < w) ? acc.v[i][j][e] : 0.0;
      }
#pragma unroll 8
  for (int e = threadIdx.x; e < TB * TB; e += MT) {
    const int r = e >> 6, c = e & (TB - 1);
    ux[r * LDS + c] = ld_if(UT + (size_t)(x0 + r) * TB + c, r < nrow && c < w);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < TB * TB; e += MT) {
    const int c = e >> 6, r = e & (TB - 1);
    if (c < w && r < nrow) Z[(size_t)(c0 + c) * m + off + x0 + r] = -ys[r * LDS + c];
  }
  for (int e = threadIdx.x; e < TB * TB; e += MT) {
    const int r = e >> 6, c = e & (TB - 1);
    if (c < w && r < nrow) Z[(size_t)(off + x0 + r) * m + c0 + c] = -ys[r * LDS + c];
  }
  acc.zero();   // U(X)^T Y(X)
  dmma_tile_smem(ux, ys, (nrow + 3) & ~3, acc);
  double *P = A.P + (size_t)blockIdx.x * (TB * TB);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<double2 *>(P + acc_row(i) * TB + acc_col(j, 0)) =
          make_double2(acc.v[i][j][0], acc.v[i][j][1]);
}

// Z_KK = T^T T + the row blocks' shares.  unit = (s, column block, first task, tasks).
__global__ void __launch_bounds__(MT) k_adj_zkk(DevSym S, AdjDev A, const int4 *units) {
  extern __shared__ double zsm[];
  pdl_trigger();
  const int4 un = units[blockIdx.x];
  const int s = un.x, c0 = un.y * TB;
  const int m = nrows_of(S, s), w = min(TB, S.super[s + 1] - S.super[s] - c0);
  load_tinv(zsm, S.dinv + ((size_t)S.dinv_off[s] + un.y) * (TB * TB), w);
  __syncthreads();
  TileAcc acc;
  acc.zero();
  dmma_tile_smem(zsm, zsm, TB, acc);
  pdl_wait();
  for (int t = un.z; t < un.z + un.w; ++t) {
    const double *P = A.P + (size_t)t * (TB * TB);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 p = *reinterpret_cast<const double2 *>(P + acc_row(i) * TB + acc_col(j, 0));
        acc.v[i][j][0] += p.x;
        acc.v[i][j][1] += p.y;
      }
  }
  double *Z = A.Z + A.zoff[s] + (size_t)c0 * m + c0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = acc_row(i), c = acc_col(j, e);
        if (r < w && c <= r) {
          Z[(size_t)c * m + r] = acc.v[i][j][e];
          Z[(size_t)r * m + c] = acc.v[i][j][e];
        }
      }
}

// Gradient of the entries of A in a wide supernode's columns: one warp per (s, column).
__global__ void k_adj_grad(DevSym S, AdjDev A, const int2 *cols, int count) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  pdl_trigger();
  pdl_wait();
  if (t >= count) return;
  const int s = cols[t].x, j = cols[t].y, c = j - S.super[s];
  const double *col = A.Z + A.zoff[s] + (size_t)c * nrows_of(S, s);
  for (int p = S.Ap[j] + lane; p < S.Ap[j + 1]; p += 32) {
    const int pos = A.apos[p];
    if (pos < 0) { atomicExch(&S.status[1], 1); A.grad[p] = 0.0; continue; }
    A.grad[p] = col[pos] * (pos == c ? 1.0 : 2.0);
  }
}

// Supernode holding column j.
__device__ __forceinline__ int snode_of(const DevSym &S, int j) {
  int lo = 0, hi = S.nsuper;   // last s with super[s] <= j
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (S.super[mid] <= j) lo = mid; else hi = mid;
  }
  return lo;
}

// Partial sums of log L_jj (fixed grid, fixed order: deterministic).
constexpr int LD_BLOCKS = 256;
__global__ void __launch_bounds__(256) k_logdet(DevSym S, double *partial) {
  __shared__ double red[256];
  double acc = 0.0;
  for (int j = blockIdx.x * 256 + threadIdx.x; j < S.n; j += LD_BLOCKS * 256) {
    const int s = snode_of(S, j);
    const int c = j - S.super[s];
    acc += log(S.L[S.xptr[s] + (size_t)c * nrows_of(S, s) + c]);
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// grad[p] = -(lam_i x_j + lam_j x_i) for i != j, -lam_i x_i on the diagonal.
__global__ void k_solve_grad(DevSym S, const double *x, const double *lam, double *grad) {
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= S.n) return;
  const double xj = x[j], lj = lam[j];
  for (int p = S.Ap[j] + lane; p < S.Ap[j + 1]; p += 32) {
    const int i = S.Ai[p];
    grad[p] = (i == j) ? -lam[i] * xj : -(lam[i] * xj + lj * x[i]);
  }
}

}  // namespace

// ---------------------------------------------------------------------------------------

// Reverse sweep: waves of supernodes, parents before children.
struct AdjointPlan {
  struct Step { int task_off, task_cnt, unit_off, unit_cnt; };   // one 64-column step of a wave
  struct AdjWave {
    int warp_off, warp_cnt, cta_off, cta_cnt, cta_smem, copy_off, copy_cnt, col_off, col_cnt;
    std::vector<Step> steps;
  };
  std::vector<AdjWave> waves;
  std::vector<int> warp_list, cta_list, parent;
  std::vector<int4> copies, tasks, units;
  std::vector<int2> cols;          // (s, column) of the wide supernodes
  std::vector<char> kids;
  std::vector<int64_t> zoff;
  int64_t z_len = 0;
  int max_tasks = 0;
};

// Doubles of a supernode's place in Z: its whole front where it has children (they read it) or is
// wide, else its panel.
static int64_t adj_front_len(const HostSym &H, int s, bool whole) {
  const int64_t m = H.rowptr[s + 1] - H.rowptr[s];
  return (m * (whole ? m : H.super[s + 1] - H.super[s]) + 15) & ~(int64_t)15;
}

// Places of the fronts when the waves run in this order: a front is read by its children only, and
// freed once the last one is done.
static int64_t place_adjoint(const std::vector<std::vector<int>> &waves, const std::vector<int64_t> &len,
                             const FrontPlan &F, const std::vector<int> &parent, std::vector<int64_t> &zoff) {
  FrontArena A;
  std::vector<int> left(len.size());   // children not done yet
  for (size_t s = 0; s < len.size(); ++s) left[s] = F.child_ptr[s + 1] - F.child_ptr[s];
  std::vector<int> order;
  for (const std::vector<int> &here : waves) {
    order = here;   // the largest first: less is lost between them
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return len[a] > len[b]; });
    for (int s : order) zoff[s] = A.take(len[s]);
    for (int s : here) {
      if (F.child_ptr[s + 1] == F.child_ptr[s]) A.give(zoff[s], len[s]);
      const int p = parent[s];
      if (p >= 0 && --left[p] == 0) A.give(zoff[p], len[p]);
    }
  }
  return A.end();
}

// The order when a level's fronts are too many to be held together (many narrow supernodes under a
// wide border: a front is as large as the border squared): groups of at most `budget` doubles, one
// after the other, each with everything below it before the next; small subtrees first, so that
// little is held while the large ones run.
static std::vector<std::vector<int>> adjoint_groups(const std::vector<int64_t> &len, const FrontPlan &F,
                                                    const std::vector<int> &parent, int64_t budget) {
  const int ns = (int)len.size();
  std::vector<int64_t> weight(len);   // of the subtree
  std::vector<std::vector<int>> open(1), waves;   // open: lists whose parents are done, last one first
  for (int s = 0; s < ns; ++s) {   // parents have larger numbers
    if (parent[s] >= 0) weight[parent[s]] += weight[s];
    else open[0].push_back(s);
  }
  while (!open.empty()) {
    std::vector<int> here = std::move(open.back());
    open.pop_back();
    int64_t sum = 0;
    for (int s : here) sum += len[s];
    if (sum > budget && here.size() > 1) {
      std::stable_sort(here.begin(), here.end(), [&](int a, int b) { return weight[a] < weight[b]; });
      size_t k = 1;
      for (sum = len[here[0]]; k < here.size() && sum + len[here[k]] <= budget; ++k) sum += len[here[k]];
      if (k < here.size()) {
        open.emplace_back(here.begin() + k, here.end());
        here.resize(k);
      }
    }
    std::vector<int> next;
    for (int s : here) next.insert(next.end(), F.child.begin() + F.child_ptr[s], F.child.begin() + F.child_ptr[s + 1]);
    if (!next.empty()) open.push_back(std::move(next));
    waves.push_back(std::move(here));
  }
  return waves;
}

static void build_adjoint_plan(const HostSym &H, const Plan &P, const FrontPlan &F, AdjointPlan &AP) {
  const std::vector<int> &super = H.super;
  const int ns = (int)super.size() - 1, nlev = (int)P.waves.size();
  auto width = [&](int s) { return super[s + 1] - super[s]; };
  auto rows = [&](int s) { return (int)(H.rowptr[s + 1] - H.rowptr[s]); };
  std::vector<int> level(ns, 0);
  AP.parent.assign(ns, -1);
  AP.kids.assign(ns, 0);
  AP.zoff.assign(ns, 0);
  for (int s = 0; s < ns; ++s)
    for (int q = F.child_ptr[s]; q < F.child_ptr[s + 1]; ++q) {
      AP.parent[F.child[q]] = s;
      AP.kids[s] = 1;
      level[s] = std::max(level[s], level[F.child[q]] + 1);
    }
  std::vector<char> tiled(ns, 0);
  for (int s : P.big_list) tiled[s] = 1;
  std::vector<int64_t> len(ns);
  for (int s = 0; s < ns; ++s) len[s] = adj_front_len(H, s, AP.kids[s] || tiled[s]);
  // a wave per level, the root's first, where that needs no more memory than the factorization's
  // blocks may take (grids: 0.3 to 0.9 times L); else groups of a quarter of it
  std::vector<std::vector<int>> lists(nlev);
  for (int s = 0; s < ns; ++s) lists[nlev - 1 - level[s]].push_back(s);
  AP.z_len = place_adjoint(lists, len, F, AP.parent, AP.zoff);
  const int64_t limit = front_memory_limit(H.xsize);
  if (AP.z_len > limit) {
    std::vector<int64_t> zoff(ns, 0);
    std::vector<std::vector<int>> groups = adjoint_groups(len, F, AP.parent, limit / 4);
    const int64_t z_len = place_adjoint(groups, len, F, AP.parent, zoff);
    if (z_len < AP.z_len) {
      AP.z_len = z_len;
      AP.zoff = std::move(zoff);
      lists = std::move(groups);
    }
  }
  AP.waves.resize(lists.size());
  for (size_t v = 0; v < lists.size(); ++v) {
    const std::vector<int> &here = lists[v];
    AdjointPlan::AdjWave &W = AP.waves[v];
    W.warp_off = (int)AP.warp_list.size();
    W.cta_off = (int)AP.cta_list.size();
    W.copy_off = (int)AP.copies.size();
    W.col_off = (int)AP.cols.size();
    W.cta_smem = 0;
    int fit = 0, maxnb = 0;
    auto warp_fits = [&](int s) {
      const int w = width(s), m = rows(s);
      return !tiled[s] && w <= ZW_W && m <= FRONT_WARP_M && front_wp(w) * front_ld(w, m) <= FRONT_WARP_ELEMS;
    };
    for (int s : here) fit += warp_fits(s);
    for (int s : here) {
      const int w = width(s), m = rows(s);
      if (tiled[s]) {
        for (int j0 = 0; j0 < m - w; j0 += TB)
          for (int i0 = 0; i0 < m - w; i0 += TB) AP.copies.push_back(make_int4(s, i0, j0, 0));
        for (int j = 0; j < w; ++j) AP.cols.push_back(make_int2(s, super[s] + j));
        maxnb = std::max(maxnb, (w + TB - 1) / TB);
      } else if (fit >= FRONT_WARP_LEVEL_MIN && warp_fits(s)) {
        AP.warp_list.push_back(s);
      } else {
        const bool y_global = adj_small_smem(w, m, false) > ADJ_SMEM_MAX;
        AP.cta_list.push_back(y_global ? ~s : s);
        W.cta_smem = std::max<int>(W.cta_smem, (int)adj_small_smem(w, m, y_global));
      }
    }
    W.warp_cnt = (int)AP.warp_list.size() - W.warp_off;
    W.cta_cnt = (int)AP.cta_list.size() - W.cta_off;
    W.copy_cnt = (int)AP.copies.size() - W.copy_off;
    W.col_cnt = (int)AP.cols.size() - W.col_off;
    for (int t = 0; t < maxnb; ++t) {   // last column block first
      AdjointPlan::Step st{(int)AP.tasks.size(), 0, (int)AP.units.size(), 0};
      for (int s : here) {
        if (!tiled[s]) continue;
        const int w = width(s), b = (w + TB - 1) / TB - 1 - t;
        if (b < 0) continue;
        const int first = (int)AP.tasks.size() - st.task_off, mr = rows(s) - std::min(w, (b + 1) * TB);
        for (int x0 = 0; x0 < mr; x0 += TB) AP.tasks.push_back(make_int4(s, b, x0, first));
        AP.units.push_back(make_int4(s, b, first, (int)AP.tasks.size() - st.task_off - first));
      }
      st.task_cnt = (int)AP.tasks.size() - st.task_off;
      st.unit_cnt = (int)AP.units.size() - st.unit_off;
      AP.max_tasks = std::max(AP.max_tasks, st.task_cnt);
      W.steps.push_back(st);
    }
  }
}

bool check_adjoint_plan(const HostSym &H, const Plan &P, const FrontPlan &F, std::string &err) {
  if (!F.closed) return true;
  AdjointPlan AP;
  build_adjoint_plan(H, P, F, AP);
  const int ns = (int)H.super.size() - 1;
  auto width = [&](int s) { return H.super[s + 1] - H.super[s]; };
  auto bad = [&](const char *what, int s) {
    err = std::string("reverse sweep: ") + what + ", supernode " + std::to_string(s);
    return false;
  };
  std::vector<char> tiled(ns, 0), done(ns, 0);
  for (int s : P.big_list) tiled[s] = 1;
  std::vector<int64_t> len(ns);
  std::vector<int> left(ns), blocks(ns, 0), cols(ns, 0);
  for (int s = 0; s < ns; ++s) {
    left[s] = F.child_ptr[s + 1] - F.child_ptr[s];
    len[s] = adj_front_len(H, s, left[s] > 0 || tiled[s]);
  }
  std::map<int64_t, int64_t> live;   // the fronts held, by place
  for (const AdjointPlan::AdjWave &W : AP.waves) {
    std::vector<int> here;
    for (int k = W.warp_off; k < W.warp_off + W.warp_cnt; ++k) here.push_back(AP.warp_list[k]);
    for (int k = W.cta_off; k < W.cta_off + W.cta_cnt; ++k)
      here.push_back(AP.cta_list[k] < 0 ? ~AP.cta_list[k] : AP.cta_list[k]);
    for (int s : here)
      if (s < 0 || s >= ns || tiled[s]) return bad("a wide supernode among the small", s);
    for (size_t t = 0; t < W.steps.size(); ++t) {
      const AdjointPlan::Step &st = W.steps[t];
      int next = 0;
      for (int k = st.unit_off; k < st.unit_off + st.unit_cnt; ++k) {
        const int4 un = AP.units[k];
        const int s = un.x, nb = (width(s) + TB - 1) / TB;
        if (t == 0) here.push_back(s);
        if (!tiled[s] || un.y != nb - 1 - (int)t || un.z != next) return bad("column block out of order", s);
        const int mr = (int)(H.rowptr[s + 1] - H.rowptr[s]) - std::min(width(s), (un.y + 1) * TB);
        if (un.w != (mr + TB - 1) / TB || next + un.w > st.task_cnt) return bad("rows of a column block", s);
        for (int q = 0; q < un.w; ++q) {
          const int4 tk = AP.tasks[st.task_off + next + q];
          if (tk.x != s || tk.y != un.y || tk.z != q * TB || tk.w != next) return bad("task of a column block", s);
        }
        next += un.w;
        ++blocks[s];
      }
      if (next != st.task_cnt || next > AP.max_tasks) return bad("tasks of a step", -1);
    }
    for (int k = W.col_off; k < W.col_off + W.col_cnt; ++k) {
      const int s = AP.cols[k].x;
      if (!tiled[s] || AP.cols[k].y != H.super[s] + cols[s]++) return bad("gradient column", s);
    }
    for (int s : here) {
      if (done[s]) return bad("a supernode twice", s);
      const int p = AP.parent[s];
      if (p >= 0 && done[p] != 2) return bad("a supernode before its parent", s);
      done[s] = 1;
      const int64_t at = AP.zoff[s];
      auto nx = live.lower_bound(at);
      if (at < 0 || at + len[s] > AP.z_len || (nx != live.end() && nx->first < at + len[s]) ||
          (nx != live.begin() && std::prev(nx)->second > at))
        return bad("fronts overlap", s);
      live[at] = at + len[s];
    }
    for (int s : here) {
      done[s] = 2;
      if (tiled[s] && (blocks[s] != (width(s) + TB - 1) / TB || cols[s] != width(s)))
        return bad("column blocks or gradient columns missing", s);
      if (left[s] == 0) live.erase(AP.zoff[s]);
      const int p = AP.parent[s];
      if (p >= 0 && --left[p] == 0) live.erase(AP.zoff[p]);
    }
  }
  for (int s = 0; s < ns; ++s)
    if (!done[s]) return bad("a supernode in no wave", s);
  return true;
}

bool Engine::prepare_adjoint(std::string &err) {
  if (adj_) return true;
  if (!front_ || !front_->closed) {
    err = "adjoint: row list not closed under the elimination (invalid structure)";
    return false;
  }
  if (!prepare_tree(err)) return false;
  std::shared_ptr<AdjointPlan> plan = std::make_shared<AdjointPlan>();
  AdjointPlan &AP = *plan;
  build_adjoint_plan(hsym_, plan_, *front_, AP);
  TableUpload up;
  up.add(d_adj_parent_, AP.parent);
  up.add(d_adj_kids_, AP.kids);
  up.add(d_adj_zoff_, AP.zoff);
  up.add(d_adj_warp_, AP.warp_list);
  up.add(d_adj_cta_, AP.cta_list);
  up.add(d_adj_copies_, AP.copies);
  up.add(d_adj_tasks_, AP.tasks);
  up.add(d_adj_units_, AP.units);
  up.add(d_adj_cols_, AP.cols);
  if (!up.commit(mem_, tables_, stream_, err)) return false;
  cudaError_t e = cudaSuccess;
  const size_t scratch = sizeof(double) * TB * TB * std::max(AP.max_tasks, 1);
  if (e == cudaSuccess) e = mem_.get(d_adj_Z_, sizeof(double) * std::max<int64_t>(AP.z_len, 1));
  if (e == cudaSuccess) e = mem_.get(d_adj_UT_, scratch);
  if (e == cudaSuccess) e = mem_.get(d_adj_P_, scratch);
  if (e == cudaSuccess) e = mem_.get(d_adj_grad_, sizeof(double) * std::max<int64_t>(nnz_, 1));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_adj_small, cudaFuncAttributeMaxDynamicSharedMemorySize, ADJ_SMEM_MAX);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_adj_warp, cudaFuncAttributeMaxDynamicSharedMemorySize, ZW_WARPS * ZW_SLICE);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_adj_u, cudaFuncAttributeMaxDynamicSharedMemorySize, TT_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_adj_zrk, cudaFuncAttributeMaxDynamicSharedMemorySize, TT_SMEM);
  if (e != cudaSuccess) {
    release_adjoint();
    err = std::string("adjoint setup: ") + cudaGetErrorString(e);
    return false;
  }
  adj_ = plan;
  return true;
}

void Engine::release_adjoint() {
  for (double **p : {&d_adj_Z_, &d_adj_UT_, &d_adj_P_, &d_adj_grad_, &d_adj_partial_}) mem_.put(*p);
  if (adj_graph_) cudaGraphExecDestroy(adj_graph_);
  adj_graph_ = nullptr;
  d_adj_parent_ = d_adj_warp_ = d_adj_cta_ = nullptr;
  d_adj_kids_ = nullptr;
  d_adj_zoff_ = nullptr;
  d_adj_copies_ = d_adj_tasks_ = d_adj_units_ = nullptr;
  d_adj_cols_ = nullptr;
  adj_.reset();
}

bool Engine::logdet(double *out, std::string &err) {
  cudaSetDevice(device_);
  cudaError_t e = cudaSuccess;
  if (!d_adj_partial_) e = mem_.get(d_adj_partial_, sizeof(double) * LD_BLOCKS);
  double part[LD_BLOCKS];
  if (e == cudaSuccess) {
    k_logdet<<<LD_BLOCKS, 256, 0, stream_>>>(sym_, d_adj_partial_);
    e = cudaMemcpyAsync(part, d_adj_partial_, sizeof(part), cudaMemcpyDeviceToHost, stream_);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
  if (e != cudaSuccess) {
    err = std::string("logdet: ") + cudaGetErrorString(e);
    return false;
  }
  double s = 0.0;
  for (int i = 0; i < LD_BLOCKS; ++i) s += part[i];
  *out = 2.0 * s;
  return true;
}

// The reverse sweep's launches (fixed by the structure), gradient into d_adj_grad_.  A chain of
// short kernels: each is started early and does what L alone allows (the small fronts' inverses and
// U, the wide ones' U and T^T T) before it waits for the one ahead.
void Engine::run_adjoint() {
  const AdjointPlan &AP = *adj_;
  LaunchQueue q{stream_, false};
  const AdjDev A{d_adj_parent_, d_frel_, d_fapos_, d_adj_zoff_, d_adj_kids_,
                 d_adj_Z_,      d_adj_UT_, d_adj_P_, d_adj_grad_};
  for (const AdjointPlan::AdjWave &W : AP.waves) {
    if (W.copy_cnt > 0) launch_early(q, 1, k_adj_copy, W.copy_cnt, 256, 0, sym_, A, d_adj_copies_ + W.copy_off);
    if (W.cta_cnt > 0)
      launch_early(q, 1, k_adj_small, W.cta_cnt, ZC_T, W.cta_smem, sym_, A, d_adj_cta_ + W.cta_off);
    if (W.warp_cnt > 0)
      launch_early(q, 1, k_adj_warp, (W.warp_cnt + ZW_WARPS - 1) / ZW_WARPS, ZW_WARPS * 32, ZW_WARPS * ZW_SLICE,
                   sym_, A, d_adj_warp_ + W.warp_off, W.warp_cnt);
    for (const AdjointPlan::Step &t : W.steps) {
      if (t.task_cnt > 0) {
        launch_early(q, 1, k_adj_u, t.task_cnt, MT, TT_SMEM, sym_, A, d_adj_tasks_ + t.task_off);
        launch_early(q, 1, k_adj_zrk, t.task_cnt, MT, TT_SMEM, sym_, A, d_adj_tasks_ + t.task_off);
      }
      if (t.unit_cnt > 0)
        launch_early(q, 1, k_adj_zkk, t.unit_cnt, MT, TB * LDS * 8, sym_, A, d_adj_units_ + t.unit_off);
    }
    if (W.col_cnt > 0)
      launch_early(q, 1, k_adj_grad, (W.col_cnt * 32 + 255) / 256, 256, 0, sym_, A, d_adj_cols_ + W.col_off, W.col_cnt);
  }
}

bool Engine::logdet_grad(double *grad, std::string &err) {
  cudaSetDevice(device_);
  if (!prepare_adjoint(err)) return false;
  cudaStream_t st = stream_;
  cudaMemsetAsync(d_status_ + 1, 0, sizeof(int), st);
  cudaError_t e = cudaSuccess;
  if (use_graph_ && swept_ && !adj_graph_) {
    cudaGraph_t g = nullptr;
    e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      run_adjoint();
      e = cudaStreamEndCapture(st, &g);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&adj_graph_, g, 0);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess) {
      adj_graph_ = nullptr;
      err = std::string("logdet gradient: ") + cudaGetErrorString(e);
      return false;
    }
  }
  if (adj_graph_) e = cudaGraphLaunch(adj_graph_, st);
  else run_adjoint();
  swept_ = true;
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(grad, d_adj_grad_, sizeof(double) * nnz_, cudaMemcpyDeviceToDevice, st);
  int flag = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&flag, d_status_ + 1, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    err = std::string("logdet gradient: ") + cudaGetErrorString(e);
    return false;
  }
  if (flag) {
    err = "logdet gradient: a nonzero of A is outside the pattern of L";
    return false;
  }
  return true;
}

bool Engine::solve_grad(const double *x, const double *lam, double *grad, std::string &err) {
  cudaSetDevice(device_);
  const int blocks = (int)(((int64_t)n_ * 32 + 255) / 256);
  k_solve_grad<<<blocks, 256, 0, stream_>>>(sym_, x, lam, grad);
  cudaError_t e = cudaStreamSynchronize(stream_);
  if (e != cudaSuccess) {
    err = std::string("solve gradient: ") + cudaGetErrorString(e);
    return false;
  }
  return true;
}

}  // namespace swc
