// Supernodal triangular solves, sparse matrix-vector product and vector kernels for
// iterative refinement.  No reference counterpart for the backward solve; the forward
// solve follows the reference's layout-compatible blockedLsolve
// (triangularSolve/Triangular_BCSC.h:14-48) in gather (left-looking) form, so every
// supernode of a level runs in parallel with no atomics and a fixed summation order.
#include <cuda_runtime.h>

#include <cstdint>

#include "swc_engine.h"
#include "swc_chain.h"
#include "swc_tile.h"

namespace swc {

namespace {

constexpr int ST = 256;   // threads of the solve kernels

// Forward solve, level by level (leaves first):
//   k_fwd_small   small supernodes, one CTA each: y[cols of s] := L_ss^{-1} (y[cols of s] - sum
//                 of the contributions the descendants stored for those columns), then the
//                 contributions of its rows below, c_s = L_rs y[cols of s].  Column j's
//                 contributions are listed in cidx[cptr[j] .. cptr[j+1]) (one entry per
//                 off-diagonal row of L equal to j, in increasing supernode order).
//   k_fwd_chain, k_fwd_contrib   tiled supernodes: the chained diagonal blocks, then one CTA
//                 per slab of rows.
// c_s lives at contrib + rowptr[s] - super[s] (one entry per off-diagonal row).
// The small kernels are bound by latency: the whole panel is loaded into shared memory while the
// contributions (or the rows below) are gathered, so nothing after that waits for L, and one
// launch per level does what the diagonal solve and the contributions (backward: the gather and
// the solve) did in two: a solve of the 60^3 7-point grid 1413 -> 1301 us (B200).
// The contributions q0, q0 + step, .. < q1 of a column's list, four at a time: an index and the
// value behind it are two trips to memory, which a plain loop makes one entry after the other.
__device__ __forceinline__ double sum_contribs(const double *cr, const int *cidx, int q0, int q1, int step) {
  double acc = 0.0;
  for (int q = q0; q < q1; q += 4 * step) {
    int at[4];
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) at[u] = cidx[min(q + u * step, q1 - 1)];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = ld_if(cr + at[u], q + u * step < q1);
    acc += (v[0] + v[1]) + (v[2] + v[3]);
  }
  return acc;
}
// Four threads of one warp per column (sub = 0 .. 3): the sum in all four.
__device__ __forceinline__ double sum_contribs4(const double *cr, const int *cidx, int q0, int q1, int sub) {
  double acc = sum_contribs(cr, cidx, q0 + sub, q1, 4);
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  return acc + __shfl_xor_sync(0xffffffffu, acc, 2);
}

__device__ __forceinline__ void stage_panel(double *P, const double *Ls, int count) {
  int e = threadIdx.x;
  for (; e + 7 * ST < count; e += 8 * ST) {
    double t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = Ls[e + u * ST];
#pragma unroll
    for (int u = 0; u < 8; ++u) P[e + u * ST] = t[u];
  }
  for (; e < count; e += ST) P[e] = Ls[e];
}

// shared memory: the panel (column-major, ld m), then the right-hand side (w) and, backward, the
// gathered rows below (m - w)
static_assert(SMALL_MAX_W == 64, "two rows per lane of the solving warp");
__global__ void __launch_bounds__(ST) k_fwd_small(DevSym S, const int *list, double *y, double *contrib,
                                                  const int *cptr, const int *cidx, int n, int nrhs,
                                                  int64_t cstride) {
  extern __shared__ double P[];
  pdl_trigger();
  const int s = list[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  double *v = P + m * w;
  stage_panel(P, S.L + S.xptr[s], m * w);
  pdl_wait();
  for (int rhs = 0; rhs < nrhs; ++rhs) {
    double *yr = y + (size_t)rhs * n + f;
    double *cr = contrib + (size_t)rhs * cstride;
    // column i of s receives the contributions listed for it (descendant order)
    {
      const int i = tid >> 2;
      const int q0 = i < w ? cptr[f + i] : 0, q1 = i < w ? cptr[f + i + 1] : 0;
      const double yi = i < w ? yr[i] : 0.0, acc = sum_contribs4(cr, cidx, q0, q1, tid & 3);
      if ((tid & 3) == 0 && i < w) v[i] = yi - acc;
    }
    __syncthreads();
    if (warp == 0) {   // rows lane and lane + 32
      const int i0 = lane, i1 = lane + 32;
      double x0 = i0 < w ? v[i0] : 0.0, x1 = i1 < w ? v[i1] : 0.0;
      const double d0 = i0 < w ? 1.0 / P[i0 * m + i0] : 0.0, d1 = i1 < w ? 1.0 / P[i1 * m + i1] : 0.0;
      const int wa = min(w, 32);
      for (int j = 0; j < wa; ++j) {
        if (lane == j) x0 *= d0;
        const double xj = __shfl_sync(0xffffffffu, x0, j);
        if (i0 > j && i0 < w) x0 = fma(-P[j * m + i0], xj, x0);
        if (i1 < w) x1 = fma(-P[j * m + i1], xj, x1);
      }
      for (int j = 32; j < w; ++j) {
        if (i1 == j) x1 *= d1;
        const double xj = __shfl_sync(0xffffffffu, x1, j - 32);
        if (i1 > j && i1 < w) x1 = fma(-P[j * m + i1], xj, x1);
      }
      if (i0 < w) yr[i0] = v[i0] = x0;
      if (i1 < w) yr[i1] = v[i1] = x1;
    }
    __syncthreads();
    for (int a = w + tid; a < m; a += ST) {
      double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
      int k = 0;
      for (; k + 3 < w; k += 4) {
        a0 = fma(P[k * m + a], v[k], a0);
        a1 = fma(P[(k + 1) * m + a], v[k + 1], a1);
        a2 = fma(P[(k + 2) * m + a], v[k + 2], a2);
        a3 = fma(P[(k + 3) * m + a], v[k + 3], a3);
      }
      for (; k < w; ++k) a0 = fma(P[k * m + a], v[k], a0);
      cr[(rb - f) + (a - w)] = (a0 + a1) + (a2 + a3);
    }
    __syncthreads();
  }
}

// Contribution tasks (s, r0): rows r0 .. r0 + 31 (levels with few tasks) or r0 .. r0 + 127 of the
// off-diagonal block (r0 >= w), one CTA of CW warps: warp q sums the columns
// k = q (mod CW), lane l the rows r0 + l + 32 t, and the CW partial sums meet in shared memory in
// a fixed order.
// Bound by the bytes in flight (about 50 KB per SM keep the memory busy, and the top levels have
// one CTA per SM): sixteen predicated loads per lane are issued together, 64 KB per CTA.  With
// four at a time the ten levels of the 60^3 grid took 255 us, now 192; the gathers 224, now 197.
constexpr int CR = SOLVE_CONTRIB_ROWS, CRW = SOLVE_CONTRIB_WIDE_ROWS, CW = 16, CT = 32 * CW;
constexpr int CU = 16;   // loads of L in flight per lane
// rows r0 .. r0 + R - 1, R / 32 of them per lane, CU columns' worth of loads at a time
template <int R>
__device__ __forceinline__ void fwd_contrib_rows(const DevSym &S, int2 task, const double *y, double *contrib,
                                                 int n, int nrhs, int64_t cstride, double *part) {
  constexpr int RL = R / 32, C = CU / RL;
  const int s = task.x, r0 = task.y;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  const double *row = S.L + S.xptr[s] + r0 + lane;
  bool first = true;
  for (int rhs = 0; rhs < nrhs; ++rhs) {
    const double *yr = y + (size_t)rhs * n + f;
    double acc[RL][2];
#pragma unroll
    for (int t = 0; t < RL; ++t) acc[t][0] = acc[t][1] = 0.0;
    for (int k0 = q; k0 < w; k0 += C * CW) {
      double l[C][RL];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int k = k0 + c * CW;
#pragma unroll
        for (int t = 0; t < RL; ++t)
          l[c][t] = ld_if(row + (size_t)k * m + 32 * t, k < w && r0 + lane + 32 * t < m);
      }
      if (first) pdl_wait();
      first = false;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int k = k0 + c * CW;
        const double yk = yr[min(k, w - 1)], yc = k < w ? yk : 0.0;
#pragma unroll
        for (int t = 0; t < RL; ++t) acc[t][c & 1] = fma(l[c][t], yc, acc[t][c & 1]);
      }
    }
#pragma unroll
    for (int t = 0; t < RL; ++t) part[q * R + lane + 32 * t] = acc[t][0] + acc[t][1];
    __syncthreads();
    if ((int)threadIdx.x < R) {
      const int a = r0 + (int)threadIdx.x;
      if (a < m) {
        double t = 0.0;
#pragma unroll
        for (int g = 0; g < CW; ++g) t += part[g * R + threadIdx.x];
        contrib[(size_t)rhs * cstride + (rb - f) + (a - w)] = t;
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(CT, 2) k_fwd_contrib(DevSym S, const int2 *tasks, int nbig, const double *y,
                                                       double *contrib, int n, int nrhs, int64_t cstride) {
  __shared__ double part[CW * CRW];
  pdl_trigger();
  if ((int)blockIdx.x < nbig)
    fwd_contrib_rows<CR>(S, tasks[blockIdx.x], y, contrib, n, nrhs, cstride, part);
  else
    fwd_contrib_rows<CRW>(S, tasks[blockIdx.x], y, contrib, n, nrhs, cstride, part);
}

// Backward solve, level by level (root first):
//   k_bwd_gather  tiled supernodes: x[f + j] := x[f + j] - sum_{a >= w} L(a, j) x[rows[a]] for
//                 the columns j0..j0+15 of s (one warp per column, GU loads in flight per
//                 lane); the rows below are columns of ancestors, already solved.  Then
//                 k_bwd_chain.
//   k_bwd_small   small supernodes, one CTA each: the gather and L_ss^{-T}.
constexpr int GCH = 4096;       // gathered rows staged per chunk
constexpr int GU = 16;          // loads in flight per lane
constexpr int GT = 32 * SOLVE_GATHER_COLS;   // one warp per column of the task
__global__ void __launch_bounds__(GT, 2) k_bwd_gather(DevSym S, const int2 *tasks, double *x,
                                                      int n, int nrhs) {
  __shared__ double xg[GCH];
  const int s = tasks[blockIdx.x].x, j0 = tasks[blockIdx.x].y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const int *rows = S.Ls + rb;
  const double *Ls_s = S.L + S.xptr[s];
  const int j = j0 + warp;
  const bool own = j < w;
  pdl_trigger();
  bool first = true;
  const double *col = Ls_s + (size_t)(own ? j : j0) * m + lane;
  // every column of this CTA reads the same x[rows[a]]: gather them once per chunk, while the
  // column's first loads are under way
  for (int rhs = 0; rhs < nrhs; ++rhs) {
    double *xr = x + (size_t)rhs * n;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int a0 = w; a0 < m; a0 += GCH) {
      const int len = min(GCH, m - a0);
      double c[GU];
#pragma unroll
      for (int u = 0; u < GU; ++u) c[u] = ld_if(col + a0 + 32 * u, own && 32 * u + lane < len);
      if (first) pdl_wait();
      first = false;
      __syncthreads();
#pragma unroll 4
      for (int i = threadIdx.x; i < len; i += GT) xg[i] = xr[rows[a0 + i]];
      __syncthreads();
      for (int i = 0;;) {
#pragma unroll
        for (int u = 0; u < GU; ++u) {
          const int r = i + 32 * u + lane;
          acc[u & 3] = fma(c[u], r < len ? xg[r] : 0.0, acc[u & 3]);
        }
        i += 32 * GU;
        if (i >= len) break;
#pragma unroll
        for (int u = 0; u < GU; ++u) c[u] = ld_if(col + a0 + i + 32 * u, own && i + 32 * u + lane < len);
      }
    }
    double t = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0 && own) xr[f + j] -= t;
    __syncthreads();   // these columns are written before the next right-hand side gathers
  }
}

// ---- small supernodes (w <= SOLVE_WARP_W, at most SOLVE_WARP_ROWS rows below the diagonal
// block), one warp each, lane = column of the supernode.  Forward: the contributions the
// descendants stored for its columns, the lower solve with the diagonal block (shuffles),
// then its own contributions to the rows below (lane = row); backward: the gather from the
// ancestors' solved values (lane = column, walking the rows below), then the transposed
// solve.  Level by level like the CTA kernels; a CTA holds WPC independent warps.
constexpr int WPC = ST / 32;

__global__ void __launch_bounds__(ST) k_fwd_warp(DevSym S, const int *list, int count,
                                                 double *y, double *contrib, const int *cptr,
                                                 const int *cidx, int n, int nrhs,
                                                 int64_t cstride) {
  const int t = blockIdx.x * WPC + (threadIdx.x >> 5);
  pdl_trigger();
  pdl_wait();
  if (t >= count) return;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int s = list[t];
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const double *Ls_s = S.L + S.xptr[s];
  for (int rhs = 0; rhs < nrhs; ++rhs) {
    double *yr = y + (size_t)rhs * n;
    double *cr = contrib + (size_t)rhs * cstride;
    double v = 0.0;
    if (lane < w) {
      v = yr[f + lane] - sum_contribs(cr, cidx, cptr[f + lane], cptr[f + lane + 1], 1);
    }
    // L_ss y = v
#pragma unroll 4
    for (int j = 0; j < w; ++j) {
      const double ljj = Ls_s[(size_t)j * m + j];
      const double lij = (lane > j && lane < w) ? Ls_s[(size_t)j * m + lane] : 0.0;
      if (lane == j) v = v / ljj;
      const double yj = __shfl_sync(FULL, v, j);
      if (lane > j) v = fma(-lij, yj, v);
    }
    if (lane < w) yr[f + lane] = v;
    // contributions of the rows below: c[a] = sum_j L(a, j) y_j
    for (int a0 = w; a0 < m; a0 += 32) {
      const int a = a0 + lane;
      double acc = 0.0;
#pragma unroll 4
      for (int j = 0; j < w; ++j) {
        const double yj = __shfl_sync(FULL, v, j);
        if (a < m) acc = fma(Ls_s[(size_t)j * m + a], yj, acc);
      }
      if (a < m) cr[(rb - f) + (a - w)] = acc;
    }
  }
}

__global__ void __launch_bounds__(ST) k_bwd_warp(DevSym S, const int *list, int count, double *x,
                                                 int n, int nrhs) {
  const int t = blockIdx.x * WPC + (threadIdx.x >> 5);
  pdl_trigger();
  pdl_wait();
  if (t >= count) return;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int s = list[t];
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const int *rows = S.Ls + rb;
  const double *Ls_s = S.L + S.xptr[s];
  for (int rhs = 0; rhs < nrhs; ++rhs) {
    double *xr = x + (size_t)rhs * n;
    double v = 0.0;
    if (lane < w) {
      // x_i - sum_{a >= w} L(a, i) x[rows[a]]
      const double *col = Ls_s + (size_t)lane * m;
      double a0 = 0.0, a1 = 0.0;
      int a = w;
      for (; a + 1 < m; a += 2) {
        a0 = fma(col[a], xr[rows[a]], a0);
        a1 = fma(col[a + 1], xr[rows[a + 1]], a1);
      }
      if (a < m) a0 = fma(col[a], xr[rows[a]], a0);
      v = xr[f + lane] - (a0 + a1);
    }
    // L_ss^T x = v
#pragma unroll 4
    for (int j = w - 1; j >= 0; --j) {
      const double ljj = Ls_s[(size_t)j * m + j];
      const double lji = lane < j ? Ls_s[(size_t)lane * m + j] : 0.0;
      if (lane == j) v = v / ljj;
      const double xj = __shfl_sync(FULL, v, j);
      if (lane < j) v = fma(-lji, xj, v);
    }
    if (lane < w) xr[f + lane] = v;
  }
}

__global__ void __launch_bounds__(ST) k_bwd_small(DevSym S, const int *list, double *x, int n, int nrhs) {
  extern __shared__ double P[];
  pdl_trigger();
  const int s = list[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const int *rows = S.Ls + rb;
  double *v = P + m * w, *xg = v + w;
  stage_panel(P, S.L + S.xptr[s], m * w);
  pdl_wait();
  for (int rhs = 0; rhs < nrhs; ++rhs) {
    double *xr = x + (size_t)rhs * n;
    for (int a = w + tid; a < m; a += ST) xg[a - w] = xr[rows[a]];
    __syncthreads();
    for (int j = warp; j < w; j += ST / 32) {   // a warp per column
      const double *col = P + j * m + w;
      double a0 = 0.0, a1 = 0.0;
      int i = lane;
      for (; i + 32 < m - w; i += 64) {
        a0 = fma(col[i], xg[i], a0);
        a1 = fma(col[i + 32], xg[i + 32], a1);
      }
      if (i < m - w) a0 = fma(col[i], xg[i], a0);
      a0 += a1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
      if (lane == 0) v[j] = xr[f + j] - a0;
    }
    __syncthreads();
    if (warp == 0) {
      const int i0 = lane, i1 = lane + 32;
      double x0 = i0 < w ? v[i0] : 0.0, x1 = i1 < w ? v[i1] : 0.0;
      const double d0 = i0 < w ? 1.0 / P[i0 * m + i0] : 0.0, d1 = i1 < w ? 1.0 / P[i1 * m + i1] : 0.0;
      for (int j = w - 1; j >= 32; --j) {
        if (i1 == j) x1 *= d1;
        const double xj = __shfl_sync(0xffffffffu, x1, j - 32);
        if (i1 < j) x1 = fma(-P[i1 * m + j], xj, x1);
        x0 = fma(-P[i0 * m + j], xj, x0);
      }
      for (int j = min(w, 32) - 1; j >= 0; --j) {
        if (i0 == j) x0 *= d0;
        const double xj = __shfl_sync(0xffffffffu, x0, j);
        if (i0 < j) x0 = fma(-P[i0 * m + j], xj, x0);
      }
      if (i0 < w) xr[f + i0] = x0;
      if (i1 < w) xr[f + i1] = x1;
    }
    __syncthreads();
  }
}

// Per-block counters of the chained solves: each of a block's eight warps adds 1 (release)
// once its rows of the block's solution are in global memory, so the solution of pass e
// (the e-th chain launch that includes the block since the counters were cleared) is
// complete when the counter reaches 8e.  Waits are
// bounded: after the poll budget in status[4] a waiter records a timeout in status[2] and
// stops waiting.
constexpr int CHAIN_WARPS = ST / 32;
// ---- chained dense solves with the diagonal block of a tiled-class supernode -----------
// One CTA per 64-row block k of the diagonal block; block k consumes the solved blocks
// c < k (forward) or c > k (backward) as they arrive and applies its own block through the
// stored inverse T_k of the 64x64 diagonal block.  All CTAs of a chain are resident
// together (a few hundred at most) and only wait on CTAs with a lower blockIdx, which the
// hardware dispatches first.
//
// Warp w owns rows 8w .. 8w + 7 of the block's right-hand side v: it stages its eight rows
// of each predecessor's panel block in its own shared-memory ring (cp.async, NS slots,
// NS - 1 blocks ahead), holds them and its rows of T_k in registers, and lane
// l multiplies columns l and l + 32; a butterfly of shuffles sums the eight rows across
// the lanes (row 8w + (l >> 2) in every lane of quad l >> 2).  No block barrier until the
// last predecessor is applied; then one barrier hands v to every warp for x_k = T_k v.
// The step that waits for a predecessor's solution therefore only reads it, sixteen FMAs
// and nine shuffles.
// Ring depth: CHAIN_NS_BIG for launches that fit the GPU at one CTA per SM (long chains:
// deep prefetch), CHAIN_NS_SMALL (two CTAs per SM) for levels of many short chains.
constexpr int CHAIN_NS_BIG = 5, CHAIN_NS_SMALL = 2;
constexpr int LW = TB + 1;                      // padded row of a staged block
constexpr int CHAIN_SLOT = 8 * LW;              // one warp's eight rows
// Predecessors outside the cluster come from global memory in batches of up to CHAIN_XB
// finished blocks: their counters are polled together and their solutions loaded together
// (a lane keeps the two elements it multiplies, in its warp's batch buffer), so a batch
// costs two memory round trips instead of two per block.
constexpr int CHAIN_XB = 8;
// dynamic shared memory: the ring, then each warp's batch buffer (forward: x_c(8w .. 8w+7)
// of up to eight blocks; backward: whole x_c of up to CHAIN_XB blocks)
constexpr int CHAIN_XW_FWD = TB, CHAIN_XW_BWD = CHAIN_XB * TB;
constexpr int chain_smem(int ns, int xw) { return (ns * CHAIN_SLOT + xw) * CHAIN_WARPS * 8; }

// Chains launch in thread-block clusters of CHAIN_CL consecutive tasks.  A block publishes its
// solution through global memory and its counter (for the blocks of later clusters and the
// next level's kernels) and also writes it straight into the shared memory of the later blocks
// of its supernode in its own cluster (distributed shared memory) with st.async, whose
// transaction bytes complete the receiver's mbarrier of that sender slot: a hop inside a
// cluster neither goes through L2 nor waits for a release fence.  Slot j of a block
// receives the solution of cluster rank j (64 doubles, 512 transaction bytes, armed at
// set-up).  Every CTA of a cluster (tail padding included) passes a cluster barrier after
// the mbarrier set-up and another before it exits, so no block leaves while a remote
// write to it may be in flight.
constexpr int CHAIN_CL = 8;
struct ChainCluster {
  double yin[CHAIN_CL][TB];
  unsigned long long bar[CHAIN_CL];
};

// Lane l (holding element `row` of this block's solution when (l & 3) == 0; every lane of
// quad l >> 2 holds it) sends it to the later ranks me+1 .. last of its cluster, the four
// lanes of a quad to different ranks.
__device__ __forceinline__ void chain_send(ChainCluster &cc, int me, int last, int row, double val) {
  for (int q = me + 1 + (threadIdx.x & 3); q <= last; q += 4)
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];\n" ::"r"(
                     cluster_addr(&cc.yin[me][row], q)),
                 "d"(val), "r"(cluster_addr(&cc.bar[me], q))
                 : "memory");
}
// Sum over the lanes of a[i] (this lane's part of row 8w + i): the total of row
// 8w + ((lane >> 2) & 7), in every lane of the quad.
__device__ __forceinline__ double warp_rows8(double (&a)[8], int lane) {
  const unsigned F = 0xffffffffu;
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double o = __shfl_xor_sync(F, b4 ? a[i] : a[i + 4], 16);
    a[i] = (b4 ? a[i + 4] : a[i]) + o;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double o = __shfl_xor_sync(F, b3 ? a[i] : a[i + 2], 8);
    a[i] = (b3 ? a[i + 2] : a[i]) + o;
  }
  {
    const double o = __shfl_xor_sync(F, b2 ? a[0] : a[1], 4);
    a[0] = (b2 ? a[1] : a[0]) + o;
  }
  a[0] += __shfl_xor_sync(F, a[0], 2);
  a[0] += __shfl_xor_sync(F, a[0], 1);
  return a[0];
}

// task = (s, k); forward: y[f + 64k ..] := T_k (y[...] - contributions - sum_{c<k} L_kc x_c)
// (tasks of a supernode consecutive, in increasing k; CTAs from `count` on are padding).
// Warp w takes columns 8w .. 8w + 7 of every L_kc (eight contiguous 512-byte column pieces
// of the panel, staged by the warp alone) and keeps its partial sums of all 64 rows (rows
// l and l + 32 in lane l); the eight warps' partial sums meet once, after the last
// predecessor, and x_k = T_k v is then formed with warp w owning rows 8w .. 8w + 7.
template <int NS>
__global__ void __launch_bounds__(ST, NS == CHAIN_NS_SMALL ? 2 : 1) k_fwd_chain(DevSym S, const int2 *tasks, int count,
                                                     double *y, const double *contrib,
                                                     const int *cptr, const int *cidx, int *flags,
                                                     int epoch, int n, int64_t cstride) {
  extern __shared__ double csm[];
  __shared__ double vs[TB], part[CHAIN_WARPS][TB];
  __shared__ ChainCluster cc;
  pdl_trigger();
  cluster_bars_init(cc.bar, CHAIN_CL, TB * 8);
  const int me = (int)chain_rank();
  if ((int)blockIdx.x < count) {
    const int s = tasks[blockIdx.x].x, k = tasks[blockIdx.x].y;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, w8 = wp * 8;
    const int row = w8 + ((lane >> 2) & 7);   // the row of x_k this lane's sums belong to
    const int f = S.super[s], w = S.super[s + 1] - f;
    const int m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
    const double *P = S.L + S.xptr[s];
    const int r0 = k * TB, bw = min(TB, w - r0);
    const int nb = (w + TB - 1) / TB;
    const int base = S.dinv_off[s];
    const double *T = S.dinv + ((size_t)base + k) * (TB * TB);   // T(r, c) at T[c * 64 + r]
    // predecessors c >= cfirst are in this cluster (rank me - (k - c)); the later ranks of
    // the same supernode receive this block's solution
    const int cfirst = k - me, last = me + min(nb - 1 - k, CHAIN_CL - 1 - me);
    double *ring = csm + wp * CHAIN_SLOT;   // slot j at ring + j * CHAIN_WARPS * CHAIN_SLOT
    double *xw = csm + NS * CHAIN_WARPS * CHAIN_SLOT + wp * CHAIN_XW_FWD;
    // this warp's columns of L_kc: element (r, 8w + q) = P[(64c + 8w + q) m + r0 + r] at
    // [q * LW + r] (a warp instruction copies 32 consecutive rows of one column)
    auto stage = [&](int c) {
      if (c < k) {
        double *d = ring + (c % NS) * CHAIN_WARPS * CHAIN_SLOT;
        const double *src = P + (size_t)(c * TB + w8) * m + r0;
#pragma unroll 4
        for (int t = 0; t < 16; ++t) {
          const int e = lane + 32 * t, q = e >> 6, r = e & (TB - 1);
          const bool in = r < bw;
          cp8(d + q * LW + r, in ? src + (size_t)q * m + r : src, in);
        }
      }
      stage_commit();
    };
    for (int c = 0; c < NS - 1; ++c) stage(c);
    double tr[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      tr[i][0] = T[(size_t)lane * TB + w8 + i];
      tr[i][1] = T[(size_t)(lane + 32) * TB + w8 + i];
    }
    pdl_wait();
    // right-hand side minus the descendants' contributions (read after the last barrier)
    {
      static_assert(ST == 4 * TB, "four threads per column");
      const int i = (int)threadIdx.x >> 2, j = f + r0 + i;
      const int q0 = i < bw ? cptr[j] : 0, q1 = i < bw ? cptr[j + 1] : 0;
      const double yj = i < bw ? y[j] : 0.0, v = sum_contribs4(contrib, cidx, q0, q1, threadIdx.x & 3);
      if ((threadIdx.x & 3) == 0) vs[i] = yj - v;
    }
    double acc0 = 0.0, acc1 = 0.0;   // rows lane, lane + 32 over this warp's columns
    bool ok = true;
    int xb0 = 0, nbt = 0;            // the batch in xw: blocks xb0 .. xb0 + nbt - 1
    for (int c = 0; c < k; ++c) {
      stage(c + NS - 1);                 // into the slot freed by step c - 1
      stage_wait<NS - 1>();              // block c has landed (this lane's copies)
      __syncwarp();
      const double *Lc = ring + (c % NS) * CHAIN_WARPS * CHAIN_SLOT;
      double lr[8][2];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        lr[q][0] = Lc[q * LW + lane];
        lr[q][1] = Lc[q * LW + lane + 32];
      }
      __syncwarp();                      // the slot is refilled at step c + 1
      const double *xc;                  // x_c(8w + q) at xc[q]
      if (c >= cfirst) {   // from the cluster
        const int j = me - (k - c);
        if (!warp_bar_recv(&cc.bar[j], S.status)) { ok = false; break; }
        xc = &cc.yin[j][w8];
      } else {             // from global memory, a batch of finished blocks at a time
        if (c >= xb0 + nbt) {
          xb0 = c;
          nbt = warp_wait_prefix(&flags[base + c], 1, min(CHAIN_XB, cfirst - c), CHAIN_WARPS * epoch,
                                 S.status);
          if (nbt == 0) { ok = false; break; }
          // x_{c+u}(8w + q) into xw[u * 8 + q], lane = u * 8 + q (two rounds of four blocks)
          const int q = lane & 7, u = lane >> 3;
          const double a0 = u < nbt ? __ldcg(&y[f + (c + u) * TB + w8 + q]) : 0.0;
          const double a1 = u + 4 < nbt ? __ldcg(&y[f + (c + u + 4) * TB + w8 + q]) : 0.0;
          xw[lane] = a0;
          xw[lane + 32] = a1;
          __syncwarp();
        }
        xc = xw + (c - xb0) * 8;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const double xq = xc[q];
        acc0 = fma(lr[q][0], xq, acc0);
        acc1 = fma(lr[q][1], xq, acc1);
      }
      __syncwarp();                      // xw is rewritten by the next batch
    }
    stage_wait<0>();
    part[wp][lane] = acc0;
    part[wp][lane + 32] = acc1;
    ok = __syncthreads_and(ok) != 0;
    if (ok) {
      // v(j) for j = lane, lane + 32; then x_k = T_k v
      double x0 = vs[lane], x1 = vs[lane + 32];
#pragma unroll
      for (int g = 0; g < CHAIN_WARPS; ++g) {
        x0 -= part[g][lane];
        x1 -= part[g][lane + 32];
      }
      double a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = fma(tr[i][1], x1, tr[i][0] * x0);
      const double xk = warp_rows8(a, lane);
      // the cluster's later blocks first, then global memory and the counter
      chain_send(cc, me, last, row, row < bw ? xk : 0.0);
      if ((lane & 3) == 0 && row < bw) y[f + r0 + row] = xk;
      __syncwarp();
      if (lane == 0) red_release_add(&flags[base + k], 1);
    }
  }
  cluster_sync_all();
}

// task = (s, k) in decreasing k; backward: x[f + 64k ..] := T_k^T (x[...] - sum_{c>k} L_ck^T x_c)
// (tasks of a supernode consecutive, in decreasing k; CTAs from `count` on are padding)
template <int NS>
__global__ void __launch_bounds__(ST, NS == CHAIN_NS_SMALL ? 2 : 1) k_bwd_chain(DevSym S, const int2 *tasks, int count,
                                                  double *x, int *flags, int epoch) {
  extern __shared__ double csm[];
  __shared__ double vs[TB];
  __shared__ ChainCluster cc;
  pdl_trigger();
  cluster_bars_init(cc.bar, CHAIN_CL, TB * 8);
  const int me = (int)chain_rank();
  if ((int)blockIdx.x < count) {
    const int s = tasks[blockIdx.x].x, k = tasks[blockIdx.x].y;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, w8 = wp * 8;
    const int row = w8 + ((lane >> 2) & 7);
    const int f = S.super[s], w = S.super[s + 1] - f;
    const int m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
    const double *P = S.L + S.xptr[s];
    const int r0 = k * TB, bw = min(TB, w - r0);
    const int nb = (w + TB - 1) / TB;
    const int base = S.dinv_off[s];
    const double *T = S.dinv + ((size_t)base + k) * (TB * TB);   // T(r, c) at T[c * 64 + r]
    // successors c <= clast are in this cluster (rank me - (c - k)); the later ranks (lower
    // k) of the same supernode receive this block's solution
    const int clast = k + me, last = me + min(k, CHAIN_CL - 1 - me);
    double *ring = csm + wp * CHAIN_SLOT;
    double *xw = csm + NS * CHAIN_WARPS * CHAIN_SLOT + wp * CHAIN_XW_BWD;
    // successor step t = nb - 1 - c (c = nb - 1 first); this warp's columns of block (c, k):
    // element (i, rr) = P[(r0 + w8 + i) m + 64c + rr] at [i * LW + rr]
    auto stage = [&](int t) {
      const int c = nb - 1 - t;
      if (c > k) {
        double *d = ring + (t % NS) * CHAIN_WARPS * CHAIN_SLOT;
        const int cw = min(TB, w - c * TB);
        const double *src = P + (size_t)(r0 + w8) * m + c * TB;
#pragma unroll 4
        for (int u = 0; u < 16; ++u) {
          const int e = lane + 32 * u, i = e >> 6, rr = e & 63;
          const bool in = w8 + i < bw && rr < cw;
          cp8(d + i * LW + rr, in ? src + (size_t)i * m + rr : src, in);
        }
      }
      stage_commit();
    };
    for (int t = 0; t < NS - 1; ++t) stage(t);
    double tr[8][2];   // T(rr, w8 + i) for rr = lane, lane + 32
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      tr[i][0] = T[(size_t)(w8 + i) * TB + lane];
      tr[i][1] = T[(size_t)(w8 + i) * TB + lane + 32];
    }
    pdl_wait();
    double v = (row < bw) ? x[f + r0 + row] : 0.0;
    bool ok = true;
    int xb0 = nb, nbt = 0;               // the batch in xw: blocks xb0, .., xb0 - nbt + 1
    for (int c = nb - 1; c > k; --c) {
      const int t = nb - 1 - c;
      stage(t + NS - 1);
      stage_wait<NS - 1>();              // block (c, k) has landed (this lane's copies)
      __syncwarp();
      const double *Lc = ring + (t % NS) * CHAIN_WARPS * CHAIN_SLOT;
      double lr[8][2];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        lr[i][0] = Lc[i * LW + lane];
        lr[i][1] = Lc[i * LW + lane + 32];
      }
      __syncwarp();
      double x0, x1;
      if (c <= clast) {   // from the cluster
        const int j = me - (c - k);
        if (!warp_bar_recv(&cc.bar[j], S.status)) { ok = false; break; }
        x0 = cc.yin[j][lane];
        x1 = cc.yin[j][lane + 32];
      } else {            // from global memory, a batch of blocks c, c - 1, .. at a time
        if (c <= xb0 - nbt) {
          xb0 = c;                         // blocks c, c - 1, .., c - nbt + 1
          nbt = warp_wait_prefix(&flags[base + c], -1, min(CHAIN_XB, c - clast), CHAIN_WARPS * epoch,
                                 S.status);
          if (nbt == 0) { ok = false; break; }
          double t2[CHAIN_XB][2];
#pragma unroll
          for (int u = 0; u < CHAIN_XB; ++u)
            if (u < nbt) {
              const int cu = c - u, cwu = min(TB, w - cu * TB);
              t2[u][0] = lane < cwu ? __ldcg(&x[f + cu * TB + lane]) : 0.0;
              t2[u][1] = lane + 32 < cwu ? __ldcg(&x[f + cu * TB + lane + 32]) : 0.0;
            }
#pragma unroll
          for (int u = 0; u < CHAIN_XB; ++u)
            if (u < nbt) {
              xw[u * TB + lane] = t2[u][0];
              xw[u * TB + lane + 32] = t2[u][1];
            }
        }
        x0 = xw[(xb0 - c) * TB + lane];   // written by this lane
        x1 = xw[(xb0 - c) * TB + lane + 32];
      }
      double a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = fma(lr[i][1], x1, lr[i][0] * x0);
      v -= warp_rows8(a, lane);
    }
    stage_wait<0>();
    if ((lane & 3) == 0) vs[row] = v;
    ok = __syncthreads_and(ok) != 0;
    if (ok) {
      // x_k[i] = sum_rr T(rr, i) v[rr]
      const double x0 = vs[lane], x1 = vs[lane + 32];
      double a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = fma(tr[i][1], x1, tr[i][0] * x0);
      const double xk = warp_rows8(a, lane);
      chain_send(cc, me, last, row, row < bw ? xk : 0.0);
      if ((lane & 3) == 0 && row < bw) x[f + r0 + row] = xk;
      __syncwarp();
      if (lane == 0) red_release_add(&flags[base + k], 1);
    }
  }
  cluster_sync_all();
}

// y = A x, or b - A x where b is given, for the symmetric matrix held as full CSR (both triangles).
// Eight lanes per row (rows of a stencil matrix hold 7 to 81 entries) and four rows per group of
// eight lanes at the same time: bound by the trips to memory (row pointers, entries, x), and most
// rows are over after one or two steps.
__global__ void __launch_bounds__(256) k_spmv(int n, const int *rp, const int *ci, const double *val,
                                              const double *x, const double *b, double *y) {
  constexpr int RW = 4;
  const int row0 = (blockIdx.x * 32 + (int)(threadIdx.x >> 3)) * RW;
  const int sub = threadIdx.x & 7;
  int p0[RW], p1[RW], longest = 0;
#pragma unroll
  for (int i = 0; i < RW; ++i) {
    p0[i] = rp[min(row0 + i, n)];
    p1[i] = rp[min(row0 + i + 1, n)];
    longest = max(longest, p1[i] - p0[i]);
  }
  double acc[RW] = {0.0, 0.0, 0.0, 0.0};
  for (int q = sub; q < longest; q += 8) {
    double v[RW];
    int c[RW];
#pragma unroll
    for (int i = 0; i < RW; ++i) {
      v[i] = ld_if(val + p0[i] + q, p0[i] + q < p1[i]);
      c[i] = p0[i] + q < p1[i] ? ci[p0[i] + q] : -1;
    }
#pragma unroll
    for (int i = 0; i < RW; ++i) acc[i] = fma(v[i], ld_if(x + c[i], c[i] >= 0), acc[i]);
  }
#pragma unroll
  for (int i = 0; i < RW; ++i) {
    double t = acc[i];
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    if (row0 + i < n && sub == 0) y[row0 + i] = b ? b[row0 + i] - t : t;
  }
}

// The same for nr <= 8 vectors, x interleaved by eight: lane u of a group takes vector u, so an
// entry costs one 64-byte piece of x instead of eight pieces of as many vectors; the group's lanes
// load eight entries and pass them around (the next eight on the way).  36 x 35 x 33 elastic operator,
// eight vectors: 85 + 5 us (product by vectors, then the difference) -> 72 + 4 (interleaving).
__global__ void __launch_bounds__(256) k_spmv8(int n, const int *rp, const int *ci, const double *val,
                                               const double *x8, const double *b, double *y, int nr) {
  const int row = blockIdx.x * 32 + (int)(threadIdx.x >> 3), u = threadIdx.x & 7;
  const int p0 = rp[min(row, n)], p1 = rp[min(row + 1, n)];
  const int steps = __reduce_max_sync(0xffffffffu, (p1 - p0 + 7) >> 3);
  double a0 = 0.0, a1 = 0.0;
  double vn = ld_if(val + p0 + u, p0 + u < p1);   // the next step's entries
  int cn = p0 + u < p1 ? ci[p0 + u] : -1;
  for (int t = 0; t < steps; ++t) {
    const int p = p0 + 8 * (t + 1) + u, c = cn;
    const double v = vn;
    vn = ld_if(val + p, p < p1);
    cn = p < p1 ? ci[p] : -1;
    double xv[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int ck = __shfl_sync(0xffffffffu, c, k, 8);
      xv[k] = ld_if(x8 + (int64_t)ck * 8 + u, ck >= 0);
    }
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      a0 = fma(__shfl_sync(0xffffffffu, v, k, 8), xv[k], a0);
      a1 = fma(__shfl_sync(0xffffffffu, v, k + 1, 8), xv[k + 1], a1);
    }
  }
  if (row < n && u < nr) {
    const size_t at = (size_t)u * n + row;
    y[at] = b ? b[at] - (a0 + a1) : a0 + a1;
  }
}

// out[i] = sum_j |A(i, j)| (rows of the full CSR)
__global__ void k_rowabs(int n, const int *rp, const double *val, double *out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double acc = 0.0;
  for (int p = rp[i]; p < rp[i + 1]; ++p) acc += fabs(val[p]);
  out[i] = acc;
}

// full-CSR values from the lower-CSC values through the precomputed map
__global__ void k_gather_vals(int nnz, const int *map, const double *ax, double *val) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nnz) val[i] = ax[map[i]];
}

// p = z + beta p
__global__ void k_xpby(size_t len, const double *z, double beta, double *p) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < len) p[i] = fma(beta, p[i], z[i]);
}

__global__ void k_axpy(size_t len, double a, const double *x, double *y) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < len) y[i] = fma(a, x[i], y[i]);
}

// per-vector max |x| and sum x*y for nrhs vectors of length n (out[2*r], out[2*r+1]), then (x2 given)
// max |x2| of as many more,
// deterministic: NORM_BLOCKS fixed slices per vector, then one CTA per vector sums the
// slices in order.
constexpr int NORM_BLOCKS = 128;
__global__ void k_norms_part(int n, int nrhs, const double *x, const double *y, const double *x2, double *part) {
  __shared__ double smax[ST], sdot[ST];
  const int r = blockIdx.y, b = blockIdx.x;
  const double *xr = r < nrhs ? x + (size_t)r * n : x2 + (size_t)(r - nrhs) * n;
  const double *yr = y && r < nrhs ? y + (size_t)r * n : nullptr;
  const int per = (n + NORM_BLOCKS - 1) / NORM_BLOCKS;
  const int lo = b * per, hi = min(n, lo + per);
  double mx = 0.0, dt = 0.0;
  for (int i = lo + threadIdx.x; i < hi; i += ST) {
    mx = fmax(mx, fabs(xr[i]));
    if (yr) dt = fma(xr[i], yr[i], dt);
  }
  smax[threadIdx.x] = mx;
  sdot[threadIdx.x] = dt;
  __syncthreads();
  for (int o = ST / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + o]);
      sdot[threadIdx.x] += sdot[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * ((size_t)r * NORM_BLOCKS + b)] = smax[0];
    part[2 * ((size_t)r * NORM_BLOCKS + b) + 1] = sdot[0];
  }
}
__global__ void k_norms_final(const double *part, double *out) {
  __shared__ double smax[NORM_BLOCKS], sdot[NORM_BLOCKS];
  const int r = blockIdx.x, t = threadIdx.x;
  smax[t] = part[2 * ((size_t)r * NORM_BLOCKS + t)];
  sdot[t] = part[2 * ((size_t)r * NORM_BLOCKS + t) + 1];
  __syncthreads();
  for (int o = NORM_BLOCKS / 2; o > 0; o >>= 1) {
    if (t < o) {
      smax[t] = fmax(smax[t], smax[t + o]);
      sdot[t] += sdot[t + o];
    }
    __syncthreads();
  }
  if (t == 0) {
    out[2 * r] = smax[0];
    out[2 * r + 1] = sdot[0];
  }
}

}  // namespace

// the chains' grids: whole clusters of CHAIN_CL CTAs; launches that fit the SMs at one CTA each take
// the deep ring, which fills an SM's shared memory; beside the other half of the tree, those that
// leave it half of the SMs (solve of the 60^3 grid: all SMs 1049 us, half 1027, none 1072)
static int g_num_sms = 148;
static int chain_grid(int count) { return (count + CHAIN_CL - 1) / CHAIN_CL * CHAIN_CL; }

bool solve_configure(int max_w, std::string &err) {
  size_t smem = sizeof(double) * (size_t)(max_w > 0 ? max_w : 1);
  if (smem > 220 * 1024) {
    err = "supernode too wide for the shared-memory triangular solve";
    return false;
  }
  cudaError_t e = cudaFuncSetAttribute(k_fwd_small, cudaFuncAttributeMaxDynamicSharedMemorySize, SOLVE_SMALL_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_fwd_chain<CHAIN_NS_BIG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             chain_smem(CHAIN_NS_BIG, CHAIN_XW_FWD));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_fwd_chain<CHAIN_NS_SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             chain_smem(CHAIN_NS_SMALL, CHAIN_XW_FWD));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_bwd_chain<CHAIN_NS_BIG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             chain_smem(CHAIN_NS_BIG, CHAIN_XW_BWD));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_bwd_chain<CHAIN_NS_SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             chain_smem(CHAIN_NS_SMALL, CHAIN_XW_BWD));
  if (e == cudaSuccess) {
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_bwd_small, cudaFuncAttributeMaxDynamicSharedMemorySize, SOLVE_SMALL_SMEM);
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return false;
  }
  return true;
}

void launch_fwd_small(const DevSym &S, const int *list, int count, int smem, double *y,
                      double *contrib, const int *cptr, const int *cidx, int n, int nrhs,
                      int64_t cstride, LaunchQueue &st) {
  if (count > 0)
    launch_early(st, 1, k_fwd_small, count, ST, smem, S, list, y, contrib, cptr, cidx, n, nrhs, cstride);
}
void launch_fwd_contrib(const DevSym &S, const int2 *tasks, int count, int nbig, const double *y,
                        double *contrib, int n, int nrhs, int64_t cstride, LaunchQueue &st) {
  if (count > 0)
    launch_early(st, 1, k_fwd_contrib, count, CT, 0, S, tasks, nbig, y, contrib, n, nrhs, cstride);
}
void launch_fwd_warp(const DevSym &S, const int *list, int count, double *y, double *contrib,
                     const int *cptr, const int *cidx, int n, int nrhs, int64_t cstride,
                     LaunchQueue &st) {
  if (count > 0)
    launch_early(st, 1, k_fwd_warp, (count + WPC - 1) / WPC, ST, 0, S, list, count, y, contrib, cptr, cidx,
                 n, nrhs, cstride);
}
void launch_bwd_warp(const DevSym &S, const int *list, int count, double *x, int n, int nrhs,
                     LaunchQueue &st) {
  if (count > 0)
    launch_early(st, 1, k_bwd_warp, (count + WPC - 1) / WPC, ST, 0, S, list, count, x, n, nrhs);
}
void launch_bwd_gather(const DevSym &S, const int2 *tasks, int count, double *x, int n, int nrhs,
                       LaunchQueue &st) {
  if (count > 0) launch_early(st, 1, k_bwd_gather, count, GT, 0, S, tasks, x, n, nrhs);
}
void launch_bwd_small(const DevSym &S, const int *list, int count, int smem, double *x, int n,
                      int nrhs, LaunchQueue &st) {
  if (count > 0) launch_early(st, 1, k_bwd_small, count, ST, smem, S, list, x, n, nrhs);
}
void launch_fwd_chain(const DevSym &S, const int2 *tasks, int count, double *y,
                      const double *contrib, const int *cptr, const int *cidx, int *flags,
                      int epoch, int n, int64_t cstride, bool beside, LaunchQueue &st) {
  if (count <= 0) return;
  const int grid = chain_grid(count);
  if (grid <= (beside ? g_num_sms / 2 : g_num_sms))
    launch_early(st, CHAIN_CL, k_fwd_chain<CHAIN_NS_BIG>, grid, ST, chain_smem(CHAIN_NS_BIG, CHAIN_XW_FWD), S,
                 tasks, count, y, contrib, cptr, cidx, flags, epoch, n, cstride);
  else
    launch_early(st, CHAIN_CL, k_fwd_chain<CHAIN_NS_SMALL>, grid, ST, chain_smem(CHAIN_NS_SMALL, CHAIN_XW_FWD), S,
                 tasks, count, y, contrib, cptr, cidx, flags, epoch, n, cstride);
}
void launch_bwd_chain(const DevSym &S, const int2 *tasks, int count, double *x, int *flags,
                      int epoch, bool beside, LaunchQueue &st) {
  if (count <= 0) return;
  const int grid = chain_grid(count);
  if (grid <= (beside ? g_num_sms / 2 : g_num_sms))
    launch_early(st, CHAIN_CL, k_bwd_chain<CHAIN_NS_BIG>, grid, ST, chain_smem(CHAIN_NS_BIG, CHAIN_XW_BWD), S,
                 tasks, count, x, flags, epoch);
  else
    launch_early(st, CHAIN_CL, k_bwd_chain<CHAIN_NS_SMALL>, grid, ST, chain_smem(CHAIN_NS_SMALL, CHAIN_XW_BWD), S,
                 tasks, count, x, flags, epoch);
}
void launch_spmv(int n, const int *rp, const int *ci, const double *val, const double *x, const double *b,
                 double *y, cudaStream_t st) {
  k_spmv<<<(n + 127) / 128, 256, 0, st>>>(n, rp, ci, val, x, b, y);
}
void launch_spmv8(int n, const int *rp, const int *ci, const double *val, const double *x8, const double *b,
                  double *y, int nr, cudaStream_t st) {
  k_spmv8<<<(n + 31) / 32, 256, 0, st>>>(n, rp, ci, val, x8, b, y, nr);
}
void launch_gather_vals(int nnz, const int *map, const double *ax, double *val, cudaStream_t st) {
  if (nnz > 0) k_gather_vals<<<(nnz + 255) / 256, 256, 0, st>>>(nnz, map, ax, val);
}
void launch_rowabs(int n, const int *rp, const double *val, double *out, cudaStream_t st) {
  k_rowabs<<<(n + 255) / 256, 256, 0, st>>>(n, rp, val, out);
}
void launch_xpby(size_t len, const double *z, double beta, double *p, cudaStream_t st) {
  if (len) k_xpby<<<(unsigned)((len + 255) / 256), 256, 0, st>>>(len, z, beta, p);
}
void launch_axpy(size_t len, double a, const double *x, double *y, cudaStream_t st) {
  if (len) k_axpy<<<(unsigned)((len + 255) / 256), 256, 0, st>>>(len, a, x, y);
}
void launch_norms(int n, int nrhs, const double *x, const double *y, const double *x2, double *out, double *part,
                  cudaStream_t st) {
  const int sets = x2 ? 2 * nrhs : nrhs;
  k_norms_part<<<dim3(NORM_BLOCKS, sets), ST, 0, st>>>(n, nrhs, x, y, x2, part);
  k_norms_final<<<sets, NORM_BLOCKS, 0, st>>>(part, out);
}
int norm_scratch_doubles(int nrhs) { return 4 * NORM_BLOCKS * nrhs; }

}  // namespace swc
