// Triangular solves of up to eight right-hand sides at a time.  The vectors are interleaved
// (x8[i * 8 + r]), so every gather of a row brings all right-hand sides in one 64-byte piece,
// L is read once for all of them, and every block product is an FP64 tensor-core product with
// N = 8 (DMMA m8n8k4: A 8 rows of L, B 4 rows x 8 right-hand sides).  Bound: the chain of
// dependent blocks and levels (one for all right-hand sides instead of one each), then the two
// passes over L.  Against one pass per right-hand side (B200, 8 right-hand sides): a solve of a
// 301 x 287 5-point grid 2152 -> 496 us, of a 36 x 35 x 33 3-unknown 27-point grid (L 1.15 GB)
// about 7.0 -> 2.0 ms.  Two to seven right-hand sides take the same pass with zero columns.
//
// Forward, level by level (leaves first): small supernodes take the contributions of their
// descendants, solve with their diagonal block and form the contributions of their rows below
// in one kernel (a warp or a CTA each); tiled ones are solved by the chained blocks and form
// their contributions in a second kernel.  Backward: the mirror image.
//
// A right-hand side's result does not depend on the others of its group, nor on its place among
// them (a tensor-core product's columns are independent).  The kernels come with the vectors
// interleaved by R = 8, and by 4, 2 and 1 (a plain vector) with zero columns for the others: the same
// result bit for bit, for callers whose scratch has no room for eight.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "swc_chain.h"
#include "swc_engine.h"
#include "swc_tile.h"

namespace swc {

namespace {

constexpr int R8 = 8;
constexpr int NT8 = 256, W8 = NT8 / 32;

// Element e (row e / 8, right-hand side e % 8) in vectors interleaved by R: its place, and its value,
// zero where there is none.
template <int R>
__device__ __forceinline__ int place8(int e) {
  return R == R8 ? e : (e >> 3) * R + (e & 7);
}
template <int R>
__device__ __forceinline__ double at8(const double *x, int e) {
  return R == R8 || (e & 7) < R ? x[place8<R>(e)] : 0.0;
}
// Right-hand side r of row i; zero where there is none.
template <int R>
__device__ __forceinline__ double rhs_of(const double *x, int64_t i, int r) {
  return r < R ? x[i * R + r] : 0.0;
}

// Right-hand sides 2 kq, 2 kq + 1 of a row.
template <int R>
__device__ __forceinline__ void store_pair(double *row, int kq, double a, double b) {
  if (R == 1 && kq == 0) row[0] = a;
  if (R > 1 && 2 * kq < R) *reinterpret_cast<double2 *>(row + 2 * kq) = make_double2(a, b);
}

// v - sum of the contributions listed for column j, right-hand side r.
template <int R>
__device__ __forceinline__ double take_contribs(const double *c8, const int *cptr, const int *cidx,
                                                int j, int r, double v) {
  const int q1 = cptr[j + 1];
  for (int q = cptr[j]; q < q1; q += 4) {
    int at[4];
    double t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) at[u] = cidx[min(q + u, q1 - 1)];
#pragma unroll
    for (int u = 0; u < 4; ++u) t[u] = ld_if(c8 + (size_t)at[u] * R + r, q + u < q1 && r < R);
    v -= (t[0] + t[1]) + (t[2] + t[3]);
  }
  return v;
}

// Contributions of rows a0 .. a0 + 7 of supernode s: L(a, 0 .. w - 1) y, y in shared memory
// ([column][right-hand side]).
template <int R>
__device__ __forceinline__ void contrib_rows8(const double *Ls, int m, int w, int a0, const double *v,
                                              double *out) {
  const int lane = threadIdx.x & 31, g = lane >> 2, kq = lane & 3;
  const int a = a0 + g;
  const bool in = a < m;
  const double *col = Ls + (in ? a : 0);
  double c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
  for (int k = 0; k < w; k += 16) {
    double l[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) l[u] = ld_if(col + (size_t)(k + 4 * u + kq) * m, in && k + 4 * u + kq < w);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = k + 4 * u + kq;
      if (k + 4 * u < w) dmma(u & 1 ? c1 : c0, l[u], c < w ? v[c * R8 + g] : 0.0);
    }
  }
  if (in) store_pair<R>(out + (size_t)(a - w) * R, kq, c0[0] + c1[0], c0[1] + c1[1]);
}

// ---- small supernodes (w <= SMALL_MAX_W), one CTA each; warp r solves right-hand side r with
// lanes as rows (row lane and lane + 32), everything else is shared by the CTA.
constexpr int LDW = SMALL_MAX_W + 1;
constexpr int SMALL8_SMEM = (SMALL_MAX_W * LDW + SMALL_MAX_W * R8) * 8;
static_assert(SMALL_MAX_W == 64 && W8 == R8, "two rows per lane, a warp per right-hand side");
static_assert(W8 * SMALL_MAX_W * R8 <= SMALL_MAX_W * LDW, "partial sums fit the block's place");

__device__ __forceinline__ void stage_block(double *Ld, const double *Ls, int m, int w) {
  for (int e = threadIdx.x; e < w * w; e += NT8) {
    const int j = e / w, i = e - j * w;
    if (i >= j) Ld[j * LDW + i] = Ls[(size_t)j * m + i];
  }
}

template <int R>
__global__ void __launch_bounds__(NT8) k_fwd_small8(DevSym S, const int *list, double *y8, double *c8,
                                                    const int *cptr, const int *cidx) {
  extern __shared__ double sm8[];
  pdl_trigger();
  double *Ld = sm8, *v = sm8 + SMALL_MAX_W * LDW;   // v[column][rhs]
  const int s = list[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const double *Ls = S.L + S.xptr[s];
  stage_block(Ld, Ls, m, w);
  pdl_wait();
  for (int e = tid; e < w * R8; e += NT8)
    v[e] = take_contribs<R>(c8, cptr, cidx, f + (e >> 3), e & 7, at8<R>(y8 + (size_t)f * R, e));
  __syncthreads();
  {
    const int i0 = lane, i1 = lane + 32;
    double x0 = i0 < w ? v[i0 * R8 + warp] : 0.0, x1 = i1 < w ? v[i1 * R8 + warp] : 0.0;
    const double d0 = i0 < w ? 1.0 / Ld[i0 * LDW + i0] : 0.0, d1 = i1 < w ? 1.0 / Ld[i1 * LDW + i1] : 0.0;
    const int wa = min(w, 32);
    for (int j = 0; j < wa; ++j) {
      if (lane == j) x0 *= d0;
      const double xj = __shfl_sync(0xffffffffu, x0, j);
      if (i0 > j && i0 < w) x0 = fma(-Ld[j * LDW + i0], xj, x0);
      if (i1 < w) x1 = fma(-Ld[j * LDW + i1], xj, x1);
    }
    for (int j = 32; j < w; ++j) {
      if (i1 == j) x1 *= d1;
      const double xj = __shfl_sync(0xffffffffu, x1, j - 32);
      if (i1 > j && i1 < w) x1 = fma(-Ld[j * LDW + i1], xj, x1);
    }
    if (i0 < w) v[i0 * R8 + warp] = x0;
    if (i1 < w) v[i1 * R8 + warp] = x1;
  }
  __syncthreads();
  for (int e = tid; e < w * R8; e += NT8)
    if ((e & 7) < R) y8[(size_t)f * R + place8<R>(e)] = v[e];
  double *out = c8 + (size_t)(rb - f) * R;
  for (int a0 = w + 8 * warp; a0 < m; a0 += 8 * W8) contrib_rows8<R>(Ls, m, w, a0, v, out);
}

template <int R>
__global__ void __launch_bounds__(NT8) k_bwd_small8(DevSym S, const int *list, double *x8) {
  extern __shared__ double sm8[];
  pdl_trigger();
  double *Ld = sm8, *v = sm8 + SMALL_MAX_W * LDW;
  const int s = list[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, kq = lane & 3;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const int *rows = S.Ls + rb;
  const double *Ls = S.L + S.xptr[s];
  // sum over the rows below of L(a, j) x[rows[a]]: warps take four rows at a time, eight
  // columns per product
  const int nt = (w + 7) >> 3;
  pdl_wait();
  double c[SMALL_MAX_W / 8][2];
#pragma unroll
  for (int i = 0; i < SMALL_MAX_W / 8; ++i) c[i][0] = c[i][1] = 0.0;
  for (int a0 = w + 4 * warp; a0 < m; a0 += 4 * W8) {
    const int a = a0 + kq;
    const bool in = a < m;
    double l[SMALL_MAX_W / 8];
#pragma unroll
    for (int i = 0; i < SMALL_MAX_W / 8; ++i) l[i] = ld_if(Ls + (size_t)(8 * i + g) * m + a, in && 8 * i + g < w);
    const double b = ld_if(x8 + (size_t)rows[in ? a : 0] * R + g, in && g < R);
#pragma unroll
    for (int i = 0; i < SMALL_MAX_W / 8; ++i)
      if (i < nt) dmma(c[i], l[i], b);
  }
  double *part = sm8;   // [warp][column][rhs], before the diagonal block is staged
#pragma unroll
  for (int i = 0; i < SMALL_MAX_W / 8; ++i)
    if (i < nt)
      *reinterpret_cast<double2 *>(part + (size_t)(warp * SMALL_MAX_W + 8 * i + g) * R8 + 2 * kq) =
          make_double2(c[i][0], c[i][1]);
  __syncthreads();
  for (int e = tid; e < w * R8; e += NT8) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < W8; ++q) t += part[q * SMALL_MAX_W * R8 + e];
    v[e] = at8<R>(x8 + (size_t)f * R, e) - t;
  }
  __syncthreads();
  stage_block(Ld, Ls, m, w);
  __syncthreads();
  {
    const int i0 = lane, i1 = lane + 32;
    double x0 = i0 < w ? v[i0 * R8 + warp] : 0.0, x1 = i1 < w ? v[i1 * R8 + warp] : 0.0;
    const double d0 = i0 < w ? 1.0 / Ld[i0 * LDW + i0] : 0.0, d1 = i1 < w ? 1.0 / Ld[i1 * LDW + i1] : 0.0;
    for (int j = w - 1; j >= 32; --j) {
      if (i1 == j) x1 *= d1;
      const double xj = __shfl_sync(0xffffffffu, x1, j - 32);
      if (i1 < j) x1 = fma(-Ld[i1 * LDW + j], xj, x1);
      x0 = fma(-Ld[i0 * LDW + j], xj, x0);
    }
    for (int j = min(w, 32) - 1; j >= 0; --j) {
      if (i0 == j) x0 *= d0;
      const double xj = __shfl_sync(0xffffffffu, x0, j);
      if (i0 < j) x0 = fma(-Ld[i0 * LDW + j], xj, x0);
    }
    if (i0 < w) v[i0 * R8 + warp] = x0;
    if (i1 < w) v[i1 * R8 + warp] = x1;
  }
  __syncthreads();
  for (int e = tid; e < w * R8; e += NT8)
    if ((e & 7) < R) x8[(size_t)f * R + place8<R>(e)] = v[e];
}

// ---- the small supernodes of crowded levels (w <= SOLVE_WARP_W), one warp each: lane (r, q)
// owns rows q, q + 4, .. of right-hand side r.
constexpr int WN = 4, LDT = SOLVE_WARP_W + 1, NX = SOLVE_WARP_W / 4;
struct Warp8 {
  double L[SOLVE_WARP_W * LDT];
  double v[SOLVE_WARP_W * R8];
};

__device__ __forceinline__ void stage_block_warp(Warp8 &M, const double *Ls, int m, int w, int lane) {
  for (int j = 0; j < w; ++j)
    if (lane >= j && lane < w) M.L[j * LDT + lane] = Ls[(size_t)j * m + lane];
}

template <int R>
__global__ void __launch_bounds__(WN * 32) k_fwd_warp8(DevSym S, const int *list, int count, double *y8,
                                                       double *c8, const int *cptr, const int *cidx) {
  __shared__ Warp8 sm[WN];
  const int t = blockIdx.x * WN + (threadIdx.x >> 5);
  pdl_trigger();
  pdl_wait();
  if (t >= count) return;
  Warp8 &M = sm[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, r = lane & 7, q = lane >> 3;
  const int s = list[t];
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const double *Ls = S.L + S.xptr[s];
  stage_block_warp(M, Ls, m, w, lane);
  double x[NX], d[NX];
#pragma unroll
  for (int u = 0; u < NX; ++u) {
    const int i = 4 * u + q;
    x[u] = i < w ? take_contribs<R>(c8, cptr, cidx, f + i, r, rhs_of<R>(y8, f + i, r)) : 0.0;
  }
  __syncwarp();
#pragma unroll
  for (int u = 0; u < NX; ++u) d[u] = 4 * u + q < w ? 1.0 / M.L[(4 * u + q) * LDT + 4 * u + q] : 0.0;
#pragma unroll
  for (int u = 0; u < NX; ++u)
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int j = 4 * u + p;
      if (j < w) {
        if (q == p) x[u] *= d[u];
        const double xj = __shfl_sync(0xffffffffu, x[u], 8 * p + r);
#pragma unroll
        for (int z = u; z < NX; ++z) {
          const int i = 4 * z + q;
          if (i > j && i < w) x[z] = fma(-M.L[j * LDT + i], xj, x[z]);
        }
      }
    }
#pragma unroll
  for (int u = 0; u < NX; ++u) {
    const int i = 4 * u + q;
    if (i < w) {
      M.v[i * R8 + r] = x[u];
      if (r < R) y8[(size_t)(f + i) * R + r] = x[u];
    }
  }
  __syncwarp();
  double *out = c8 + (size_t)(rb - f) * R;
  for (int a0 = w; a0 < m; a0 += 8) contrib_rows8<R>(Ls, m, w, a0, M.v, out);
}

template <int R>
__global__ void __launch_bounds__(WN * 32) k_bwd_warp8(DevSym S, const int *list, int count, double *x8) {
  __shared__ Warp8 sm[WN];
  const int t = blockIdx.x * WN + (threadIdx.x >> 5);
  pdl_trigger();
  pdl_wait();
  if (t >= count) return;
  Warp8 &M = sm[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, r = lane & 7, q = lane >> 3, g = lane >> 2, kq = lane & 3;
  const int s = list[t];
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const int *rows = S.Ls + rb;
  const double *Ls = S.L + S.xptr[s];
  stage_block_warp(M, Ls, m, w, lane);
  const int nt = (w + 7) >> 3;
  double c[SOLVE_WARP_W / 8][2];
#pragma unroll
  for (int i = 0; i < SOLVE_WARP_W / 8; ++i) c[i][0] = c[i][1] = 0.0;
#pragma unroll 2
  for (int a0 = w; a0 < m; a0 += 4) {
    const int a = a0 + kq;
    const bool in = a < m;
    double l[SOLVE_WARP_W / 8];
#pragma unroll
    for (int i = 0; i < SOLVE_WARP_W / 8; ++i) l[i] = ld_if(Ls + (size_t)(8 * i + g) * m + a, in && 8 * i + g < w);
    const double b = ld_if(x8 + (size_t)rows[in ? a : 0] * R + g, in && g < R);
#pragma unroll
    for (int i = 0; i < SOLVE_WARP_W / 8; ++i)
      if (i < nt) dmma(c[i], l[i], b);
  }
#pragma unroll
  for (int i = 0; i < SOLVE_WARP_W / 8; ++i)
    if (i < nt)
      *reinterpret_cast<double2 *>(M.v + (8 * i + g) * R8 + 2 * kq) = make_double2(c[i][0], c[i][1]);
  __syncwarp();
  double x[NX], d[NX];
#pragma unroll
  for (int u = 0; u < NX; ++u) {
    const int i = 4 * u + q;
    x[u] = i < w ? rhs_of<R>(x8, f + i, r) - M.v[i * R8 + r] : 0.0;
    d[u] = i < w ? 1.0 / M.L[i * LDT + i] : 0.0;
  }
#pragma unroll
  for (int u = NX - 1; u >= 0; --u)
#pragma unroll
    for (int p = 3; p >= 0; --p) {
      const int j = 4 * u + p;
      if (j < w) {
        if (q == p) x[u] *= d[u];
        const double xj = __shfl_sync(0xffffffffu, x[u], 8 * p + r);
#pragma unroll
        for (int z = 0; z <= u; ++z) {
          const int i = 4 * z + q;
          if (i < j) x[z] = fma(-M.L[i * LDT + j], xj, x[z]);
        }
      }
    }
#pragma unroll
  for (int u = 0; u < NX; ++u) {
    const int i = 4 * u + q;
    if (i < w && r < R) x8[(size_t)(f + i) * R + r] = x[u];
  }
}

// ---- contributions of tiled supernodes.  Levels with at least one 128-row task per SM: 128
// rows per CTA, warp q forms rows 16 q .. 16 q + 15 over all columns; other levels: 32 rows
// per CTA of 16 warps that split the columns, partial sums in shared memory.
constexpr int C8_U = 8;   // four columns each: loads in flight per lane and row
template <int R>
__global__ void __launch_bounds__(NT8) k_contrib8(DevSym S, const int2 *tasks, const double *y8,
                                                  double *c8) {
  pdl_trigger();
  const int s = tasks[blockIdx.x].x;
  const int lane = threadIdx.x & 31, g = lane >> 2, kq = lane & 3;
  const int a0 = tasks[blockIdx.x].y + 16 * (int)(threadIdx.x >> 5);
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const double *Ls = S.L + S.xptr[s];
  const double *yv = y8 + (size_t)f * R + g;
  const bool in0 = a0 + g < m, in1 = a0 + 8 + g < m;
  const double *p0 = Ls + a0 + g;
  double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  bool first = true;
  for (int k = 0; k < w; k += 4 * C8_U) {
    double l0[C8_U], l1[C8_U], b[C8_U];
#pragma unroll
    for (int u = 0; u < C8_U; ++u) {
      const int col = k + 4 * u + kq;
      l0[u] = ld_if(p0 + (size_t)col * m, in0 && col < w);
      l1[u] = ld_if(p0 + 8 + (size_t)col * m, in1 && col < w);
    }
    if (first) pdl_wait();
    first = false;
#pragma unroll
    for (int u = 0; u < C8_U; ++u) b[u] = ld_if(yv + (size_t)(k + 4 * u + kq) * R, k + 4 * u + kq < w && g < R);
#pragma unroll
    for (int u = 0; u < C8_U; ++u) {
      dmma(c[0], l0[u], b[u]);
      dmma(c[1], l1[u], b[u]);
    }
  }
  double *out = c8 + (size_t)((rb - f) + (a0 + g - w)) * R;
  if (in0) store_pair<R>(out, kq, c[0][0], c[0][1]);
  if (in1) store_pair<R>(out + 8 * R, kq, c[1][0], c[1][1]);
}

constexpr int CS_W = 16;   // warps of the column-split kernel
template <int R>
__global__ void __launch_bounds__(CS_W * 32, 1) k_contrib8_split(DevSym S, const int2 *tasks,
                                                              const double *y8, double *c8) {
  __shared__ __align__(16) double part[CS_W][32 * R8];
  pdl_trigger();
  const int s = tasks[blockIdx.x].x, a0 = tasks[blockIdx.x].y;
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5, g = lane >> 2, kq = lane & 3;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const double *Ls = S.L + S.xptr[s];
  const double *yv = y8 + (size_t)f * R + g;
  const double *p[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = Ls + (a0 + 8 * i + g < m ? a0 + 8 * i + g : 0);
  double c[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i][0] = c[i][1] = 0.0;
  bool first = true;
  for (int k = 16 * wq; k < w || first; k += 16 * CS_W) {
    double l[4][4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int i = 0; i < 4; ++i) l[u][i] = ld_if(p[i] + (size_t)(k + 4 * u + kq) * m, k + 4 * u + kq < w);
    if (first) pdl_wait();
    first = false;
#pragma unroll
    for (int u = 0; u < 4; ++u) b[u] = ld_if(yv + (size_t)(k + 4 * u + kq) * R, k + 4 * u + kq < w && g < R);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int i = 0; i < 4; ++i) dmma(c[i], l[u][i], b[u]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<double2 *>(&part[wq][(8 * i + g) * R8 + 2 * kq]) = make_double2(c[i][0], c[i][1]);
  __syncthreads();
  const int e = threadIdx.x;
  if (e < 32 * R8 && a0 + (e >> 3) < m && (e & 7) < R) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < CS_W; ++q) t += part[q][e];
    c8[(size_t)((rb - f) + (a0 - w)) * R + place8<R>(e)] = t;
  }
}

// ---- gathers of tiled supernodes: x[cols j0 .. j0 + 15] -= L(rows below, cols)^T x[rows];
// warps take 32 rows at a time, partial sums in shared memory.  As with the column-split
// contributions above, the top levels have one CTA per SM and the bytes in flight set the rate:
// sixteen predicated loads of L per lane and sixteen warps, 64 KB.
constexpr int G8_W = 16;
template <int R>
__global__ void __launch_bounds__(G8_W * 32, 1) k_gather8(DevSym S, const int2 *tasks, double *x8) {
  __shared__ __align__(16) double part[G8_W][SOLVE_GATHER_COLS * R8];
  pdl_trigger();
  static_assert(SOLVE_GATHER_COLS == 16, "two products per four rows");
  const int s = tasks[blockIdx.x].x, j0 = tasks[blockIdx.x].y;
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5, g = lane >> 2, kq = lane & 3;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb);
  const int *rows = S.Ls + rb;
  const double *p0 = S.L + S.xptr[s] + (size_t)(j0 + g < w ? j0 + g : j0) * m;
  const double *p1 = S.L + S.xptr[s] + (size_t)(j0 + 8 + g < w ? j0 + 8 + g : j0) * m;
  double c[2][2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) c[i][h][0] = c[i][h][1] = 0.0;
  bool first = true;
  for (int a0 = w + 32 * wq; a0 < m || first; a0 += 32 * G8_W) {
    double l0[8], l1[8], b[8];
    int row[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int a = a0 + 4 * u + kq;
      row[u] = rows[min(a, m - 1)];
      l0[u] = ld_if(p0 + a, a < m);
      l1[u] = ld_if(p1 + a, a < m);
    }
    if (first) pdl_wait();
    first = false;
#pragma unroll
    for (int u = 0; u < 8; ++u) b[u] = ld_if(x8 + (size_t)row[u] * R + g, a0 + 4 * u + kq < m && g < R);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      dmma(c[0][u & 1], l0[u], b[u]);
      dmma(c[1][u & 1], l1[u], b[u]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    *reinterpret_cast<double2 *>(&part[wq][(8 * i + g) * R8 + 2 * kq]) =
        make_double2(c[i][0][0] + c[i][1][0], c[i][0][1] + c[i][1][1]);
  __syncthreads();
  const int e = threadIdx.x;
  if (e < SOLVE_GATHER_COLS * R8 && j0 + (e >> 3) < w && (e & 7) < R) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < G8_W; ++q) t += part[q][e];
    x8[(size_t)(f + j0) * R + place8<R>(e)] -= t;
  }
}

// ---- chained blocks of tiled supernodes: the scheme of k_fwd_chain / k_bwd_chain (clusters
// of CL consecutive blocks, st.async hand-over inside a cluster, counters in global memory
// across clusters, columns of the panel block owned by warps) with eight right-hand sides.
constexpr int CL = 8, NS8 = 4;
constexpr int LW8 = TB + 4;              // padded column of a staged block: conflict-free operands
constexpr int SLOT8 = 8 * LW8;           // one warp's eight columns
constexpr int XB8 = 4;                   // predecessors outside the cluster fetched at a time
constexpr int BLK8 = TB * R8;            // one block's solution
constexpr int CHAIN8_SMEM = (NS8 * W8 * SLOT8 + W8 * XB8 * 8 * R8 + CL * BLK8 + BLK8) * 8;
static_assert(SLOT8 >= BLK8, "a warp's partial sums fit its first slot");

// Rows 8 warp + g, right-hand sides 2 kq, 2 kq + 1 of this block's solution to the later ranks
// of its cluster.
__device__ __forceinline__ void chain8_send(double *yin, unsigned long long *bar, int me, int last,
                                            int e, double a, double b) {
  for (int q = me + 1; q <= last; ++q) {
    const uint32_t d = cluster_addr(yin + me * BLK8 + e, q), mb = cluster_addr(&bar[me], q);
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];\n" ::"r"(d),
                 "d"(a), "r"(mb)
                 : "memory");
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];\n" ::"r"(d + 8),
                 "d"(b), "r"(mb)
                 : "memory");
  }
}

// The block's rows 8 warp .. 8 warp + 7 of T v (tr: this warp's rows of T as operands), sent on.
template <int R>
__device__ __forceinline__ void chain8_finish(const double (&tr)[16], const double *vs, double *yin,
                                              unsigned long long *bar, int me, int last, int bw,
                                              double *dst, int *flag) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, kq = lane & 3;
  double c[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i][0] = c[i][1] = 0.0;
#pragma unroll
  for (int t = 0; t < 16; ++t) dmma(c[t & 3], tr[t], vs[(4 * t + kq) * R8 + g]);
  const double a = (c[0][0] + c[1][0]) + (c[2][0] + c[3][0]);
  const double b = (c[0][1] + c[1][1]) + (c[2][1] + c[3][1]);
  const int row = 8 * wp + g;
  const bool in = row < bw;
  chain8_send(yin, bar, me, last, row * R8 + 2 * kq, in ? a : 0.0, in ? b : 0.0);
  if (in) store_pair<R>(dst + (size_t)row * R, kq, a, b);
  __syncwarp();
  if (lane == 0) red_release_add(flag, 1);
}

template <int R>
__global__ void __launch_bounds__(NT8, 1) k_fwd_chain8(DevSym S, const int2 *tasks, int count, double *y8,
                                                       const double *c8, const int *cptr,
                                                       const int *cidx, int *flags) {
  extern __shared__ double sm8[];
  __shared__ unsigned long long bar[CL];
  double *yin = sm8 + NS8 * W8 * SLOT8 + W8 * XB8 * 8 * R8, *vs = yin + CL * BLK8;
  pdl_trigger();
  cluster_bars_init(bar, CL, BLK8 * 8);
  const int me = (int)chain_rank();
  if ((int)blockIdx.x < count) {
    const int s = tasks[blockIdx.x].x, k = tasks[blockIdx.x].y;
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, g = lane >> 2, kq = lane & 3;
    const int w8 = 8 * wp;
    const int f = S.super[s], w = S.super[s + 1] - f;
    const int m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
    const double *P = S.L + S.xptr[s];
    const int r0 = k * TB, bw = min(TB, w - r0), nb = (w + TB - 1) / TB, base = S.dinv_off[s];
    const double *T = S.dinv + ((size_t)base + k) * (TB * TB);   // T(r, c) at T[c * 64 + r]
    const int cfirst = k - me, last = me + min(nb - 1 - k, CL - 1 - me);
    double *ring = sm8 + wp * SLOT8;
    double *xw = sm8 + NS8 * W8 * SLOT8 + wp * XB8 * 8 * R8;
    auto stage = [&](int c) {
      if (c < k) {
        double *d = ring + (c % NS8) * W8 * SLOT8;
        const double *src = P + (size_t)(c * TB + w8) * m + r0;
#pragma unroll 4
        for (int t = 0; t < 16; ++t) {
          const int e = lane + 32 * t, q = e >> 6, r = e & (TB - 1);
          const bool in = r < bw;
          cp8(d + q * LW8 + r, in ? src + (size_t)q * m + r : src, in);
        }
      }
      stage_commit();
    };
    for (int c = 0; c < NS8 - 1; ++c) stage(c);
    double tr[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) tr[t] = T[(4 * t + kq) * TB + w8 + g];
    pdl_wait();
    // right-hand sides minus the descendants' contributions
#pragma unroll
    for (int h = 0; h < BLK8 / NT8; ++h) {
      const int e = tid + h * NT8, row = e >> 3;
      vs[e] = row < bw ? take_contribs<R>(c8, cptr, cidx, f + r0 + row, e & 7,
                                          at8<R>(y8 + (size_t)(f + r0) * R, e)) : 0.0;
    }
    double acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0.0;
    bool ok = true;
    int xb0 = 0, nbt = 0;
    for (int c = 0; c < k; ++c) {
      stage(c + NS8 - 1);
      stage_wait<NS8 - 1>();
      __syncwarp();
      const double *Lc = ring + (c % NS8) * W8 * SLOT8;
      double a[2][8];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 8; ++i) a[h][i] = Lc[(4 * h + kq) * LW8 + 8 * i + g];
      __syncwarp();                      // the slot is refilled at step c + 1
      double b[2];                       // x_c(8 wp + 4 h + kq, g)
      if (c >= cfirst) {
        const int j = me - (k - c);
        if (!warp_bar_recv(&bar[j], S.status)) { ok = false; break; }
        b[0] = yin[j * BLK8 + (w8 + kq) * R8 + g];
        b[1] = yin[j * BLK8 + (w8 + 4 + kq) * R8 + g];
      } else {
        if (c >= xb0 + nbt) {
          xb0 = c;
          nbt = warp_wait_prefix(&flags[base + c], 1, min(XB8, cfirst - c), W8, S.status);
          if (nbt == 0) { ok = false; break; }
          double t[XB8][2];
#pragma unroll
          for (int u = 0; u < XB8; ++u)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              t[u][h] = u < nbt && g < R ? __ldcg(&y8[(size_t)(f + (c + u) * TB + w8 + 4 * h + kq) * R + g]) : 0.0;
#pragma unroll
          for (int u = 0; u < XB8; ++u)
#pragma unroll
            for (int h = 0; h < 2; ++h) xw[u * 64 + h * 32 + lane] = t[u][h];   // read by this lane
        }
        b[0] = xw[(c - xb0) * 64 + lane];
        b[1] = xw[(c - xb0) * 64 + 32 + lane];
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 8; ++i) dmma(acc[i], a[h][i], b[h]);
    }
    stage_wait<0>();
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<double2 *>(ring + (8 * i + g) * R8 + 2 * kq) = make_double2(acc[i][0], acc[i][1]);
    ok = __syncthreads_and(ok) != 0;
#pragma unroll
    for (int h = 0; h < BLK8 / NT8; ++h) {
      const int e = tid + h * NT8;
      double t = 0.0;
#pragma unroll
      for (int q = 0; q < W8; ++q) t += sm8[q * SLOT8 + e];
      vs[e] -= t;
    }
    __syncthreads();
    if (ok) chain8_finish<R>(tr, vs, yin, bar, me, last, bw, y8 + (size_t)(f + r0) * R, &flags[base + k]);
  }
  cluster_sync_all();
}

template <int R>
__global__ void __launch_bounds__(NT8, 1) k_bwd_chain8(DevSym S, const int2 *tasks, int count, double *x8,
                                                       int *flags) {
  extern __shared__ double sm8[];
  __shared__ unsigned long long bar[CL];
  double *yin = sm8 + NS8 * W8 * SLOT8 + W8 * XB8 * 8 * R8, *vs = yin + CL * BLK8;
  pdl_trigger();
  cluster_bars_init(bar, CL, BLK8 * 8);
  const int me = (int)chain_rank();
  if ((int)blockIdx.x < count) {
    const int s = tasks[blockIdx.x].x, k = tasks[blockIdx.x].y;
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, g = lane >> 2, kq = lane & 3;
    const int w8 = 8 * wp;
    const int f = S.super[s], w = S.super[s + 1] - f;
    const int m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
    const double *P = S.L + S.xptr[s];
    const int r0 = k * TB, bw = min(TB, w - r0), nb = (w + TB - 1) / TB, base = S.dinv_off[s];
    const double *T = S.dinv + ((size_t)base + k) * (TB * TB);
    const int clast = k + me, last = me + min(k, CL - 1 - me);
    double *ring = sm8 + wp * SLOT8;
    auto stage = [&](int t) {   // successor c = nb - 1 - t: column 8 wp + i, row rr at [i][rr]
      const int c = nb - 1 - t;
      if (c > k) {
        double *d = ring + (t % NS8) * W8 * SLOT8;
        const int cw = min(TB, w - c * TB);
        const double *src = P + (size_t)(r0 + w8) * m + c * TB;
#pragma unroll 4
        for (int u = 0; u < 16; ++u) {
          const int e = lane + 32 * u, i = e >> 6, rr = e & 63;
          const bool in = w8 + i < bw && rr < cw;
          cp8(d + i * LW8 + rr, in ? src + (size_t)i * m + rr : src, in);
        }
      }
      stage_commit();
    };
    for (int t = 0; t < NS8 - 1; ++t) stage(t);
    double tr[16];   // T^T(8 wp + g, 4 t + kq)
#pragma unroll
    for (int t = 0; t < 16; ++t) tr[t] = T[(w8 + g) * TB + 4 * t + kq];
    pdl_wait();
    double acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0.0;
    auto fetch = [&](int c, double (&b)[16]) {
      const int cw = min(TB, w - c * TB);
#pragma unroll
      for (int t = 0; t < 16; ++t)
        b[t] = 4 * t + kq < cw && g < R ? __ldcg(&x8[(size_t)(f + c * TB + 4 * t + kq) * R + g]) : 0.0;
    };
    bool ok = true;
    int xb0 = nb, nbt = 0;
    double bn[16];   // the next block's solution when it is known to be finished
    for (int c = nb - 1; c > k; --c) {
      const int t0 = nb - 1 - c;
      stage(t0 + NS8 - 1);
      stage_wait<NS8 - 1>();
      __syncwarp();
      const double *Lc = ring + (t0 % NS8) * W8 * SLOT8;
      double a[16], b[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) a[t] = Lc[g * LW8 + 4 * t + kq];
      __syncwarp();
      if (c <= clast) {
        const int j = me - (c - k);
        if (!warp_bar_recv(&bar[j], S.status)) { ok = false; break; }
#pragma unroll
        for (int t = 0; t < 16; ++t) b[t] = yin[j * BLK8 + (4 * t + kq) * R8 + g];
      } else {
        if (c <= xb0 - nbt) {
          xb0 = c;
          nbt = warp_wait_prefix(&flags[base + c], -1, min(8, c - clast), 2 * W8, S.status);
          if (nbt == 0) { ok = false; break; }
          fetch(c, bn);
        }
#pragma unroll
        for (int t = 0; t < 16; ++t) b[t] = bn[t];
        if (c - 1 > clast && c - 1 > xb0 - nbt) fetch(c - 1, bn);
      }
#pragma unroll
      for (int t = 0; t < 16; ++t) dmma(acc[t & 3], a[t], b[t]);
    }
    stage_wait<0>();
    {
      const int row = w8 + g;
      const double s0 = (acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0]);
      const double s1 = (acc[0][1] + acc[1][1]) + (acc[2][1] + acc[3][1]);
      double2 v = make_double2(0.0, 0.0);
      if (R > 1 && row < bw && 2 * kq < R)
        v = *reinterpret_cast<const double2 *>(&x8[(size_t)(f + r0 + row) * R + 2 * kq]);
      if (R == 1 && row < bw && kq == 0) v.x = x8[f + r0 + row];
      *reinterpret_cast<double2 *>(vs + row * R8 + 2 * kq) = make_double2(v.x - s0, v.y - s1);
    }
    ok = __syncthreads_and(ok) != 0;
    if (ok) chain8_finish<R>(tr, vs, yin, bar, me, last, bw, x8 + (size_t)(f + r0) * R, &flags[base + k]);
  }
  cluster_sync_all();
}

// nr vectors of length n (leading dimension n) to the form interleaved by R, zeros beyond nr; and back.
template <int R>
__global__ void k_pack8(int n, int nr, const double *x, double *x8) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(e / R), r = (int)(e % R);
  if (i < n) x8[e] = r < nr ? x[(size_t)r * n + i] : 0.0;
}
template <int R>
__global__ void k_unpack8(int n, int nr, const double *x8, double *x) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(e / R), r = (int)(e % R);
  if (i < n && r < nr) x[(size_t)r * n + i] = x8[e];
}

// fn with the interleaving as a constant
template <class F>
void with_stride(int stride, F fn) {
  if (stride == 8) fn(std::integral_constant<int, 8>());
  else if (stride == 4) fn(std::integral_constant<int, 4>());
  else if (stride == 2) fn(std::integral_constant<int, 2>());
  else fn(std::integral_constant<int, 1>());
}

}  // namespace

bool solve8_configure(std::string &err) {
  cudaError_t e = cudaSuccess;
  for (auto k : {k_fwd_chain8<8>, k_fwd_chain8<4>, k_fwd_chain8<2>, k_fwd_chain8<1>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CHAIN8_SMEM);
  for (auto k : {k_bwd_chain8<8>, k_bwd_chain8<4>, k_bwd_chain8<2>, k_bwd_chain8<1>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CHAIN8_SMEM);
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return false;
  }
  return true;
}

void launch_pack8(int n, int nr, const double *x, double *x8, int stride, cudaStream_t st) {
  const unsigned grid = (unsigned)(((int64_t)n * stride + 255) / 256);
  with_stride(stride, [&](auto R) { k_pack8<R.value><<<grid, 256, 0, st>>>(n, nr, x, x8); });
}
void launch_unpack8(int n, int nr, const double *x8, double *x, int stride, cudaStream_t st) {
  const unsigned grid = (unsigned)(((int64_t)n * stride + 255) / 256);
  with_stride(stride, [&](auto R) { k_unpack8<R.value><<<grid, 256, 0, st>>>(n, nr, x8, x); });
}

template <int R>
static void solve8_levels(const DevSym &S, const SolvePlan &SP, const Solve8Dev &D, double *x8, double *c8,
                          int l0, int l1, bool fwd, LaunchQueue &st) {
  auto chain = [&](int off, int cnt) {
    const int grid = (cnt + CL - 1) / CL * CL;
    if (cnt <= 0) return;
    if (fwd)
      launch_early(st, CL, k_fwd_chain8<R>, grid, NT8, CHAIN8_SMEM, S, D.fchain + off, cnt, x8, c8, D.cptr, D.cidx,
                   D.flags);
    else
      launch_early(st, CL, k_bwd_chain8<R>, grid, NT8, CHAIN8_SMEM, S, D.bchain + off, cnt, x8, D.flags);
  };
  for (int l = l0; fwd && l < l1; ++l) {
    const int nw = SP.warp_off[l + 1] - SP.warp_off[l], ns = SP.level_off[l + 1] - SP.level_off[l];
    const int nc = SP.c8_off[l + 1] - SP.c8_off[l];
    if (nw > 0)
      launch_early(st, 1, k_fwd_warp8<R>, (nw + WN - 1) / WN, WN * 32, 0, S, D.warp_list + SP.warp_off[l], nw, x8,
                   c8, D.cptr, D.cidx);
    if (ns > 0)
      launch_early(st, 1, k_fwd_small8<R>, ns, NT8, SMALL8_SMEM, S, D.list + SP.level_off[l], x8, c8, D.cptr, D.cidx);
    chain(SP.chain_off[l], SP.chain_off[l + 1] - SP.chain_off[l]);
    if (nc > 0 && SP.c8_split[l])
      launch_early(st, 1, k_contrib8_split<R>, nc, CS_W * 32, 0, S, D.c8_tasks + SP.c8_off[l], x8, c8);
    else if (nc > 0)
      launch_early(st, 1, k_contrib8<R>, nc, NT8, 0, S, D.c8_tasks + SP.c8_off[l], x8, c8);
  }
  for (int l = l1 - 1; !fwd && l >= l0; --l) {
    const int nw = SP.warp_off[l + 1] - SP.warp_off[l], ns = SP.level_off[l + 1] - SP.level_off[l];
    const int ng = SP.g8_off[l + 1] - SP.g8_off[l];
    if (ng > 0) launch_early(st, 1, k_gather8<R>, ng, G8_W * 32, 0, S, D.g8_tasks + SP.g8_off[l], x8);
    chain(SP.chain_off[l], SP.chain_off[l + 1] - SP.chain_off[l]);
    if (ns > 0) launch_early(st, 1, k_bwd_small8<R>, ns, NT8, SMALL8_SMEM, S, D.list + SP.level_off[l], x8);
    if (nw > 0)
      launch_early(st, 1, k_bwd_warp8<R>, (nw + WN - 1) / WN, WN * 32, 0, S, D.warp_list + SP.warp_off[l], nw, x8);
  }
}

void launch_solve8(const DevSym &S, const SolvePlan &SP, const Solve8Dev &D, double *x8, double *c8, int stride,
                   int l0, int l1, bool fwd, LaunchQueue &st) {
  with_stride(stride, [&](auto R) { solve8_levels<R.value>(S, SP, D, x8, c8, l0, l1, fwd, st); });
}

}  // namespace swc
