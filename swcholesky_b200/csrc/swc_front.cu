// Multifrontal FP64 kernels: the fronts of small supernodes in shared memory (one warp or one
// CTA each, walked from a device queue or launched per level), the extend-add of children's
// contribution blocks into the panels of wide supernodes, and the tiles of their own
// contribution blocks.  The reference's counterpart is the update loop of its executor
// (cholesky/sw_parallel_PB_Cholesky_05.c:254-378), which revisits every descendant instead.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "swc_front.h"
#include "swc_tile.h"

namespace swc {

namespace {

constexpr int FT = 256, FW = FT / 32;       // CTA fronts: threads, warps
constexpr int WW = 4;                       // warp fronts: warps per CTA
constexpr int WARP_SLICE = FRONT_WARP_ELEMS * 8 + 64 * 8 + FRONT_KIDS * FRONT_WARP_M * 2;
constexpr int WARP_SMEM = WW * WARP_SLICE;

template <int NW>
__device__ __forceinline__ void group_sync() {
  if (NW == 1) __syncwarp(); else __syncthreads();
}

// The whole factorization of one small front s in shared memory by NW warps:
//   assembly of A and of the children's blocks into the padded panel P, Cholesky by 8-column
//   blocks (the 8x8 diagonal blocks by one warp with their inverses, everything else 8x8x4
//   DMMA products), the panel to L, and the contribution block
//   CB_s = (children's blocks) - L_rs L_rs^T to global memory unless cb_by_tiles.
// Bound: latency (the chain of 8x8 pivots blocks, then barriers); a front of 16 columns and 50
// rows takes a few microseconds.  T: 64 doubles (inverse of the current diagonal block), inv:
// FRONT_KIDS row maps of m entries.
template <int NW>
__device__ void front_body(const DevSym &S, const FrontDev &F, int s, bool cb_by_tiles, double *P,
                           double *T, short *inv) {
  constexpr int NTH = 32 * NW;
  const int t = NW == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  const int lane = t & 31, warp = t >> 5, g = lane >> 2, kq = lane & 3;
  const int f = S.super[s], w = S.super[s + 1] - f;
  const int64_t rb = S.rowptr[s];
  const int m = (int)(S.rowptr[s + 1] - rb), r = m - w;
  const int wp = front_wp(w), ld = front_ld(w, m), pad = wp - w;
  const int nrb = (wp + ((r + 7) & ~7)) >> 3, nkb = wp >> 3;   // 8-row / 8-column blocks
  const int ch0 = F.child_ptr[s], ch1 = F.child_ptr[s + 1];

  for (int i = t; i < wp * ld; i += NTH) P[i] = 0.0;
  group_sync<NW>();
  if (t < pad) P[(w + t) * ld + w + t] = 1.0;
  // A: one warp per column (front row i at i, or i + pad below the padded columns)
  for (int j = warp; j < w; j += NW)
    for (int p = S.Ap[f + j] + lane; p < S.Ap[f + j + 1]; p += 32) {
      const int pos = F.apos[p];
      if (pos >= 0) P[j * ld + (pos < w ? pos : pos + pad)] = S.Ax[p];
      else atomicExch(&S.status[1], 1);
    }
  group_sync<NW>();
  // children's blocks, the columns that are columns of s
  for (int q = ch0; q < ch1; ++q) {
    const int c = F.child[q];
    const int64_t ro = S.rowptr[c] - S.super[c];
    const int rc = (int)(S.rowptr[c + 1] - S.rowptr[c]) - (S.super[c + 1] - S.super[c]);
    const int n1 = F.child_n1[c];
    const int *rel = F.rel + ro;
    const double *cb = F.cb + F.cb_off[c];
    for (int j = warp; j < n1; j += NW) {
      const int pj = rel[j];
      for (int i = j + lane; i < rc; i += 32) {
        const int pi = rel[i];
        P[pj * ld + (pi < w ? pi : pi + pad)] += cb[(size_t)j * rc + i];
      }
    }
    group_sync<NW>();
  }

  // Cholesky of the panel by 8-column blocks; warp 0 factors the next diagonal block while the
  // others update the rest
  if (warp == 0) potrf8_inv8(P, ld, T, S.status, f, w);
  group_sync<NW>();
  for (int kb = 0; kb < nkb; ++kb) {
    const int k0 = 8 * kb;
    // rows below: X = B L_kk^{-T}, four row blocks of a warp interleaved
    for (int ib0 = kb + 1 + 4 * warp; ib0 < nrb; ib0 += 4 * NW) {
      double c[4][2];
#pragma unroll
      for (int q = 0; q < 4; ++q) c[q][0] = c[q][1] = 0.0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double b = T[(4 * h + kq) * 8 + g];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (ib0 + q < nrb) dmma(c[q], P[(k0 + 4 * h + kq) * ld + 8 * (ib0 + q) + g], b);
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (ib0 + q < nrb) {
          P[(k0 + 2 * kq) * ld + 8 * (ib0 + q) + g] = c[q][0];
          P[(k0 + 2 * kq + 1) * ld + 8 * (ib0 + q) + g] = c[q][1];
        }
    }
    group_sync<NW>();
    if (kb + 1 >= nkb) break;
    // trailing blocks (ib, jb), kb < jb <= ib: minus X_ib X_jb^T
    auto update4 = [&](int jb, int ib0, int ib1) {   // row blocks ib0 .. min(ib0 + 4, ib1) - 1
      double c[4][2];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (ib0 + q < ib1) {
          c[q][0] = P[(8 * jb + 2 * kq) * ld + 8 * (ib0 + q) + g];
          c[q][1] = P[(8 * jb + 2 * kq + 1) * ld + 8 * (ib0 + q) + g];
        }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double b = neg(P[(k0 + 4 * h + kq) * ld + 8 * jb + g]);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (ib0 + q < ib1) dmma(c[q], P[(k0 + 4 * h + kq) * ld + 8 * (ib0 + q) + g], b);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (ib0 + q < ib1) {
          P[(8 * jb + 2 * kq) * ld + 8 * (ib0 + q) + g] = c[q][0];
          P[(8 * jb + 2 * kq + 1) * ld + 8 * (ib0 + q) + g] = c[q][1];
        }
    };
    const int nb = kb + 1;
    if (warp == 0) {
      update4(nb, nb, nb + 1);
      __syncwarp();
      potrf8_inv8(P + 8 * nb * ld + 8 * nb, ld, T, S.status, f + 8 * nb, w - 8 * nb);
    }
    if (NW == 1 || warp > 0) {
      const int u = NW == 1 ? 0 : warp - 1, nu = NW == 1 ? 1 : NW - 1;
      int strip = 0;
      for (int jb = nb; jb < nkb; ++jb)
        for (int ib0 = jb == nb ? jb + 1 : jb; ib0 < nrb; ib0 += 4, ++strip)
          if (strip % nu == u) update4(jb, ib0, nrb);
    }
    group_sync<NW>();
  }

  // the panel to L (upper triangle of the diagonal block: zeros, as stored by the reference)
  double *dst = S.L + S.xptr[s];
  for (int j = warp; j < w; j += NW)
    for (int i = lane; i < m; i += 32)
      dst[(size_t)j * m + i] = i < j ? 0.0 : P[j * ld + (i < w ? i : i + pad)];

  if (r == 0 || cb_by_tiles) return;
  double *cbs = F.cb + F.cb_off[s];
  const int r8 = (r + 7) >> 3;
  int q0 = ch0;
  do {
    // row maps of up to FRONT_KIDS children: inv[k * m + i] = the child's index of s's
    // off-diagonal row i, or -1
    const int kids = min(FRONT_KIDS, ch1 - q0);
    for (int i = t; i < kids * r; i += NTH) inv[i] = -1;
    group_sync<NW>();
    const double *cbc[FRONT_KIDS];
    int rc[FRONT_KIDS];
#pragma unroll
    for (int k = 0; k < FRONT_KIDS; ++k) {
      cbc[k] = nullptr;
      rc[k] = 0;
      if (k < kids) {
        const int c = F.child[q0 + k];
        rc[k] = (int)(S.rowptr[c + 1] - S.rowptr[c]) - (S.super[c + 1] - S.super[c]);
        cbc[k] = F.cb + F.cb_off[c];
        const int *rel = F.rel + (S.rowptr[c] - S.super[c]);
        for (int i = F.child_n1[c] + t; i < rc[k]; i += NTH) inv[k * r + rel[i] - w] = (short)i;
      }
    }
    group_sync<NW>();
    int strip = 0;
    for (int bj = 0; bj < r8; ++bj)
      for (int bi0 = bj; bi0 < r8; bi0 += 4, ++strip) {
        if (strip % NW != warp) continue;
        double c[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q][0] = c[q][1] = 0.0;
        if (q0 == ch0) {
          for (int k = 0; k < wp; k += 4) {
            const double b = neg(P[(k + kq) * ld + wp + 8 * bj + g]);
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (bi0 + q < r8) dmma(c[q], P[(k + kq) * ld + wp + 8 * (bi0 + q) + g], b);
          }
        }
        const int j0 = 8 * bj + 2 * kq;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = 8 * (bi0 + q) + g;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = j0 + e;
            if (i < r && j <= i) {
              double v = c[q][e];
              if (q0 > ch0) v += cbs[(size_t)j * r + i];
#pragma unroll
              for (int k = 0; k < FRONT_KIDS; ++k)
                if (k < kids) {
                  const int pi = inv[k * r + i], pj = inv[k * r + j];
                  if (pi >= 0 && pj >= 0) v += cbc[k][(size_t)pj * rc[k] + pi];
                }
              cbs[(size_t)j * r + i] = v;
            }
          }
        }
      }
    q0 += FRONT_KIDS;
    group_sync<NW>();
  } while (q0 < ch1);
}

// Lane q waits (bounded by the poll budget) for the done flag of s's child q.
__device__ __forceinline__ void wait_children(const DevSym &S, const FrontDev &F, int s,
                                              const int *done) {
  const long long budget = wait_budget(S.status);
  bool timed_out = false;
  for (int q = F.child_ptr[s] + (int)(threadIdx.x & 31); q < F.child_ptr[s + 1] && !timed_out; q += 32) {
    const int *flag = done + F.child[q];
    long long it = 0;
    while (ld_acquire_k(flag) == 0) {
      if (++it > budget) {
        atomicExch(&S.status[3], 1);
        timed_out = true;
        break;
      }
      __nanosleep(32);
    }
  }
}

// The fronts of the bottom of the tree (a set closed under descendants) in one persistent
// launch: CTAs take fronts from a device queue in level order, wait for the fronts' children
// (acquire on their done flags), factor and publish their own flag (release).  A CTA only
// waits for fronts taken before its own, so the walk progresses whatever the number of
// resident CTAs.  qctr[0]: queue head, qctr[1 + s]: done flags, zeroed before the launch.
__global__ void __launch_bounds__(FT) k_front_cta_walk(DevSym S, FrontDev F, const int *order,
                                                       int count, int *qctr) {
  extern __shared__ double fsm[];
  __shared__ int item;
  int *done = qctr + 1;
  for (;;) {
    if (threadIdx.x == 0) item = atomicAdd(qctr, 1);
    __syncthreads();
    const int idx = item;
    if (idx >= count) break;
    const int s = order[idx];
    if (threadIdx.x < 32) wait_children(S, F, s, done);
    __syncthreads();
    front_body<FW>(S, F, s, false, fsm + 64, fsm, reinterpret_cast<short *>(
        fsm + 64 + front_wp(S.super[s + 1] - S.super[s]) *
                       front_ld(S.super[s + 1] - S.super[s], (int)(S.rowptr[s + 1] - S.rowptr[s]))));
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      st_release_k(done + s, 1);
    }
  }
}

// The same at warp granularity, for the crowded levels of tiny fronts.
__global__ void __launch_bounds__(WW * 32) k_front_warp_walk(DevSym S, FrontDev F, const int *order,
                                                             int count, int *qctr, int *qhead) {
  extern __shared__ double fsm[];
  const int lane = threadIdx.x & 31;
  double *T = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(fsm) +
                                         (size_t)(threadIdx.x >> 5) * WARP_SLICE);
  double *P = T + 64;
  short *inv = reinterpret_cast<short *>(P + FRONT_WARP_ELEMS);
  int *done = qctr + 1;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = atomicAdd(qhead, 1);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (idx >= count) break;
    const int s = order[idx];
    wait_children(S, F, s, done);
    __syncwarp();
    front_body<1>(S, F, s, false, P, T, inv);
    __syncwarp();
    if (lane == 0) {
      __threadfence();
      st_release_k(done + s, 1);
    }
  }
}

// One CTA per small front of a level.
__global__ void __launch_bounds__(FT) k_front_small(DevSym S, FrontDev F, const int *list) {
  extern __shared__ double fsm[];
  const int e = list[blockIdx.x], s = e < 0 ? ~e : e;
  const int w = S.super[s + 1] - S.super[s], m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
  front_body<FW>(S, F, s, e < 0, fsm + 64, fsm,
                 reinterpret_cast<short *>(fsm + 64 + front_wp(w) * front_ld(w, m)));
}

// Children's blocks into one 64x64 tile: row maps of up to FRONT_KIDS pairs at a time.  Pair
// (c, a0, b0, na | nb << 16): rows a0 .. a0 + na - 1 of child c's block fall in the tile's rows
// [rbase, rbase + 64), rows b0 .. b0 + nb - 1 in its columns [cbase, cbase + 64) (positions
// in the parent's row list).
struct PairMaps {
  short ia[FRONT_KIDS][TB], ib[FRONT_KIDS][TB];
  const double *cb[FRONT_KIDS];   // the child's block, from its entry (a0, b0)
  int ld[FRONT_KIDS];
};

__device__ __forceinline__ void load_pair_maps(const DevSym &S, const FrontDev &F, const int4 *pairs,
                                               int q, int kids, int rbase, int cbase, PairMaps &M,
                                               int nth) {
  for (int i = threadIdx.x; i < kids * TB; i += nth) M.ia[i >> 6][i & 63] = M.ib[i >> 6][i & 63] = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < kids * 2 * TB; i += nth) {
    const int k = i >> 7, u = i & 63;
    const int4 pr = pairs[q + k];
    const int c = pr.x;
    const int *rel = F.rel + (S.rowptr[c] - S.super[c]);
    if (i & 64) {
      if (u < (pr.w >> 16)) M.ib[k][rel[pr.z + u] - cbase] = (short)u;
    } else {
      if (u < (pr.w & 0xffff)) M.ia[k][rel[pr.y + u] - rbase] = (short)u;
      if (u == 0) {
        const int rc = (int)(S.rowptr[c + 1] - S.rowptr[c]) - (S.super[c + 1] - S.super[c]);
        M.cb[k] = F.cb + F.cb_off[c] + (size_t)pr.z * rc + pr.y;
        M.ld[k] = rc;
      }
    }
  }
  __syncthreads();
}

// Extend-add into the panels of tiled supernodes: task = (s, r0, c0, first pair), a 64x64 tile
// of the panel that some child's block reaches.  Bound: memory (the blocks are read once and
// the touched tiles read and written once).
__global__ void __launch_bounds__(FT) k_front_extend(DevSym S, FrontDev F, const int4 *tasks,
                                                     const int *end, const int4 *pairs) {
  __shared__ PairMaps M;
  const int4 tk = tasks[blockIdx.x];
  const int p_end = end[blockIdx.x];
  const int s = tk.x, r0 = tk.y, c0 = tk.z;
  const int w = S.super[s + 1] - S.super[s], m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
  double *Lt = S.L + S.xptr[s] + (size_t)c0 * m + r0;
  const int row = threadIdx.x & 63, cq = threadIdx.x >> 6;   // columns cq, cq + 4, ..
  constexpr int NE = TB * TB / FT;
  double v[NE];
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const int col = cq + 4 * e;
    v[e] = (r0 + row < m && c0 + col < w && r0 + row >= c0 + col) ? Lt[(size_t)col * m + row] : 0.0;
  }
  for (int q = tk.w; q < p_end; q += FRONT_KIDS) {
    const int kids = min(FRONT_KIDS, p_end - q);
    if (q > tk.w) __syncthreads();
    load_pair_maps(S, F, pairs, q, kids, r0, c0, M, FT);
    for (int k = 0; k < kids; ++k) {
      const int pi = M.ia[k][row];
      const double *cb = M.cb[k] + pi;
      const int ldc = M.ld[k];
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        const int col = cq + 4 * e, pj = M.ib[k][col];
        if (pi >= 0 && pj >= 0 && r0 + row >= c0 + col) v[e] += cb[(size_t)pj * ldc];
      }
    }
  }
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const int col = cq + 4 * e;
    if (r0 + row < m && c0 + col < w && r0 + row >= c0 + col) Lt[(size_t)col * m + row] = v[e];
  }
}

// One 64x64 tile of the contribution block of s: minus L_rs L_rs^T (DMMA, K = w) plus the
// children's blocks.  task = (s, i0, j0, first pair), offsets in the block.  The accumulator
// collects minus the children's entries and the product, and is stored back negated.
constexpr int SCHUR_SMEM = 2 * STAGE * 8;
__global__ void __launch_bounds__(MT, 4) k_front_schur(DevSym S, FrontDev F, const int4 *tasks,
                                                       const int *end, const int4 *pairs) {
  extern __shared__ double fsm[];
  __shared__ PairMaps M;
  const int4 tk = tasks[blockIdx.x];
  const int p_end = end[blockIdx.x];
  const int s = tk.x, i0 = tk.y, j0 = tk.z;
  const int w = S.super[s + 1] - S.super[s], m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
  const int r = m - w;
  TileAcc acc;
  acc.zero();
  for (int q = tk.w; q < p_end; q += FRONT_KIDS) {
    const int kids = min(FRONT_KIDS, p_end - q);
    if (q > tk.w) __syncthreads();
    load_pair_maps(S, F, pairs, q, kids, w + i0, w + j0, M, MT);
    for (int k = 0; k < kids; ++k) {
      const double *cb = M.cb[k];
      const int ldc = M.ld[k];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int pi = M.ia[k][acc_row(i)];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int pj = M.ib[k][acc_col(j, e)];
            if (pi >= 0 && pj >= 0 && i0 + acc_row(i) >= j0 + acc_col(j, e))
              acc.v[i][j][e] -= cb[(size_t)pj * ldc + pi];
          }
      }
    }
  }
  const double *Lr = S.L + S.xptr[s] + w;
  dmma_tile_product(Lr + i0, m, min(TB, r - i0), Lr + j0, m, min(TB, r - j0), w, fsm, acc);
  double *cbs = F.cb + F.cb_off[s];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int ri = i0 + acc_row(i);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cj = j0 + acc_col(j, e);
        if (ri < r && cj <= ri) cbs[(size_t)cj * r + ri] = neg(acc.v[i][j][e]);
      }
  }
}

int resident_ctas(const void *fn, int threads, int smem) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem) != cudaSuccess || per < 1)
    per = 1;
  return sms * per;
}

}  // namespace

bool front_configure(std::string &err) {
  cudaError_t e = cudaFuncSetAttribute(k_front_cta_walk, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       200 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_small, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_warp_walk, cudaFuncAttributeMaxDynamicSharedMemorySize, WARP_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_schur, cudaFuncAttributeMaxDynamicSharedMemorySize, SCHUR_SMEM);
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return false;
  }
  return true;
}

int front_cta_walk_ctas(int smem, int count) {
  return std::max(1, std::min(count, resident_ctas((const void *)k_front_cta_walk, FT, smem)));
}
int front_warp_walk_ctas(int count) {
  return std::max(1, std::min((count + WW - 1) / WW,
                              resident_ctas((const void *)k_front_warp_walk, WW * 32, WARP_SMEM)));
}
void launch_front_warp_walk(const DevSym &S, const FrontDev &F, const int *order, int count,
                            int ctas, int *qctr, int *qhead, cudaStream_t st) {
  if (count > 0)
    k_front_warp_walk<<<ctas, WW * 32, WARP_SMEM, st>>>(S, F, order, count, qctr, qhead);
}
void launch_front_cta_walk(const DevSym &S, const FrontDev &F, const int *order, int count,
                           int smem, int ctas, int *qctr, cudaStream_t st) {
  if (count > 0) k_front_cta_walk<<<ctas, FT, smem, st>>>(S, F, order, count, qctr);
}
void launch_front_small(const DevSym &S, const FrontDev &F, const int *list, int count, int smem,
                        cudaStream_t st) {
  if (count > 0) k_front_small<<<count, FT, smem, st>>>(S, F, list);
}
void launch_front_extend(const DevSym &S, const FrontDev &F, const int4 *tasks, const int *end,
                         const int4 *pairs, int count, cudaStream_t st) {
  if (count > 0) k_front_extend<<<count, FT, 0, st>>>(S, F, tasks, end, pairs);
}
void launch_front_schur(const DevSym &S, const FrontDev &F, const int4 *tasks, const int *end,
                        const int4 *pairs, int count, cudaStream_t st) {
  if (count > 0) k_front_schur<<<count, MT, SCHUR_SMEM, st>>>(S, F, tasks, end, pairs);
}

}  // namespace swc
