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

constexpr int FT = 256, FW = FT / 32;       // CTA fronts: threads, warps (largest)
// Walks of at least this many fronts use CTAs of 128 threads, three to an SM, others one of 256:
// long walks are bound by how many fronts are in flight (60^3 7-point grid, 5,900 fronts:
// 15.58 against 15.81 ms), short ones by each front's latency (100 x 100 5-point grid, 1,221
// fronts: 319 against 390 us).
constexpr int FRONT_MANY = 2048;
constexpr int ET = 256;                     // extend-add tiles
constexpr int WW = 4;                       // warp fronts: warps per CTA
constexpr int WARP_SLICE = FRONT_WARP_ELEMS * 8 + 64 * 8 + FRONT_KIDS * FRONT_WARP_M * 2;
constexpr int WARP_SMEM = WW * WARP_SLICE;

template <int NW>
__device__ __forceinline__ void group_sync() {
  if (NW == 1) __syncwarp(); else __syncthreads();
}

// The whole factorization of one small front in shared memory by NW warps:
//   row maps of the children (up to FRONT_KIDS at a time), the padded panel P gathered from the
//   children's blocks through them, A's entries, the panel's Cholesky (chol_panel), the panel to
//   L, and the contribution block CB = (children's blocks) - L_rs L_rs^T to global memory
//   (unless d.cb < 0).
// Bound: latency.  A front passes four dependent global loads (its children's descriptors,
// their row maps, their blocks; A's entries beside them), the chain of pivots and seven or so
// barriers; the loads of a phase are issued together, several per thread.  sc: 64 doubles per
// warp, inv: FRONT_KIDS row maps of m entries (inv[k * mm + i]: child k's index of row i, or -1).
template <int NW>
__device__ __forceinline__ void build_maps(const FrontDev &F, int q0, int kids, int w, int m, int mm,
                                           short *inv, const double *(&cb)[FRONT_KIDS],
                                           int (&rc)[FRONT_KIDS]) {
  constexpr int NTH = 32 * NW;
  const int t = NW == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  int64_t rel[FRONT_KIDS];
#pragma unroll
  for (int k = 0; k < FRONT_KIDS; ++k) {
    cb[k] = nullptr;
    rc[k] = 0;
    rel[k] = 0;
    if (k < kids) {
      const FrontChild c = F.child[q0 + k];
      rc[k] = c.rc;
      rel[k] = c.rel;
      cb[k] = F.cb + c.cb;
    }
  }
  for (int i = t; i < kids * mm; i += NTH) inv[i] = -1;
  group_sync<NW>();
#pragma unroll
  for (int k = 0; k < FRONT_KIDS; ++k)
    for (int i = t; i < rc[k]; i += NTH) inv[k * mm + F.rel[rel[k] + i]] = (short)i;
  group_sync<NW>();
}

template <int NW>
__device__ void front_body(const DevSym &S, const FrontDev &F, const FrontDesc &d, double *P, double *sc,
                           short *inv) {
  constexpr int NTH = 32 * NW;
  const int t = NW == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  const int lane = t & 31, warp = t >> 5, g = lane >> 2, kq = lane & 3;
  const int w = d.w, m = d.m, r = m - w;
  const int wp = front_wp(w), ld = front_ld(w, m), pad = wp - w, mm = (m + 3) & ~3;
  const int nrb = (wp + ((r + 7) & ~7)) >> 3, nkb = wp >> 3;   // 8-row / 8-column blocks
  const double *cb[FRONT_KIDS];
  int rc[FRONT_KIDS];
  int kids = min(FRONT_KIDS, d.ch1 - d.ch0);
  build_maps<NW>(F, d.ch0, kids, w, m, mm, inv, cb, rc);

  // the panel from the children's blocks (padded diagonal: ones), four entries per thread at a time
  for (int q0 = d.ch0;;) {
    const bool first = q0 == d.ch0;
    for (int e0 = t; e0 < wp * ld; e0 += 4 * NTH) {
      double v[4][FRONT_KIDS];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = e0 + u * NTH, j = e / ld, i = e - j * ld;
        const int row = i < wp ? i : i - pad;
        const bool in = e < wp * ld && j < w && (i < wp ? i < w && i >= j : row < m);
#pragma unroll
        for (int k = 0; k < FRONT_KIDS; ++k) {
          v[u][k] = 0.0;
          if (k < kids) {
            const int pi = in ? inv[k * mm + row] : -1, pj = in ? inv[k * mm + j] : -1;
            v[u][k] = ld_if(cb[k] + (int64_t)pj * rc[k] + pi, pi >= 0 && pj >= 0);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = e0 + u * NTH;
        if (e < wp * ld) {
          const int j = e / ld;
          double x = first ? (j >= w && e == j * ld + j ? 1.0 : 0.0) : P[e];
#pragma unroll
          for (int k = 0; k < FRONT_KIDS; ++k) x += v[u][k];
          P[e] = x;
        }
      }
    }
    q0 += FRONT_KIDS;
    if (q0 >= d.ch1) break;
    group_sync<NW>();
    kids = min(FRONT_KIDS, d.ch1 - q0);
    build_maps<NW>(F, q0, kids, w, m, mm, inv, cb, rc);
  }
  group_sync<NW>();
  for (int p = d.a0 + t; p < d.a1; p += NTH) {
    const int pos = F.ppos[p];
    if (pos >= 0) P[pos] += S.Ax[p];
    else atomicExch(&S.status[1], 1);
  }
  group_sync<NW>();

  chol_panel<NW>(P, ld, nkb, nrb, sc, S.status, d.f, w);

  // the panel to L (upper triangle of the diagonal block: zeros, as stored by the reference)
  double *dst = S.L + d.xoff;
  for (int j = warp; j < w; j += NW)
    for (int i = lane; i < m; i += 32)
      dst[(size_t)j * m + i] = i < j ? 0.0 : P[j * ld + (i < w ? i : i + pad)];

  if (r == 0 || d.cb < 0) return;
  double *cbs = F.cb + d.cb;
  const int r8 = (r + 7) >> 3;
  const bool many = d.ch1 - d.ch0 > FRONT_KIDS;
  for (int q0 = d.ch0;;) {
    const bool first = q0 == d.ch0;
    if (many) {
      kids = min(FRONT_KIDS, d.ch1 - q0);
      group_sync<NW>();
      build_maps<NW>(F, q0, kids, w, m, mm, inv, cb, rc);
    }
    const short *im = inv + w;   // off-diagonal rows
    int strip = 0;
    for (int bj = 0; bj < r8; ++bj)
      for (int bi0 = bj; bi0 < r8; bi0 += 4, ++strip) {
        if (strip % NW != warp) continue;
        // the children's entries first: in flight during the product
        const int j0 = 8 * bj + 2 * kq;
        double v[FRONT_KIDS][4][2], old[4][2];
        int pj[FRONT_KIDS][2];
#pragma unroll
        for (int k = 0; k < FRONT_KIDS; ++k)
#pragma unroll
          for (int e = 0; e < 2; ++e) pj[k][e] = k < kids && j0 + e < r ? im[k * mm + j0 + e] : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = 8 * (bi0 + q) + g;
#pragma unroll
          for (int e = 0; e < 2; ++e)
            old[q][e] = first ? 0.0 : ld_if(cbs + (size_t)(j0 + e) * r + i, i < r && j0 + e <= i);
#pragma unroll
          for (int k = 0; k < FRONT_KIDS; ++k) {
            v[k][q][0] = v[k][q][1] = 0.0;
            if (k < kids) {
              const int pi = i < r ? im[k * mm + i] : -1;
#pragma unroll
              for (int e = 0; e < 2; ++e)
                v[k][q][e] = ld_if(cb[k] + (int64_t)pj[k][e] * rc[k] + pi, pi >= 0 && pj[k][e] >= 0 && j0 + e <= i);
            }
          }
        }
        double c[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q][0] = c[q][1] = 0.0;
        if (first)
          for (int k = 0; k < wp; k += 4) {
            const double b = neg(P[(k + kq) * ld + wp + 8 * bj + g]);
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (bi0 + q < r8) dmma(c[q], P[(k + kq) * ld + wp + 8 * (bi0 + q) + g], b);
          }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = 8 * (bi0 + q) + g;
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (i < r && j0 + e <= i) {
              double x = c[q][e] + old[q][e];
#pragma unroll
              for (int k = 0; k < FRONT_KIDS; ++k) x += v[k][q][e];
              cbs[(size_t)(j0 + e) * r + i] = x;
            }
        }
      }
    q0 += FRONT_KIDS;
    if (q0 >= d.ch1) break;
  }
}

// Lane q waits (bounded by the poll budget) for the done flag of the front's child q.
__device__ __forceinline__ void wait_children(const DevSym &S, const FrontDev &F, const FrontDesc &d,
                                              const int *done) {
  const long long budget = wait_budget(S.status);
  bool timed_out = false;
  for (int q = d.ch0 + (int)(threadIdx.x & 31); q < d.ch1 && !timed_out; q += 32) {
    const int *flag = done + F.child[q].s;
    long long it = 0;
    while (ld_acquire_k(flag) == 0) {
      if (++it > budget) {
        atomicExch(&S.status[3], 1);
        timed_out = true;
        break;
      }
      if (it > 64) __nanosleep(32);
    }
  }
}

// The fronts of the bottom of the tree (a set closed under descendants) in one persistent
// launch: CTAs take fronts from a device queue in level order, wait for the fronts' children
// (acquire on their done flags), factor and publish their own flag (release).  A CTA takes its
// next front, and loads its descriptor, while it works on the current one.  The unfinished
// front that comes first in the order is being worked on (its CTA has no earlier one left) and
// its children are finished, so the walk progresses whatever the number of resident CTAs.
// qctr[0]: queue head, qctr[1 + s]: done flags, zeroed before the launch.
template <int T>
__global__ void __launch_bounds__(T, T == 128 ? 3 : 1) k_front_cta_walk(DevSym S, FrontDev F,
                                                                       const FrontDesc *order, int count,
                                                                       int *qctr) {
  extern __shared__ double fsm[];
  __shared__ FrontDesc desc[2];
  __shared__ int item[2];
  int *done = qctr + 1;
  if (threadIdx.x == 0) {
    const int i = atomicAdd(qctr, 1);
    item[0] = i;
    if (i < count) desc[0] = order[i];
  }
  __syncthreads();
  for (int b = 0; item[b] < count; b ^= 1) {
    const FrontDesc d = desc[b];
    int next = 0;
    if (threadIdx.x == T - 32) next = atomicAdd(qctr, 1);
    if (threadIdx.x < 32) wait_children(S, F, d, done);
    __syncthreads();
    double *P = fsm + (T / 32) * 64;
    front_body<T / 32>(S, F, d, P, fsm, reinterpret_cast<short *>(P + front_wp(d.w) * front_ld(d.w, d.m)));
    if (threadIdx.x == T - 32) {
      item[b ^ 1] = next;
      if (next < count) desc[b ^ 1] = order[next];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      st_release_k(done + d.s, 1);
    }
  }
}

// The same at warp granularity, for the crowded levels of tiny fronts.
__global__ void __launch_bounds__(WW * 32, 3) k_front_warp_walk(DevSym S, FrontDev F, const FrontDesc *order,
                                                             int count, int *qctr, int *qhead) {
  extern __shared__ double fsm[];
  const int lane = threadIdx.x & 31;
  double *sc = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(fsm) +
                                          (size_t)(threadIdx.x >> 5) * WARP_SLICE);
  double *P = sc + 64;
  short *inv = reinterpret_cast<short *>(P + FRONT_WARP_ELEMS);
  int *done = qctr + 1;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = atomicAdd(qhead, 1);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (idx >= count) break;
    const FrontDesc d = order[idx];
    wait_children(S, F, d, done);
    __syncwarp();
    front_body<1>(S, F, d, P, sc, inv);
    __syncwarp();
    if (lane == 0) {
      __threadfence();
      st_release_k(done + d.s, 1);
    }
  }
}

// One CTA per small front of a level.
__global__ void __launch_bounds__(FT) k_front_small(DevSym S, FrontDev F, const FrontDesc *list) {
  extern __shared__ double fsm[];
  const FrontDesc d = list[blockIdx.x];
  double *P = fsm + FW * 64;
  front_body<FW>(S, F, d, P, fsm, reinterpret_cast<short *>(P + front_wp(d.w) * front_ld(d.w, d.m)));
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
                                               int nth, int tid = threadIdx.x, int bar = 0) {
  for (int i = tid; i < kids * TB; i += nth) M.ia[i >> 6][i & 63] = M.ib[i >> 6][i & 63] = -1;
  tile_sync(bar);
  for (int i = tid; i < kids * 2 * TB; i += nth) {
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
  tile_sync(bar);
}

// Extend-add into the panels of tiled supernodes: task = (s, r0, c0, first pair), a 64x64 tile
// of the panel that some child's block reaches.  Bound: memory (the blocks are read once and
// the touched tiles read and written once).
__global__ void __launch_bounds__(ET) k_front_extend(DevSym S, FrontDev F, const int4 *tasks,
                                                     const int *end, const int4 *pairs) {
  __shared__ PairMaps M;
  const int4 tk = tasks[blockIdx.x];
  const int p_end = end[blockIdx.x];
  const int s = tk.x, r0 = tk.y, c0 = tk.z;
  const int w = S.super[s + 1] - S.super[s], m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
  double *Lt = S.L + S.xptr[s] + (size_t)c0 * m + r0;
  const int row = threadIdx.x & 63, cq = threadIdx.x >> 6;   // columns cq, cq + 4, ..
  constexpr int NE = TB * TB / ET;
  pdl_trigger();
  int kids = min(FRONT_KIDS, p_end - tk.w);
  load_pair_maps(S, F, pairs, tk.w, kids, r0, c0, M, ET);   // symbolic data
  pdl_wait();
  double v[NE];
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const int col = cq + 4 * e;
    v[e] = ld_if(Lt + (size_t)col * m + row, r0 + row < m && c0 + col < w && r0 + row >= c0 + col);
  }
  for (int q = tk.w; q < p_end; q += FRONT_KIDS) {
    if (q > tk.w) {
      kids = min(FRONT_KIDS, p_end - q);
      __syncthreads();
      load_pair_maps(S, F, pairs, q, kids, r0, c0, M, ET);
    }
    for (int k = 0; k < kids; ++k) {
      const int pi = M.ia[k][row];
      const double *cb = M.cb[k] + pi;
      const int ldc = M.ld[k];
      double t[NE];
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        const int col = cq + 4 * e, pj = M.ib[k][col];
        t[e] = ld_if(cb + (int64_t)pj * ldc, pi >= 0 && pj >= 0 && r0 + row >= c0 + col);
      }
#pragma unroll
      for (int e = 0; e < NE; ++e) v[e] += t[e];
    }
  }
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const int col = cq + 4 * e;
    if (r0 + row < m && c0 + col < w && r0 + row >= c0 + col) Lt[(size_t)col * m + row] = v[e];
  }
}

// One 64x64 tile of the contribution block of s: minus L_rs L_rs^T over the columns k0 .. k1 - 1
// (DMMA) plus, at k0 = 0, the children's blocks, else what the block holds.  task = (s, i0, j0,
// first pair), offsets in the block.  The accumulator collects minus the tile's value and the
// product, and is stored back negated.
template <bool EARLY>
__device__ __forceinline__ void schur_tile(const DevSym &S, const FrontDev &F, int4 tk, int p_end,
                                           const int4 *pairs, int k0, int k1, double *stages, PairMaps &M,
                                           int tid, int bar) {
  const int s = tk.x, i0 = tk.y, j0 = tk.z;
  const int w = S.super[s + 1] - S.super[s], m = (int)(S.rowptr[s + 1] - S.rowptr[s]);
  const int r = m - w;
  double *cbs = F.cb + F.cb_off[s];
  k1 = min(k1, w);
  int kids = min(FRONT_KIDS, p_end - tk.w);
  if (k0 == 0 && kids > 0) load_pair_maps(S, F, pairs, tk.w, kids, w + i0, w + j0, M, MT, tid, bar);
  if (EARLY) pdl_wait();   // so far symbolic data
  TileAcc acc;
  if (k0 == 0) acc.zero();
  else
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int ri = i0 + acc_row(i, tid), cj = j0 + acc_col(j, e, tid);
          acc.v[i][j][e] = neg(ld_if(cbs + (int64_t)cj * r + ri, ri < r && cj <= ri));
        }
  for (int q = tk.w; q < p_end && k0 == 0; q += FRONT_KIDS) {
    if (q > tk.w) {
      kids = min(FRONT_KIDS, p_end - q);
      tile_sync(bar);
      load_pair_maps(S, F, pairs, q, kids, w + i0, w + j0, M, MT, tid, bar);
    }
    for (int k = 0; k < kids; ++k) {
      const double *cb = M.cb[k];
      const int ldc = M.ld[k];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int pi = M.ia[k][acc_row(i, tid)];
        double t[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int pj = M.ib[k][acc_col(j, e, tid)];
            t[j][e] = ld_if(cb + (int64_t)pj * ldc + pi,
                            pi >= 0 && pj >= 0 && i0 + acc_row(i, tid) >= j0 + acc_col(j, e, tid));
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) acc.v[i][j][e] -= t[j][e];
      }
    }
  }
  const double *Lr = S.L + S.xptr[s] + (size_t)k0 * m + w;
  dmma_tile_product(Lr + i0, m, min(TB, r - i0), Lr + j0, m, min(TB, r - j0), k1 - k0, stages, acc, tid, bar);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int ri = i0 + acc_row(i, tid);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cj = j0 + acc_col(j, e, tid);
        if (ri < r && cj <= ri) cbs[(size_t)cj * r + ri] = neg(acc.v[i][j][e]);
      }
  }
}

constexpr int SCHUR_SMEM = 2 * STAGE * 8;
__global__ void __launch_bounds__(MT, 4) k_front_schur(DevSym S, FrontDev F, const int4 *tasks,
                                                       const int *end, const int4 *pairs, int k0, int k1) {
  extern __shared__ double fsm[];
  __shared__ PairMaps M;
  pdl_trigger();
  schur_tile<true>(S, F, tasks[blockIdx.x], end[blockIdx.x], pairs, k0, k1, fsm, M, threadIdx.x, 0);
}

// The same beside the chain of diagonal blocks (see BG), as the panel's columns get done.
__global__ void __launch_bounds__(BG * MT, 1) k_front_schur_bg(DevSym S, FrontDev F, const int4 *tasks,
                                                               const int *end, const int4 *pairs, int count,
                                                               int k0, int k1) {
  extern __shared__ double fsm[];
  __shared__ PairMaps M[BG];
  const int grp = threadIdx.x / MT, tid = threadIdx.x - grp * MT;
  for (int q = blockIdx.x * BG + grp; q < count; q += BG * gridDim.x) {
    schur_tile<false>(S, F, tasks[q], end[q], pairs, k0, k1, fsm + grp * 2 * STAGE, M[grp], tid, 1 + grp);
    tile_sync(1 + grp);
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
  cudaError_t e = cudaFuncSetAttribute(k_front_cta_walk<FT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       200 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_cta_walk<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_small, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_warp_walk, cudaFuncAttributeMaxDynamicSharedMemorySize, WARP_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_schur, cudaFuncAttributeMaxDynamicSharedMemorySize, SCHUR_SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_schur_bg, cudaFuncAttributeMaxDynamicSharedMemorySize, BG_SMEM);
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return false;
  }
  return true;
}

int front_cta_walk_ctas(int smem, int count) {
  const int most = count >= FRONT_MANY ? resident_ctas((const void *)k_front_cta_walk<128>, 128, smem)
                                       : resident_ctas((const void *)k_front_cta_walk<FT>, FT, smem);
  return std::max(1, std::min(count, most));
}
int front_warp_walk_ctas(int count) {
  return std::max(1, std::min((count + WW - 1) / WW,
                              resident_ctas((const void *)k_front_warp_walk, WW * 32, WARP_SMEM)));
}
void launch_front_warp_walk(const DevSym &S, const FrontDev &F, const FrontDesc *order, int count,
                            int ctas, int *qctr, int *qhead, cudaStream_t st) {
  if (count > 0)
    k_front_warp_walk<<<ctas, WW * 32, WARP_SMEM, st>>>(S, F, order, count, qctr, qhead);
}
void launch_front_cta_walk(const DevSym &S, const FrontDev &F, const FrontDesc *order, int count,
                           int smem, int ctas, int *qctr, cudaStream_t st) {
  if (count >= FRONT_MANY) k_front_cta_walk<128><<<ctas, 128, smem, st>>>(S, F, order, count, qctr);
  else if (count > 0) k_front_cta_walk<FT><<<ctas, FT, smem, st>>>(S, F, order, count, qctr);
}
void launch_front_small(const DevSym &S, const FrontDev &F, const FrontDesc *list, int count, int smem,
                        cudaStream_t st) {
  if (count > 0) k_front_small<<<count, FT, smem, st>>>(S, F, list);
}
void launch_front_extend(const DevSym &S, const FrontDev &F, const int4 *tasks, const int *end,
                         const int4 *pairs, int count, LaunchQueue q) {
  if (count > 0) launch_early(q, 1, k_front_extend, count, ET, 0, S, F, tasks, end, pairs);
}
void launch_front_schur(const DevSym &S, const FrontDev &F, const int4 *tasks, const int *end,
                        const int4 *pairs, int count, int k0, int k1, int bg_ctas, LaunchQueue q) {
  if (count <= 0) return;
  if (bg_ctas > 0)
    k_front_schur_bg<<<std::min(bg_ctas, (count + BG - 1) / BG), BG * MT, BG_SMEM, q.st>>>(S, F, tasks, end, pairs,
                                                                                        count, k0, k1);
  else
    launch_early(q, 1, k_front_schur, count, MT, SCHUR_SMEM, S, F, tasks, end, pairs, k0, k1);
}

}  // namespace swc
