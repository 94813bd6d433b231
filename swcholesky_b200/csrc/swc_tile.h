// Device helpers shared by the FP64 factorization kernels: release/acquire flags, the FP64
// tensor-core (DMMA) 64x64 tile product and the 8x8 Cholesky every dense kernel is built on.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "swc_engine.h"

namespace swc {

namespace {

__device__ __forceinline__ int lbound(const int *a, int len, int key) {
  int lo = 0, hi = len;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ int ld_acquire_k(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_k(int *p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Programmatic launches: a kernel's CTAs start while the one before still runs, and pdl_wait waits
// until that one (and so all before it, every kernel having waited itself) has finished, its writes
// visible.  The solves' kernels ask for their parts of L first, which no solve changes.  A captured
// launch behind events of other streams waits for those kernels at pdl_wait too, not at its start:
// nothing that any earlier kernel of the sequence writes is read before it.  The trigger stands
// first: the waiting CTAs take only what the running kernel's CTAs, all started by then, leave free.
// With this and the predicated loads a solve of the 301 x 287 grid with eight right-hand sides went
// from 435 to 370 us, one of the 60^3 grid with one from 1158 to 1124 us (B200).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// *p where ok, else 0: one predicated load.  A branch around a load that is summed at once makes
// the warp wait for it before the next one; these are all in flight together.
__device__ __forceinline__ double ld_if(const double *p, bool ok) {
  double v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
               "@q ld.global.f64 %0, [%1];\n\t}\n"
               : "=d"(v)
               : "l"(p), "r"((int)ok));
  return v;
}

constexpr int KC = 16;

// 64x64 FP64 tile product on the tensor cores (DMMA, mma.sync m8n8k4 .f64):
//   C[i][j] = sum_k A[i][k] * B[j][k],  A = rows [0,na) of a column-major panel (lda),
//                                       B = rows [0,nb) of a column-major panel (ldb).
// 128 threads = 4 warps in a 2x2 grid, each warp a 32x32 sub-tile of 4x4 MMA tiles.
// Operands stream through shared memory in k-chunks of KC columns with a two-stage
// cp.async pipeline; rows beyond na / nb and columns beyond K are zero-filled.
// Fragment layout of m8n8k4 .f64: A[lane/4][lane%4], B[k = lane%4][n = lane/4],
// C[lane/4][2*(lane%4) + e].
constexpr int MT = 128;               // threads of the tensor-core tile kernels
constexpr int LDS = TB + 4;           // padded row of a staged k-slice: 64-bit fragment loads conflict-free
constexpr int STAGE = 2 * KC * LDS;   // doubles per pipeline stage (A and B slices)
// Tile launches that run beside the chain of diagonal blocks: one CTA per SM of three groups, so the
// SMs the launch leaves free stay free.  It asks for more than half of an SM's 228 KB of shared memory
// (1 KB of it per CTA is the system's), whatever its registers would allow; its stages need 102 KB.
constexpr int SM_SMEM = 228 * 1024;
constexpr int BG = 3, BG_SMEM = SM_SMEM / 2;
static_assert(BG_SMEM >= BG * 2 * STAGE * 8 && 2 * (BG_SMEM + 1024) > SM_SMEM, "the stages fit, a second CTA does not");
static_assert(MT == 2 * TB, "staging pattern: two threads per tile row");

__device__ __forceinline__ void cp_async8(double *smem, const double *gmem, bool pred) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int sz = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

struct TileAcc {
  double v[4][4][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j][0] = v[i][j][1] = 0.0;
  }
};

// The tile functions run on 128 threads: a whole block (bar 0), or one of several groups of a
// block, with the thread's index in its group and a named barrier of its own.
__device__ __forceinline__ void tile_sync(int bar) {
  if (bar == 0) __syncthreads();
  else asm volatile("bar.sync %0, 128;\n" ::"r"(bar) : "memory");
}

// Thread t copies tile row t % 64 at chunk offsets t / 64, t / 64 + 2, ... (one pointer
// step per copy).
__device__ __forceinline__ void load_chunk(const double *__restrict__ Pa, int lda, int na,
                                           const double *__restrict__ Pb, int ldb, int nb,
                                           int K, int k0, double *st, int tid) {
  const int i = tid & (TB - 1), kq = tid >> 6;
  double *As = st + kq * LDS + i, *Bs = st + KC * LDS + kq * LDS + i;
  const double *pa = Pa + (size_t)(k0 + kq) * lda + i, *pb = Pb + (size_t)(k0 + kq) * ldb + i;
  const bool ina = i < na, inb = i < nb;
#pragma unroll
  for (int it = 0; it < KC / 2; ++it) {
    const bool kin = k0 + kq + 2 * it < K;
    cp_async8(As + 2 * it * LDS, kin && ina ? pa : Pa, kin && ina);
    cp_async8(Bs + 2 * it * LDS, kin && inb ? pb : Pb, kin && inb);
    pa += (size_t)2 * lda;
    pb += (size_t)2 * ldb;
  }
  cp_async_commit();
}

// BEGUN: the caller has synchronised and asked for chunk 0 itself, before loads of its own.
template <bool BEGUN = false>
__device__ __forceinline__ void dmma_tile_product(const double *__restrict__ Pa, int lda, int na,
                                                  const double *__restrict__ Pb, int ldb, int nb,
                                                  int K, double *stages, TileAcc &acc,
                                                  int tid = threadIdx.x, int bar = 0) {
  const int lane = tid & 31, warp = tid >> 5;
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32;
  const int kq = lane & 3, g = lane >> 2;
  const int nchunks = (K + KC - 1) / KC;
  if (!BEGUN) {
    tile_sync(bar);   // stages free (previous users done)
    load_chunk(Pa, lda, na, Pb, ldb, nb, K, 0, stages, tid);
  }
  for (int c = 0; c < nchunks; ++c) {
    if (c + 1 < nchunks) {
      load_chunk(Pa, lda, na, Pb, ldb, nb, K, (c + 1) * KC, stages + ((c + 1) & 1) * STAGE, tid);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    tile_sync(bar);
    const double *As = stages + (c & 1) * STAGE, *Bs = As + KC * LDS;
#pragma unroll
    for (int k4 = 0; k4 < KC; k4 += 4) {
      double a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[(k4 + kq) * LDS + wr + 8 * i + g];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[(k4 + kq) * LDS + wc + 8 * j + g];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma(acc.v[i][j], a[i], b[j]);
    }
    tile_sync(bar);
  }
}

// acc += A B^T of operands in shared memory ([k][row] and [k][column], leading dimension LDS),
// K a multiple of 4, by the same four warps.
__device__ __forceinline__ void dmma_tile_smem(const double *As, const double *Bs, int K, TileAcc &acc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32;
  const int kq = lane & 3, g = lane >> 2;
  for (int k4 = 0; k4 < K; k4 += 4) {
    double a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = As[(k4 + kq) * LDS + wr + 8 * i + g];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = Bs[(k4 + kq) * LDS + wc + 8 * j + g];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dmma(acc.v[i][j], a[i], b[j]);
  }
}

// Sign flip through the integer pipe (FP64 arithmetic outside the tensor cores is slow).
__device__ __forceinline__ double neg(double x) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ULL);
}

// Position of accumulator element (i, j, e) of this thread inside the 64x64 tile.
__device__ __forceinline__ int acc_row(int i, int tid = threadIdx.x) {
  return ((tid >> 5) >> 1) * 32 + 8 * i + ((tid & 31) >> 2);
}
__device__ __forceinline__ int acc_col(int j, int e, int tid = threadIdx.x) {
  return ((tid >> 5) & 1) * 32 + 8 * j + 2 * (tid & 3) + e;
}

// Cholesky of a panel in shared memory by NW = 1, 4 or 8 warps: P is [column][row] with
// leading dimension ld, nkb 8-column blocks, nrb >= nkb 8-row blocks (padding: identity in the
// diagonal blocks, zeros below).  The chain of pivots sets the time, so nothing else is on it:
// each panel warp factors the 8x8 diagonal block by itself in registers (broadcast loads, no
// shuffle, no barrier) and takes its own rows' columns along in the same instructions (32 rows
// per warp, one per lane; further rows follow once the block is known).  One barrier per 8
// columns is left, after which each panel warp updates its own rows and, privately, the next
// diagonal block (8x8x4 DMMA).  Four panel warps, one per scheduler: with eight, two shared an
// FP64 unit and the chain took 1.4 times as long.  With NW = 8 warps 4-7 update the columns
// beyond the next block, beside the next pivots.  Panel warp p owns the row blocks congruent to
// p mod NP.  sc: 64 doubles per warp.  A pivot of one of the first `real` columns that is <= 0
// or NaN is reported in status[0] (gcol: the panel's first column).  rd (optional): the
// reciprocals of the diagonal, one per column.
template <int NW>
__device__ __forceinline__ void chol_panel(double *P, int ld, int nkb, int nrb, double *sc, int *status,
                                           int gcol, int real, double *rd = nullptr) {
  constexpr int NP = NW == 1 ? 1 : 4;   // panel warps
  const int lane = threadIdx.x & 31, warp = NW == 1 ? 0 : (int)(threadIdx.x >> 5);
  const int g = lane >> 2, kq = lane & 3, sub = lane & 7, sb = lane >> 3;
  sc += warp * 64;
  // minus X_kb X_kb^T on the blocks (bi, bj), bj in [jlo, jhi), of the row blocks own, own + NP,
  // .. (except the block (skip, skip)), two row blocks by two column blocks at a time
  auto update = [&](int k0, int own, int jlo, int jhi, int skip) {
    for (int i0 = own; i0 < nrb; i0 += 2 * NP)
      for (int j0 = jlo; j0 < jhi && j0 <= i0 + NP; j0 += 2) {
        double c[2][2][2];
        bool on[2][2];
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int bi = i0 + p * NP, bj = j0 + q;
            on[p][q] = bi < nrb && bj < jhi && bj <= bi && !(bi == skip && bj == skip);
            if (on[p][q]) {
              c[p][q][0] = P[(8 * bj + 2 * kq) * ld + 8 * bi + g];
              c[p][q][1] = P[(8 * bj + 2 * kq + 1) * ld + 8 * bi + g];
            }
          }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = (k0 + 4 * h + kq) * ld + g;
          double av[2], bv[2];
#pragma unroll
          for (int p = 0; p < 2; ++p) av[p] = i0 + p * NP < nrb ? P[col + 8 * (i0 + p * NP)] : 0.0;
#pragma unroll
          for (int q = 0; q < 2; ++q) bv[q] = j0 + q < jhi ? neg(P[col + 8 * (j0 + q)]) : 0.0;
#pragma unroll
          for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int q = 0; q < 2; ++q)
              if (on[p][q]) dmma(c[p][q], av[p], bv[q]);
        }
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int q = 0; q < 2; ++q)
            if (on[p][q]) {
              const int bi = i0 + p * NP, bj = j0 + q;
              P[(8 * bj + 2 * kq) * ld + 8 * bi + g] = c[p][q][0];
              P[(8 * bj + 2 * kq + 1) * ld + 8 * bi + g] = c[p][q][1];
            }
      }
  };
  if (NW > NP && warp >= NP) {   // trailing warps
    for (int kb = 0; kb < nkb; ++kb) {
      __syncthreads();
      if (kb + 2 < nkb) update(8 * kb, kb + 2 + ((warp - kb - 2) & (NP - 1)), kb + 2, nkb, -1);
    }
    __syncthreads();
    return;
  }
  for (int kb = 0; kb < nkb; ++kb) {
    const int k0 = 8 * kb, nb = kb + 1;
    const double *dg = kb == 0 ? P : sc;
    const int ldd = kb == 0 ? ld : 8;
    double a[8][8], rinv[8], x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = j; i < 8; ++i) a[i][j] = dg[j * ldd + i];
    const int ib0 = nb + ((warp - nb) & (NP - 1));   // this warp's first row block below
    int ib = ib0 + NP * sb;
    double *row = P + k0 * ld + 8 * ib + sub;
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = ib < nrb ? row[j * ld] : 0.0;
    int bad = 8;
    double inv = rsqrt(a[0][0]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const double piv = a[j][j];
      if (!(piv > 0.0) && j < bad) bad = j;
      rinv[j] = inv;
      a[j][j] = piv * inv;
      // the chain first: the next pivot and its reciprocal square root
      if (j + 1 < 8) {
        a[j + 1][j] *= inv;
        a[j + 1][j + 1] = fma(-a[j + 1][j], a[j + 1][j], a[j + 1][j + 1]);
      }
      const double inv_next = (j + 1 < 8) ? rsqrt(a[j + 1][j + 1]) : 0.0;
#pragma unroll
      for (int i = j + 2; i < 8; ++i) a[i][j] *= inv;
#pragma unroll
      for (int k = j + 1; k < 8; ++k)
#pragma unroll
        for (int i = k; i < 8; ++i)
          if (!(k == j + 1 && i == j + 1)) a[i][k] = fma(-a[i][j], a[k][j], a[i][k]);
      x[j] *= inv;
#pragma unroll
      for (int k = j + 1; k < 8; ++k) x[k] = fma(-x[j], a[k][j], x[k]);
      inv = inv_next;
    }
    if (warp == 0 && lane == 0 && bad < 8 && k0 + bad < real) atomicMin(&status[0], gcol + k0 + bad + 1);
    if (ib < nrb) {
#pragma unroll
      for (int j = 0; j < 8; ++j) row[j * ld] = x[j];
    }
    for (int ibc = ib0 + 4 * NP; ibc < nrb; ibc += 4 * NP) {   // rows beyond the first 32
      ib += 4 * NP;
      if (ib >= nrb) continue;
      double *rw = P + k0 * ld + 8 * ib + sub;
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = rw[j * ld];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        x[j] *= rinv[j];
#pragma unroll
        for (int k = j + 1; k < 8; ++k) x[k] = fma(-x[j], a[k][j], x[k]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) rw[j * ld] = x[j];
    }
    if (NW == 1) __syncwarp(); else __syncthreads();
    if (warp == (kb & (NP - 1))) {   // no warp reads the block any more
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = j; i < 8; ++i) P[(k0 + j) * ld + k0 + i] = a[i][j];
      if (rd && lane == 0)
#pragma unroll
        for (int j = 0; j < 8; ++j) rd[k0 + j] = rinv[j];
    }
    if (nb >= nkb) break;
    {
      double c[2];   // the next diagonal block, updated privately
      c[0] = P[(8 * nb + 2 * kq) * ld + 8 * nb + g];
      c[1] = P[(8 * nb + 2 * kq + 1) * ld + 8 * nb + g];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double v = P[(k0 + 4 * h + kq) * ld + 8 * nb + g];
        dmma(c, v, neg(v));
      }
      sc[(2 * kq) * 8 + g] = c[0];
      sc[(2 * kq + 1) * 8 + g] = c[1];
    }
    update(k0, ib0, nb, NW > NP ? nb + 1 : nkb, nb);
    __syncwarp();
  }
  if (NW == 1) __syncwarp(); else __syncthreads();
}

// Inverse of the 64x64 lower triangle D ([column][row], leading dimension LDS; rd: reciprocals of
// its diagonal) into the lower 8x8 blocks of E (same layout), by doubling: the 8x8 diagonal
// blocks by substitution, then T21 = -T22 (L21 T11) at 16, 32 and 64 columns, two products and
// two barriers each (W: the inner product, 16 blocks of 64 doubles).
template <int NW>
__device__ __forceinline__ void inverse64(const double *D, const double *rd, double *E, double *W) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, kq = lane & 3;
  if (tid < TB) {   // thread: one column of a diagonal block
    const int b0 = tid & ~7, j = tid & 7;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = i == j ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      x[k] *= rd[b0 + k];
#pragma unroll
      for (int i = k + 1; i < 8; ++i) x[i] = fma(-D[(b0 + k) * LDS + b0 + i], x[k], x[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) E[tid * LDS + b0 + i] = x[i];
  }
  __syncthreads();
#pragma unroll
  for (int h = 1; h <= 4; h *= 2) {
    // tile t: pair t / h^2, block (i, k) of the pair's lower left part
    for (int t = warp; t < 4 * h; t += NW) {
      const int base = 2 * h * (t / (h * h)), i = (t % (h * h)) / h, k = t % h;
      double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
      for (int j = 0; j < h; ++j)
        if (j >= k)
#pragma unroll
          for (int u = 0; u < 2; ++u)
            dmma(c[u], D[(8 * (base + j) + 4 * u + kq) * LDS + 8 * (base + h + i) + g],
                 E[(8 * (base + k) + g) * LDS + 8 * (base + j) + 4 * u + kq]);
      W[t * 64 + (2 * kq) * 8 + g] = c[0][0] + c[1][0];
      W[t * 64 + (2 * kq + 1) * 8 + g] = c[0][1] + c[1][1];
    }
    __syncthreads();
    for (int t = warp; t < 4 * h; t += NW) {
      const int base = 2 * h * (t / (h * h)), i = (t % (h * h)) / h, k = t % h;
      double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
      for (int j = 0; j < h; ++j)
        if (j <= i)
#pragma unroll
          for (int u = 0; u < 2; ++u)
            dmma(c[u], neg(E[(8 * (base + h + j) + 4 * u + kq) * LDS + 8 * (base + h + i) + g]),
                 W[((t / (h * h)) * h * h + j * h + k) * 64 + g * 8 + 4 * u + kq]);
      E[(8 * (base + k) + 2 * kq) * LDS + 8 * (base + h + i) + g] = c[0][0] + c[1][0];
      E[(8 * (base + k) + 2 * kq + 1) * LDS + 8 * (base + h + i) + g] = c[0][1] + c[1][1];
    }
    __syncthreads();
  }
}

}  // namespace

}  // namespace swc
