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

// Thread t copies tile row t % 64 at chunk offsets t / 64, t / 64 + 2, ... (one pointer
// step per copy).
__device__ __forceinline__ void load_chunk(const double *__restrict__ Pa, int lda, int na,
                                           const double *__restrict__ Pb, int ldb, int nb,
                                           int K, int k0, double *st) {
  const int i = threadIdx.x & (TB - 1), kq = threadIdx.x >> 6;
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

__device__ __forceinline__ void dmma_tile_product(const double *__restrict__ Pa, int lda, int na,
                                                  const double *__restrict__ Pb, int ldb, int nb,
                                                  int K, double *stages, TileAcc &acc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32;
  const int kq = lane & 3, g = lane >> 2;
  const int nchunks = (K + KC - 1) / KC;
  __syncthreads();   // stages free (previous users done)
  load_chunk(Pa, lda, na, Pb, ldb, nb, K, 0, stages);
  for (int c = 0; c < nchunks; ++c) {
    if (c + 1 < nchunks) {
      load_chunk(Pa, lda, na, Pb, ldb, nb, K, (c + 1) * KC, stages + ((c + 1) & 1) * STAGE);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
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
    __syncthreads();
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
__device__ __forceinline__ int acc_row(int i) {
  return ((threadIdx.x >> 5) >> 1) * 32 + 8 * i + ((threadIdx.x & 31) >> 2);
}
__device__ __forceinline__ int acc_col(int j, int e) {
  return ((threadIdx.x >> 5) & 1) * 32 + 8 * j + 2 * (threadIdx.x & 3) + e;
}

// Warp-level Cholesky of an 8x8 diagonal block (D points at its first entry, [column][row]
// with leading dimension ld) and its inverse into T (8x8, column-major).  A pivot of one of
// the first `real` columns that is <= 0 or NaN is reported (gcol: the block's first column).  Every lane factors the whole block in registers (broadcast loads of its 36
// entries), so the chain of pivots is one reciprocal square root, one product and one
// FMA per column with no shuffle on it; lane j < 8 then forms column j of the inverse by
// forward substitution.
__device__ __forceinline__ void potrf8_inv8(double *D, int ld, double *T, int *status, int gcol,
                                            int real) {
  const int lane = threadIdx.x & 31;
  double a[8][8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = j; i < 8; ++i) a[i][j] = D[j * ld + i];
  double rinv[8];
  int bad = 8;   // first column with a pivot <= 0 or NaN (reported after the chain)
  double inv = rsqrt(a[0][0]);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const double piv = a[j][j];
    if (!(piv > 0.0) && j < bad) bad = j;
    rinv[j] = inv;
    a[j][j] = piv * inv;
    // the chain first: the next pivot and its reciprocal square root, issued before the
    // rest of the column's update, which runs under its latency
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
    inv = inv_next;
  }
  if (lane == 0 && bad < 8 && bad < real) atomicMin(&status[0], gcol + bad + 1);
  // every lane stores the same 36 values (one write per address; no lane-dependent index
  // into a[][], which would move the array to local memory), once every lane has loaded them:
  // the lanes of a warp need not run in step
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = j; i < 8; ++i) D[j * ld + i] = a[i][j];
  // lane j < 8: column j of the inverse, 1/L(i,i) = rinv[i]
  const int j = lane & 7;
  double t[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    double sacc = 0.0;
#pragma unroll
    for (int k = 0; k < i; ++k)
      if (k >= j) sacc = fma(a[i][k], t[k], sacc);
    t[i] = (i < j) ? 0.0 : ((i == j) ? rinv[i] : -sacc * rinv[i]);
  }
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) T[j * 8 + i] = t[i];
  }
  __syncwarp();
}

}  // namespace

}  // namespace swc
