// Device helpers of the chained triangular solves: counters in global memory, staged copies,
// thread-block clusters.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "swc_engine.h"

namespace swc {

namespace {

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void red_release_add(int *p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Lane u < nf polls the counter at flag + dir * u (no sleep between polls: a hop between
// clusters is on the chain's critical path) until the first one has reached `target`;
// returns how many consecutive counters from the first have reached it (1 .. nf), or 0
// after a timeout (its own, or one another block recorded).  A batch is never held back
// by a block that is not finished yet.
__device__ int warp_wait_prefix(const int *flag, int dir, int nf, int target, int *status) {
  const long long budget = wait_budget(status);
  long long it = 0;
  const int lane = threadIdx.x & 31;
  bool mine = lane < nf && ld_acquire(flag + dir * lane) >= target;
  int n = 0;
  for (;;) {
    const unsigned done = __ballot_sync(0xffffffffu, mine);
    n = min(nf, __ffs(~done) - 1);
    if (n > 0) break;
    if (++it > budget || ((it & 31) == 0 && *(volatile int *)&status[2])) {
      if (lane == 0) atomicExch(&status[2], 1);
      break;
    }
    if (lane < nf && !mine) mine = ld_acquire(flag + dir * lane) >= target;
  }
  __syncwarp();   // the lanes' later loads are ordered after the polling lanes' acquires
  return n;
}

template <int N>
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }
// an empty cp.async group (keeps one group per ring step)
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp8(double *dst, const double *src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 8 : 0));
}

__device__ __forceinline__ uint32_t chain_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::
                   : "memory");
}
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// address of the same shared-memory location in the CTA of cluster rank `rank`
__device__ __forceinline__ uint32_t cluster_addr(const void *p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(smem_addr(p)), "r"(rank));
  return r;
}
// `count` mbarriers that each complete once with `bytes` transaction bytes, visible to the
// whole cluster afterwards.
__device__ __forceinline__ void cluster_bars_init(unsigned long long *bars, int count, int bytes) {
  if (threadIdx.x == 0) {
    for (int j = 0; j < count; ++j) {
      const uint32_t b = smem_addr(&bars[j]);
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(b) : "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(b), "r"(bytes)
                   : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  cluster_sync_all();
}
// Every lane waits (bounded) for the barrier's bytes; false after a timeout (its own, or one
// another block recorded) in any lane.
__device__ bool warp_bar_recv(const unsigned long long *bar, int *status) {
  const uint32_t b = smem_addr(bar);
  const long long budget = wait_budget(status);
  long long it = 0;
  int ok = 1;
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], 0;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}\n"
        : "=r"(done)
        : "r"(b)
        : "memory");
    if (done) break;
    if (++it > budget || ((it & 31) == 0 && *(volatile int *)&status[2])) {
      atomicExch(&status[2], 1);
      ok = 0;
      break;
    }
  }
  return __all_sync(0xffffffffu, ok) != 0;
}

}  // namespace

}  // namespace swc
