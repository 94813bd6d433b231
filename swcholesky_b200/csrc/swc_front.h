// Multifrontal FP64 factorization: plan (host) and launches.
//
// Every supernode s passes ONE dense contribution block to its parent in the supernodal
// elimination tree: CB_s = (contribution blocks of s's children, at s's off-diagonal rows)
// - L_rs L_rs^T, over the r = m - w off-diagonal rows of s (lower triangle, column-major,
// leading dimension r).  A front is assembled from A and the two or three blocks of its
// children instead of from every descendant that touches it (the prune set: up to hundreds
// of narrow panels per supernode, each located by its own row search), and every product is
// a dense one over contiguous rows.  Blocks are added in child order: no atomics, and the
// factor is reproducible bit for bit.  Against the left-looking kernels (B200, ms per
// factorization): 5-point grids 20 x 20 0.50 -> 0.13, 100 x 100 1.81 -> 0.42; 7-point grids
// 41 x 37 x 43 5.43 -> 3.41, 60^3 24.7 -> 16.3 (the descendants' updates 16.3 -> 6.4);
// 3-unknown 27-point grid 24 x 23 x 22 5.56 -> 3.60.  The blocks alive at once take once to twice
// the memory of L on grids and geometric graphs, but r x r doubles per front whatever its width:
// many narrow supernodes under a wide border would take hundreds of times L, and stay left-looking
// (front_memory_limit).  So do handles that cannot have the memory, prune sets that are not the
// complete descendant lists, and the mixed modes.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "swc_engine.h"

namespace swc {

// Fronts done by one warp: padded panel of at most FRONT_WARP_ELEMS doubles, at most FRONT_WARP_M
// rows.
constexpr int FRONT_WARP_ELEMS = 1280;
constexpr int FRONT_WARP_M = 128;
constexpr int FRONT_KIDS = 4;   // children whose row maps are held at a time
// Fronts of the warp kernels sit on levels of at least this many of them: below, a CTA per front
// finishes the level sooner than warps that leave the SMs idle.
constexpr int FRONT_WARP_LEVEL_MIN = 1024;

// Padded front in shared memory: the w columns padded to a multiple of 8 (identity), the
// off-diagonal rows below them, and a leading dimension of 4 mod 16 doubles, with which the
// 8x8 DMMA operand loads meet no bank conflict.
__host__ __device__ inline int front_wp(int w) { return (w + 7) & ~7; }
__host__ __device__ inline int front_ld(int w, int m) {
  const int rows = front_wp(w) + ((m - w + 7) & ~7);
  return rows + ((4 - rows) & 15);
}
inline int64_t front_smem(int w, int64_t m) {
  return 8LL * front_wp(w) * front_ld(w, (int)m) + 8 * 8 * 64 + 2LL * FRONT_KIDS * ((m + 3) & ~3LL);
}

// The adjoint's small fronts: padded panel, a second one (at least 64 doubles per warp), the
// inverse of the diagonal block (leading dimension 4 mod 16), the row map.
__host__ __device__ inline int adj_ldt(int w) { return front_wp(w) + ((4 - front_wp(w)) & 15); }
inline int64_t adj_small_smem(int w, int64_t m, bool y_global) {
  const int64_t pe = (int64_t)front_wp(w) * front_ld(w, (int)m);
  return 8 * (pe + (pe > 512 && !y_global ? pe : 512) + (int64_t)front_wp(w) * adj_ldt(w)) + 4 * (m + 1);
}

// Doubles that blocks alive together may take: four times L (measured: 5-point grids up to 2.2
// times, 7-point 1.0 to 2.0, 3-unknown 27-point 1.2 to 3.3, random geometric graphs 0.8 to 1.3), or
// 256 MB where L is small.  Beyond are bordered structures: 4,000 columns under a border of 1,000 take
// 800 times L.
inline int64_t front_memory_limit(int64_t xsize) {
  const int64_t floor = (int64_t)1 << 25;
  return 4 * xsize > floor ? 4 * xsize : floor;
}

// Placement of blocks that live over a range of waves: the first free place that fits while there are
// FEW, then the smallest, in logarithmic time (batches free and place a hundred thousand small blocks
// level by level; for small structures the index would cost more than it saves).
class FrontArena {
 public:
  int64_t take(int64_t len);
  void give(int64_t at, int64_t len);
  int64_t end() const { return end_; }

 private:
  static constexpr size_t FEW = 256;
  void put(int64_t at, int64_t len);
  std::map<int64_t, int64_t>::iterator drop(std::map<int64_t, int64_t>::iterator it);
  std::map<int64_t, int64_t> free_;                    // length by place
  std::set<std::pair<int64_t, int64_t>> by_len_;       // (length, place), once indexed_
  bool indexed_ = false;
  int64_t end_ = 0;
};

// What a front's kernel needs to know, in one load each: the front (in list order), and its
// children (in child_ptr order).
struct __align__(16) FrontDesc {
  int s, f, w, m;
  int ch0, ch1, a0, a1;            // children, entries of A in its columns
  int64_t xoff, cb;                // offsets in L and in the contribution blocks
};
struct __align__(16) FrontChild {
  int s, rc, n1, pad;              // supernode, rows of its block, rows that are columns of the parent
  int64_t rel, cb;                 // offsets of its row map and of its block
};

// Device view of the plan.
struct FrontDev {
  const FrontChild *child;
  const int *rel;                 // per off-diagonal row (at rowptr[s] - super[s]): position in
                                  // the parent's row list
  const int *ppos;                // per entry of A in a small front: its place in the padded panel
                                  // (-1: outside the pattern)
  const int64_t *cb_off;          // per supernode: its contribution block in cb
  double *cb;
};

struct FrontWave {
  int small_off = 0, small_cnt = 0, small_smem = 0;
  int ext_off = 0, ext_cnt = 0;    // tiles of tiled panels that receive children's blocks
  int sch_off = 0, sch_cnt = 0;    // tiles of contribution blocks, wide fronts first
  std::vector<int> sch_more;       // [b]: the tiles of fronts with more than b column blocks
  int sch_steps = 0;               // column blocks per part when formed beside the dense steps (0:
                                   // in one launch after them)
};

// The contribution blocks of a wave are formed in parts of a quarter of its steps (at least
// FRONT_BG_STEPS), on all but FRONT_BG_RESERVE SMs, beside the chain of diagonal blocks (about
// FRONT_STEP_US per 64 columns), where that chain is what the wave waits for: its dense products
// at FRONT_FLOPS_US flops per us take at most 1.5 times as long.  Waves of few small fronts
// gain (24 x 23 x 22 3-unknown grid 3249 -> 3155 us, 41 x 37 x 43 7-point grid 3072 -> 3039);
// with more work the launches only disturb each other (60^3: 14.6 -> 16.2 ms).
constexpr int FRONT_BG_STEPS = 3, FRONT_BG_RESERVE = 40;
constexpr double FRONT_STEP_US = 22.0, FRONT_FLOPS_US = 28e6;

struct FrontPlan {
  bool closed = false;             // the tree below holds: children's rows among the parent's
  bool ok = false;                 // the factorization allows it (see build_front_plan)
  std::vector<int> child_ptr, child, child_n1, rel;
  std::vector<int> apos;           // per entry of A: position in its column's row list (-1: none)
  std::vector<int> ppos;           // see FrontDev
  std::vector<FrontChild> kids;    // in child order
  std::vector<FrontDesc> warp_desc, cta_desc, small_desc;
  std::vector<int64_t> cb_off;
  int64_t cb_len = 0;              // doubles of contribution blocks alive at once
  std::vector<int> warp_list;      // fronts of the warp walk, in level order
  std::vector<int> cta_list;       // fronts of the CTA walk, in level order
  int cta_smem = 0;
  std::vector<int> small_list;     // per wave; ~s: its contribution block is formed by tiles
  std::vector<FrontWave> waves;
  std::vector<int4> ext_tasks, sch_tasks;   // (s, r0, c0, first pair)
  std::vector<int> ext_end, sch_end;        // one past the last pair
  std::vector<int4> ext_pairs, sch_pairs;   // (child, a0, b0, na | nb << 16)
  int launches = 0;
  KernelStats work;                // algorithmic flops (products; a child's entry added is not counted)
                                   // and bytes per kernel class
};

// Derives the multifrontal plan of an analysed structure.  P.ok stays false, and the
// left-looking kernels are used, when the prune sets are not exactly the descendants that
// touch each supernode, a child's rows are not among its parent's, or the blocks would take more
// than front_memory_limit.
void build_front_plan(int n, const int *c, const int *r, const int *Ls, const int *prunePtr,
                      const int *pruneSet, const HostSym &H, const Plan &P, const Tuning &T,
                      FrontPlan &F);

// Host check of a multifrontal plan: every front factored once, after its children; every
// entry of every child's block added once (to the panel by the front's own launch or by a
// panel tile, to the parent's block likewise); every block tile formed once; the shared memory
// of every launch sufficient; no two blocks alive in one place.  False with a message on the
// first violation (true for a plan that is not ok).
bool check_front_plan(int n, const int *Ls, const HostSym &H, const Plan &P, const FrontPlan &F,
                      std::string &err);

// Host check of the adjoint's reverse sweep (a no-op where the tree does not hold): every
// supernode once, after its parent; every wide one's column blocks, their rows and its gradient's
// columns each once, the last block first; no two fronts held in one place.
bool check_adjoint_plan(const HostSym &H, const Plan &P, const FrontPlan &F, std::string &err);

bool front_configure(std::string &err);
int front_cta_walk_ctas(int smem, int count);
int front_warp_walk_ctas(int count);
void launch_front_warp_walk(const DevSym &S, const FrontDev &F, const FrontDesc *order, int count,
                            int ctas, int *qctr, int *qhead, cudaStream_t st);
void launch_front_cta_walk(const DevSym &S, const FrontDev &F, const FrontDesc *order, int count,
                           int smem, int ctas, int *qctr, cudaStream_t st);
void launch_front_small(const DevSym &S, const FrontDev &F, const FrontDesc *list, int count, int smem,
                        cudaStream_t st);   // cb < 0: the block is formed by tiles
void launch_front_extend(const DevSym &S, const FrontDev &F, const int4 *tasks, const int *end,
                         const int4 *pairs, int count, LaunchQueue q);
// tiles of contribution blocks over the columns k0 .. k1 - 1 of each front (k1 beyond a front's
// width: to its end); bg_ctas > 0: at most that many CTAs of one per SM, beside other kernels
void launch_front_schur(const DevSym &S, const FrontDev &F, const int4 *tasks, const int *end,
                        const int4 *pairs, int count, int k0, int k1, int bg_ctas, LaunchQueue q);

}  // namespace swc
