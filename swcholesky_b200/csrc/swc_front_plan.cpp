// Host side of the multifrontal factorization: validity of the structure, the children's row
// maps, the walks, the tile tasks and the placement of the contribution blocks.
#include <algorithm>
#include <map>

#include "swc_front.h"

namespace swc {

namespace {

// Largest contribution block a walk's CTA forms by itself, and a level launch's; larger ones
// go to 64x64 tiles over the whole GPU.
constexpr int FRONT_WALK_R = 512;
constexpr int FRONT_SMALL_R = 192;

// Every supernode's prune set is exactly the set of supernodes with a row among its columns.
bool prune_sets_complete(const int *Ls, const int *prunePtr, const int *pruneSet, const HostSym &H,
                         const std::vector<int> &col2sup) {
  const int ns = (int)H.super.size() - 1;
  std::vector<int> touches(ns, 0), seen(ns, -1);
  for (int d = 0; d < ns; ++d) {
    int last = -1;
    for (int64_t q = H.rowptr[d] + (H.super[d + 1] - H.super[d]); q < H.rowptr[d + 1]; ++q) {
      const int s = col2sup[Ls[q]];
      if (s != last) ++touches[s];
      last = s;
    }
  }
  for (int s = 0; s < ns; ++s) {
    int real = 0;
    for (int q = prunePtr[s]; q < prunePtr[s + 1]; ++q) {
      const int d = pruneSet[q];
      if (H.upd_lbub[q].y <= H.upd_lbub[q].x) continue;   // touches nothing of s
      if (seen[d] == s) return false;                     // listed twice
      seen[d] = s;
      ++real;
    }
    if (real != touches[s]) return false;
  }
  return true;
}

}  // namespace

int64_t FrontArena::take(int64_t len) {
  if (!indexed_ && free_.size() > FEW) {
    for (const auto &f : free_) by_len_.insert({f.second, f.first});
    indexed_ = true;
  }
  auto it = free_.begin();
  if (indexed_) {
    const auto fit = by_len_.lower_bound({len, 0});
    it = fit == by_len_.end() ? free_.end() : free_.find(fit->second);
  } else {
    while (it != free_.end() && it->second < len) ++it;
  }
  if (it == free_.end()) {
    const int64_t at = end_;
    end_ += len;
    return at;
  }
  const int64_t at = it->first, rest = it->second - len;
  drop(it);
  if (rest) put(at + len, rest);
  return at;
}

void FrontArena::put(int64_t at, int64_t len) {
  free_.emplace(at, len);
  if (indexed_) by_len_.insert({len, at});
}

std::map<int64_t, int64_t>::iterator FrontArena::drop(std::map<int64_t, int64_t>::iterator it) {
  if (indexed_) by_len_.erase({it->second, it->first});
  return free_.erase(it);
}

void FrontArena::give(int64_t at, int64_t len) {
  auto nx = free_.lower_bound(at);
  if (nx != free_.end() && at + len == nx->first) {
    len += nx->second;
    nx = drop(nx);
  }
  if (nx != free_.begin()) {
    auto pv = std::prev(nx);
    if (pv->first + pv->second == at) {
      at = pv->first;
      len += pv->second;
      drop(pv);
    }
  }
  put(at, len);
}

void build_front_plan(int n, const int *c, const int *r, const int *Ls, const int *prunePtr,
                      const int *pruneSet, const HostSym &H, const Plan &P, const Tuning &T,
                      FrontPlan &F) {
  F = FrontPlan();
  const std::vector<int> &super = H.super;
  const std::vector<int64_t> &rowptr = H.rowptr;
  const int ns = (int)super.size() - 1, nlev = (int)P.waves.size();
  auto width = [&](int s) { return super[s + 1] - super[s]; };
  auto rows = [&](int s) { return (int)(rowptr[s + 1] - rowptr[s]); };
  std::vector<int> col2sup(n);
  for (int s = 0; s < ns; ++s)
    for (int j = super[s]; j < super[s + 1]; ++j) col2sup[j] = s;

  // tree, the children's positions in their parent, levels
  std::vector<int> parent(ns, -1), level(ns, 0);
  F.child_ptr.assign(ns + 1, 0);
  F.child_n1.assign(ns, 0);
  F.rel.assign(std::max<int64_t>(H.nls - n, 1), 0);
  for (int s = 0; s < ns; ++s) {
    const int w = width(s), m = rows(s);
    if (m == w) continue;
    const int *rs = Ls + rowptr[s] + w;
    const int p = col2sup[rs[0]];
    parent[s] = p;
    level[p] = std::max(level[p], level[s] + 1);
    F.child_ptr[p + 1]++;
    const int *rp = Ls + rowptr[p];
    const int mp = rows(p), wp = width(p);
    int *rel = F.rel.data() + (rowptr[s] - super[s]);
    int k = 0;
    for (int i = 0; i < m - w; ++i) {
      while (k < mp && rp[k] < rs[i]) ++k;
      if (k == mp || rp[k] != rs[i]) return;   // not contained: left-looking kernels
      rel[i] = k;
      F.child_n1[s] += k < wp;
    }
  }
  for (int s = 0; s < ns; ++s) F.child_ptr[s + 1] += F.child_ptr[s];
  F.child.resize(F.child_ptr[ns]);
  {
    std::vector<int> at(F.child_ptr.begin(), F.child_ptr.end() - 1);
    for (int s = 0; s < ns; ++s)
      if (parent[s] >= 0) F.child[at[parent[s]]++] = s;
  }
  // entries of A in their column's row list
  F.apos.assign(std::max(c[n], 1), -1);
  {
    std::vector<int> at(n, -1);
    for (int s = 0; s < ns; ++s) {
      const int *rs = Ls + rowptr[s];
      const int m = rows(s);
      for (int i = 0; i < m; ++i) at[rs[i]] = i;
      for (int p = c[super[s]]; p < c[super[s + 1]]; ++p)
        if (r[p] >= 0 && r[p] < n) F.apos[p] = at[r[p]];
      for (int i = 0; i < m; ++i) at[rs[i]] = -1;
    }
  }

  F.closed = true;
  if (!prune_sets_complete(Ls, prunePtr, pruneSet, H, col2sup)) return;

  // classes
  std::vector<char> tiled(ns, 0);
  for (int s : P.big_list) tiled[s] = 1;
  auto warp_fits = [&](int s) {
    const int w = width(s), m = rows(s);
    return !tiled[s] && m <= FRONT_WARP_M && front_wp(w) * front_ld(w, m) <= FRONT_WARP_ELEMS;
  };
  std::vector<int> crowd(nlev, 0);
  for (int s = 0; s < ns; ++s) crowd[level[s]] += warp_fits(s);
  std::vector<char> in_warp(ns, 0), in_cta(ns, 0), kids_warp(ns, 1), kids_walk(ns, 1);
  for (int s = 0; s < ns; ++s) {
    const int w = width(s), m = rows(s);
    in_warp[s] = T.tiny && kids_warp[s] && warp_fits(s) && crowd[level[s]] >= FRONT_WARP_LEVEL_MIN;
    if (!in_warp[s])
      in_cta[s] = T.persist && kids_walk[s] && !tiled[s] && m - w <= FRONT_WALK_R &&
                  front_smem(w, m) <= 2 * T.persist_max_smem;
    if (parent[s] >= 0) {
      if (!in_warp[s]) kids_warp[parent[s]] = 0;
      if (!in_warp[s] && !in_cta[s]) kids_walk[parent[s]] = 0;
    }
  }
  std::vector<std::vector<int>> by_level(nlev);
  for (int s = 0; s < ns; ++s) by_level[level[s]].push_back(s);

  // contribution blocks: a block lives from its supernode's wave (the walks': from the start)
  // to the end of its parent's wave (the walks': the end of the walks)
  F.cb_off.assign(ns, 0);
  FrontArena A;
  auto len = [&](int s) {
    const int64_t rr = rows(s) - width(s);
    return (rr * rr + 15) & ~(int64_t)15;
  };
  auto walk = [&](int s) { return in_warp[s] || in_cta[s]; };
  for (int s = 0; s < ns; ++s)
    if (walk(s) && len(s)) F.cb_off[s] = A.take(len(s));
  for (int s = 0; s < ns; ++s)
    if (walk(s) && len(s) && walk(parent[s])) A.give(F.cb_off[s], len(s));
  for (int lv = 0; lv < nlev; ++lv) {
    std::vector<int> here;   // the largest first: less is lost between them
    for (int s : by_level[lv])
      if (!walk(s) && len(s)) here.push_back(s);
    std::stable_sort(here.begin(), here.end(), [&](int a, int b) { return len(a) > len(b); });
    for (int s : here) F.cb_off[s] = A.take(len(s));
    for (int s : by_level[lv])
      if (!walk(s))
        for (int q = F.child_ptr[s]; q < F.child_ptr[s + 1]; ++q)
          A.give(F.cb_off[F.child[q]], len(F.child[q]));
  }
  F.cb_len = A.end();
  if (F.cb_len > front_memory_limit(H.xsize)) return;

  // tasks: the tiles of s's list with origin o (positions o + 64 t of its rows; columns up to
  // clim) and the pairs of children's rows that fall in each; tiles without pairs only if `all`
  struct Run { int tile, start, count; };
  std::vector<Run> run;
  std::vector<int> tile_of;
  std::vector<int4> tile_task;
  std::vector<std::pair<int, int4>> items;
  auto add_tiles = [&](int s, int o, int clim, bool all, std::vector<int4> &tasks, std::vector<int> &end,
                       std::vector<int4> &pairs) {
    const int m = rows(s), nt = (m - o + TB - 1) / TB, nc = (clim - o + TB - 1) / TB;
    tile_of.assign((size_t)nt * nc, -1);
    tile_task.clear();
    items.clear();
    auto tile = [&](int a, int b) {
      int &k = tile_of[(size_t)a * nc + b];
      if (k < 0) {
        k = (int)tile_task.size();
        tile_task.push_back(make_int4(s, a * TB, b * TB, 0));
      }
      return k;
    };
    if (all)
      for (int b = 0; b < nc; ++b)
        for (int a = b; a < nt; ++a) tile(a, b);
    for (int q = F.child_ptr[s]; q < F.child_ptr[s + 1]; ++q) {
      const int d = F.child[q], rd = rows(d) - width(d);
      const int *rel = F.rel.data() + (rowptr[d] - super[d]);
      run.clear();
      for (int i = (int)(std::lower_bound(rel, rel + rd, o) - rel); i < rd;) {
        const int tl = (rel[i] - o) / TB, lim = o + (tl + 1) * TB;
        int e = i + 1;
        while (e < rd && rel[e] < lim) ++e;
        run.push_back({tl, i, e - i});
        i = e;
      }
      for (size_t x = 0; x < run.size(); ++x) {
        const Run &cr = run[x];
        int nb = cr.count;   // columns below clim
        while (nb > 0 && rel[cr.start + nb - 1] >= clim) --nb;
        if (nb == 0) break;
        for (size_t y = x; y < run.size(); ++y)
          items.push_back({tile(run[y].tile, cr.tile),
                           make_int4(d, run[y].start, cr.start, run[y].count | (nb << 16))});
      }
    }
    // pairs grouped by tile, children in order
    const size_t t0 = tasks.size(), p0 = pairs.size();
    tasks.insert(tasks.end(), tile_task.begin(), tile_task.end());
    end.resize(tasks.size(), 0);
    for (const auto &it : items) ++end[t0 + it.first];
    int at = (int)p0;
    for (size_t t = t0; t < tasks.size(); ++t) {
      tasks[t].w = at;
      at += end[t];
      end[t] = tasks[t].w;
    }
    pairs.resize(at);
    for (const auto &it : items) pairs[end[t0 + it.first]++] = it.second;
  };
  F.waves.resize(nlev);
  int launches = 1 + !P.big_list.empty();
  for (int lv = 0; lv < nlev; ++lv) {
    FrontWave &W = F.waves[lv];
    W.small_off = (int)F.small_list.size();
    W.ext_off = (int)F.ext_tasks.size();
    W.sch_off = (int)F.sch_tasks.size();
    // wide fronts first: the launch's tail is made of short products
    std::vector<int> by_width;
    for (int s : by_level[lv]) {
      const int w = width(s), m = rows(s);
      if (in_warp[s]) {
        F.warp_list.push_back(s);
      } else if (in_cta[s]) {
        F.cta_list.push_back(s);
        F.cta_smem = std::max<int>(F.cta_smem, (int)front_smem(w, m));
      } else if (tiled[s]) {
        add_tiles(s, 0, w, false, F.ext_tasks, F.ext_end, F.ext_pairs);
        if (m > w) by_width.push_back(s);
      } else {
        const bool by_tiles = m - w > FRONT_SMALL_R;
        F.small_list.push_back(by_tiles ? ~s : s);
        W.small_smem = std::max<int>(W.small_smem, (int)front_smem(w, m));
        if (by_tiles) by_width.push_back(s);
      }
    }
    std::stable_sort(by_width.begin(), by_width.end(), [&](int a, int b) { return width(a) > width(b); });
    const Wave &B = P.waves[lv];
    const int nsteps = (int)B.panel_off.size();
    W.sch_more.assign(nsteps + 1, 0);
    for (int s : by_width) {
      add_tiles(s, width(s), rows(s), true, F.sch_tasks, F.sch_end, F.sch_pairs);
      for (int b = 0; b < (width(s) + TB - 1) / TB && b <= nsteps; ++b)
        W.sch_more[b] = (int)F.sch_tasks.size() - W.sch_off;
    }
    const int part = std::max(FRONT_BG_STEPS, (nsteps + 3) / 4);
    double flops = 0.0;
    for (int s : by_width) {
      const double w = width(s), rr = rows(s) - width(s);
      flops += rr * rr * w + rows(s) * w * w;
    }
    if (B.dense_cnt == 0 && nsteps > part && flops <= 1.5 * FRONT_FLOPS_US * FRONT_STEP_US * nsteps) W.sch_steps = part;
    W.small_cnt = (int)F.small_list.size() - W.small_off;
    W.ext_cnt = (int)F.ext_tasks.size() - W.ext_off;
    W.sch_cnt = (int)F.sch_tasks.size() - W.sch_off;
    launches += (W.small_cnt > 0) + (W.ext_cnt > 0) + (W.sch_cnt > 0);
    for (int b = W.sch_steps; W.sch_steps && b < nsteps; b += W.sch_steps) launches += W.sch_more[b] > 0;
    if (B.dense_cnt > 0) {
      launches += 1;
    } else {
      launches += B.big_cnt > 0;
      for (size_t j = 0; j < B.panel_cnt.size(); ++j)
        launches += (B.panel_cnt[j] > 0) + (B.syrk_nc[j] > 0) + (B.syrk_cnt[j] > B.syrk_nc[j]) + (B.diag_cnt[j] > 0);
    }
  }
  F.launches = launches + !F.warp_list.empty() + !F.cta_list.empty();

  // descriptors, and the entries of A of the small fronts in their padded panels
  for (int d : F.child)
    F.kids.push_back(FrontChild{d, rows(d) - width(d), F.child_n1[d], 0, rowptr[d] - super[d], F.cb_off[d]});
  F.ppos = F.apos;
  auto desc = [&](int s, bool by_tiles) {
    const int w = width(s), ld = front_ld(w, rows(s)), pad = front_wp(w) - w;
    for (int j = 0; j < w; ++j)
      for (int p = c[super[s] + j]; p < c[super[s] + j + 1]; ++p)
        if (F.apos[p] >= 0) F.ppos[p] = j * ld + (F.apos[p] < w ? F.apos[p] : F.apos[p] + pad);
    return FrontDesc{s, super[s], w, rows(s), F.child_ptr[s], F.child_ptr[s + 1], c[super[s]], c[super[s + 1]],
                     H.xptr[s], by_tiles ? -1 : F.cb_off[s]};
  };
  for (int s : F.warp_list) F.warp_desc.push_back(desc(s, false));
  for (int s : F.cta_list) F.cta_desc.push_back(desc(s, false));
  for (int e : F.small_list) F.small_desc.push_back(desc(e < 0 ? ~e : e, e < 0));

  // work: every product once, every entry of A, of L and of the blocks read or written once by the
  // class that does it
  F.work = P.work;
  KernelStats &K = F.work;
  K.flops[K_SMALL] = K.bytes[K_SMALL] = K.flops[K_UPDATE] = K.bytes[K_UPDATE] = 0.0;
  std::vector<char> by_tiles(ns, 0);
  for (int e : F.small_list)
    if (e < 0) by_tiles[~e] = 1;
  for (int s = 0; s < ns; ++s) {
    const double w = width(s), rr = rows(s) - width(s);
    const int own = tiled[s] || by_tiles[s] ? K_UPDATE : K_SMALL;   // who forms its block
    if (!tiled[s]) {
      K.flops[K_SMALL] += w * w * w / 3.0 + rr * w * w;
      K.bytes[K_SMALL] += 8.0 * (w + rr) * w + 12.0 * (c[super[s + 1]] - c[super[s]]);
    }
    K.flops[own] += rr * (rr + 1.0) * w;
    K.bytes[own] += 4.0 * rr * (rr + 1.0) + (own == K_UPDATE ? 8.0 * rr * w : 0.0);
    for (int q = F.child_ptr[s]; q < F.child_ptr[s + 1]; ++q) {
      const double rd = rows(F.child[q]) - width(F.child[q]), n1 = F.child_n1[F.child[q]], n2 = rd - n1;
      K.bytes[tiled[s] ? K_UPDATE : K_SMALL] += 8.0 * (n1 * rd - n1 * (n1 - 1.0) / 2.0) + 4.0 * rd;
      K.bytes[own] += 4.0 * n2 * (n2 + 1.0);
    }
  }
  for (const int4 &t : F.ext_tasks) {   // tiles of tiled panels, read and written
    const int nr = std::min(TB, rows(t.x) - t.y), nc = std::min(TB, width(t.x) - t.z);
    K.bytes[K_UPDATE] += 16.0 * (t.y == t.z ? nr * nc - nc * (nc - 1) / 2 : nr * nc);
  }
  F.ok = true;
}

bool check_front_plan(int n, const int *Ls, const HostSym &H, const Plan &P, const FrontPlan &F,
                      std::string &err) {
  if (!F.ok) return true;
  const std::vector<int> &super = H.super;
  const std::vector<int64_t> &rowptr = H.rowptr;
  const int ns = (int)super.size() - 1;
  auto width = [&](int s) { return super[s + 1] - super[s]; };
  auto rows = [&](int s) { return (int)(rowptr[s + 1] - rowptr[s]); };
  auto bad = [&](const char *what, int s) {
    err = std::string("front plan: ") + what + ", supernode " + std::to_string(s);
    return false;
  };
  if ((int)F.child_ptr.size() != ns + 1 || F.waves.size() != P.waves.size() ||
      (int64_t)F.rel.size() < H.nls - n)
    return bad("array sizes", -1);
  if (F.cb_len > front_memory_limit(H.xsize)) return bad("contribution blocks larger than their bound", -1);
  // the children's maps
  std::vector<int> parent(ns, -1), level(ns, 0);
  for (int s = 0; s < ns; ++s)
    for (int q = F.child_ptr[s]; q < F.child_ptr[s + 1]; ++q) {
      const int d = F.child[q], rd = rows(d) - width(d);
      if (d < 0 || d >= s || parent[d] >= 0) return bad("a child listed twice or out of order", s);
      parent[d] = s;
      level[s] = std::max(level[s], level[d] + 1);
      const int *rel = F.rel.data() + (rowptr[d] - super[d]);
      int n1 = 0;
      for (int i = 0; i < rd; ++i) {
        if (rel[i] < 0 || rel[i] >= rows(s) || Ls[rowptr[s] + rel[i]] != Ls[rowptr[d] + width(d) + i])
          return bad("row map", d);
        n1 += rel[i] < width(s);
      }
      if (n1 != F.child_n1[d]) return bad("rows among the parent's columns", d);
    }
  for (int s = 0; s < ns; ++s)
    if ((rows(s) > width(s)) != (parent[s] >= 0)) return bad("no parent", s);
  // every front once: 1 warp walk, 2 CTA walk, 3 level launch, 4 tiled
  std::vector<char> how(ns, 0), tiles(ns, 0);
  auto place = [&](int s, int k) {
    if (s < 0 || s >= ns || how[s]) return false;
    how[s] = (char)k;
    return true;
  };
  std::vector<char> done(ns, 0);
  for (int k = 0; k < 2; ++k)
    for (int s : k ? F.cta_list : F.warp_list) {
      if (!place(s, k + 1)) return bad("front in two lists", s);
      for (int q = F.child_ptr[s]; q < F.child_ptr[s + 1]; ++q)
        if (!done[F.child[q]]) return bad("a walk's child after its parent", s);
      done[s] = 1;
      const int w = width(s), m = rows(s);
      if (k == 0 ? front_wp(w) * front_ld(w, m) > FRONT_WARP_ELEMS || m > FRONT_WARP_M
                 : front_smem(w, m) > F.cta_smem)
        return bad("front larger than its walk's shared memory", s);
    }
  for (size_t lv = 0; lv < F.waves.size(); ++lv) {
    const FrontWave &W = F.waves[lv];
    for (int k = W.small_off; k < W.small_off + W.small_cnt; ++k) {
      const int s = F.small_list[k] < 0 ? ~F.small_list[k] : F.small_list[k];
      if (!place(s, 3) || level[s] != (int)lv) return bad("front in two lists or another level", s);
      if (front_smem(width(s), rows(s)) > W.small_smem || W.small_smem > 200 * 1024)
        return bad("front larger than its launch's shared memory", s);
      tiles[s] = F.small_list[k] < 0;
    }
    const Wave &B = P.waves[lv];
    for (int k = B.big_off; k < B.big_off + B.big_cnt; ++k) {
      if (!place(P.big_list[k], 4) || level[P.big_list[k]] != (int)lv)
        return bad("tiled front in two lists or another level", P.big_list[k]);
      tiles[P.big_list[k]] = 1;
    }
  }
  for (int s = 0; s < ns; ++s)
    if (!how[s]) return bad("front in no list", s);
  // tiles: per front the entries its tiles receive from children, and its block's tiles
  std::vector<int64_t> got_panel(ns, 0), got_block(ns, 0), block_tiles(ns, 0);
  for (int part = 0; part < 2; ++part) {
    const std::vector<int4> &tk = part ? F.sch_tasks : F.ext_tasks, &pr = part ? F.sch_pairs : F.ext_pairs;
    const std::vector<int> &end = part ? F.sch_end : F.ext_end;
    std::map<std::pair<int, std::pair<int, int>>, int> seen;
    for (size_t lv = 0; lv < F.waves.size(); ++lv) {
      const FrontWave &W = F.waves[lv];
      const int t0 = part ? W.sch_off : W.ext_off, t1 = t0 + (part ? W.sch_cnt : W.ext_cnt);
      for (int t = t0; t < t1; ++t) {
        const int s = tk[t].x, w = width(s), o = part ? w : 0, lim = part ? rows(s) : w;
        if (s < 0 || s >= ns || level[s] != (int)lv || !tiles[s] || (!part && how[s] != 4))
          return bad("tile of a front that has none, or in another level", s);
        if (tk[t].y % TB || tk[t].z % TB || tk[t].z > tk[t].y || o + tk[t].y >= rows(s) ||
            o + tk[t].z >= lim || seen[{s, {tk[t].y, tk[t].z}}]++)
          return bad("tile misplaced or twice", s);
        block_tiles[s] += part;
        for (size_t b = 0; part && b < W.sch_more.size(); ++b)
          if ((t - t0 < W.sch_more[b]) != ((int)b * TB < w)) return bad("tiles of the wider fronts not first", s);
        for (int q = tk[t].w; q < end[t]; ++q) {
          const int d = pr[q].x, na = pr[q].w & 0xffff, nb = pr[q].w >> 16;
          if (d < 0 || d >= ns || parent[d] != s || na <= 0 || nb <= 0 || na > TB || nb > TB ||
              pr[q].y < 0 || pr[q].z < 0 || pr[q].y + na > rows(d) - width(d))
            return bad("pair of a tile", s);
          const int *rel = F.rel.data() + (rowptr[d] - super[d]);
          if (rel[pr[q].y] < o + tk[t].y || rel[pr[q].y + na - 1] >= o + tk[t].y + TB ||
              rel[pr[q].z] < o + tk[t].z || rel[pr[q].z + nb - 1] >= std::min(lim, o + tk[t].z + TB))
            return bad("rows of a pair outside its tile", s);
          const bool diag = pr[q].y == pr[q].z;
          const int64_t e = diag ? (int64_t)nb * (nb + 1) / 2 + (int64_t)(na - nb) * nb : (int64_t)na * nb;
          (part ? got_block : got_panel)[s] += e;
        }
      }
    }
  }
  for (int s = 0; s < ns; ++s) {
    if (!tiles[s]) continue;
    int64_t panel = 0, block = 0;
    for (int q = F.child_ptr[s]; q < F.child_ptr[s + 1]; ++q) {
      const int64_t rd = rows(F.child[q]) - width(F.child[q]), n1 = F.child_n1[F.child[q]];
      panel += n1 * rd - n1 * (n1 - 1) / 2;
      block += (rd - n1) * (rd - n1 + 1) / 2;
    }
    const int64_t nt = (rows(s) - width(s) + TB - 1) / TB;
    if ((how[s] == 4 && got_panel[s] != panel) || got_block[s] != block || block_tiles[s] != nt * (nt + 1) / 2)
      return bad("entries of the children's blocks or tiles missing", s);
  }
  // blocks alive together do not overlap: waves in order, the walks first
  std::map<int64_t, int64_t> live;
  auto put = [&](int s) {
    const int64_t rr = rows(s) - width(s), at = F.cb_off[s], e = at + rr * rr;
    if (rr == 0) return true;
    auto nx = live.lower_bound(at);
    if (at < 0 || e > F.cb_len || (nx != live.end() && nx->first < e)) return false;
    if (nx != live.begin() && std::prev(nx)->second > at) return false;
    live[at] = e;
    return true;
  };
  for (int s = 0; s < ns; ++s)
    if (how[s] <= 2 && !put(s)) return bad("contribution blocks overlap", s);
  for (int s = 0; s < ns; ++s)
    if (how[s] <= 2 && parent[s] >= 0 && how[parent[s]] <= 2) live.erase(F.cb_off[s]);
  std::vector<std::vector<int>> by_level(F.waves.size());
  for (int s = 0; s < ns; ++s)
    if (how[s] > 2) by_level[level[s]].push_back(s);
  for (const std::vector<int> &v : by_level) {
    for (int s : v)
      if (!put(s)) return bad("contribution blocks overlap", s);
    for (int s : v)
      for (int q = F.child_ptr[s]; q < F.child_ptr[s + 1]; ++q) live.erase(F.cb_off[F.child[q]]);
  }
  return true;
}

}  // namespace swc
