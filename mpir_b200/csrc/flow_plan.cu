// Work items of the dataflow triangular solves (solve.cu), from the
// supernodal schedule.
#include <algorithm>
#include <cstdint>
#include <stdexcept>

#include "engine.hpp"

namespace mpir {

void Plan::build_flow() {
  const int64_t ns = S.ns;
  flow_part_elems = flow_inv_elems = flow_wpanel_total = 0;
  std::vector<FlowFront>   warp;
  std::vector<FlowItem>    fwd, bwd;
  std::vector<FlowInvDesc> inv;
  std::vector<FlowFront>   fr(ns);
  // Child contributions of every front's rows (row i of front J at zofs[J] + i):
  // the first child's beside the row, the others' after their count, in child
  // order (the forward solves add them in this order).
  flow_entry(S.z_elems);
  std::vector<uint32_t>   more, cnt, src;
  std::vector<FlowGather> first(S.z_elems, FlowGather{kFlowNone, kFlowNone});
  // Sums, by level and by the depth of a sum of sums.
  std::vector<std::vector<std::vector<FlowItem>>> sums(S.nlevels);
  std::vector<int32_t>                            level;
  std::vector<std::vector<uint32_t>>              lists;  // of a front's rows with many contributions
  std::vector<int64_t>                            list_row;
  flow_z_elems = S.z_elems;
  auto put = [&](int64_t row, const uint32_t *e, uint32_t n) {
    FlowGather &g = first[row];
    if (n > 0) g.first = e[0];
    if (n > 1) {
      g.more = flow_entry(static_cast<int64_t>(more.size()));
      more.push_back(n - 1);
      more.insert(more.end(), e + 1, e + n);
    }
  };
  for (int64_t J = 0; J < ns; J++) {
    const int64_t h = S.h(J);
    cnt.assign(h + 1, 0);
    for (int64_t c = S.child_ptr[J]; c < S.child_ptr[J + 1]; c++) {
      const int64_t C = S.child_list[c];
      for (int64_t q = S.srowptr[C] + S.w(C); q < S.srowptr[C + 1]; q++) cnt[S.srel[q] + 1]++;
    }
    for (int64_t i = 0; i < h; i++) cnt[i + 1] += cnt[i];
    src.resize(cnt[h]);
    for (int64_t c = S.child_ptr[J]; c < S.child_ptr[J + 1]; c++) {
      const int64_t C = S.child_list[c], wc = S.w(C);
      for (int64_t a = wc; a < S.h(C); a++)
        src[cnt[S.srel[S.srowptr[C] + a]]++] = flow_entry(S.zofs[C] + a);
    }
    // cnt[i] is now the end of row i
    for (int64_t i = 0; i < h; i++) {
      const uint32_t e = i > 0 ? cnt[i - 1] : 0, n = cnt[i] - e;
      if (n <= kFlowFan) {
        put(S.zofs[J] + i, src.data() + e, n);
      } else {
        lists.emplace_back(src.begin() + e, src.begin() + e + n);
        list_row.push_back(S.zofs[J] + i);
      }
    }
    if (lists.empty()) continue;
    if (level.empty()) {
      level.resize(ns);
      for (int32_t t = 0; t < S.nlevels; t++)
        for (int64_t q = S.level_ptr[t]; q < S.level_ptr[t + 1]; q++) level[S.level_sup[q]] = t;
    }
    auto &out = sums[level[J]];
    bool  any = true;
    for (size_t depth = 0; any; depth++) {
      any               = false;
      const int64_t z0  = flow_z_elems, m0 = static_cast<int64_t>(more.size());
      for (auto &l : lists) {
        if (l.size() <= (depth == 0 ? kFlowFan : 8)) continue;
        std::vector<uint32_t> up;
        for (size_t q = 0; q < l.size(); q += kFlowFan) {
          const size_t n = std::min<size_t>(kFlowFan, l.size() - q);
          more.insert(more.end(), l.begin() + q, l.begin() + q + n);
          more.insert(more.end(), kFlowFan - n, kFlowNone);
          up.push_back(flow_entry(flow_z_elems++));
        }
        l   = std::move(up);
        any = true;
      }
      if (out.size() <= depth && any) out.resize(depth + 1);
      for (int64_t z = z0; z < flow_z_elems; z += kFlowFan) {
        FlowItem it{};
        it.f.zofs = z;
        it.f.rows = m0 + (z - z0) * kFlowFan;
        it.kind   = kFwdSum;
        it.nr     = static_cast<int32_t>(std::min<int64_t>(kFlowFan, flow_z_elems - z));
        out[depth].push_back(it);
      }
    }
    for (size_t q = 0; q < lists.size(); q++)
      put(list_row[q], lists[q].data(), static_cast<uint32_t>(lists[q].size()));
    lists.clear();
    list_row.clear();
  }
  host_.flow_gfirst = std::move(first);
  host_.flow_gmore  = std::move(more);
  // Front descriptors; the inverses and the chunk partials of those that are
  // not solved by one warp.
  std::vector<uint8_t> top(ns, 0);  // in the last level
  if (S.nlevels > 0)
    for (int64_t q = S.level_ptr[S.nlevels - 1]; q < S.level_ptr[S.nlevels]; q++) top[S.level_sup[q]] = 1;
  std::vector<FlowInvDesc> inv_top;
  for (int64_t J = 0; J < ns; J++) {
    FlowFront    &f = fr[J];
    const int64_t w = S.w(J), h = S.h(J);
    f.panel  = S.slofs[J];
    f.zofs   = S.zofs[J];
    f.inv    = -1;
    f.part   = -1;
    f.rows   = S.srowptr[J];
    f.h      = static_cast<int32_t>(h);
    f.w      = static_cast<int32_t>(w);
    f.col0   = static_cast<int32_t>(S.sfirst[J]);
    f.chunks = 0;
    f.gate   = -1;
    f.pad    = 0;
    if (h > w) {
      // The parent's columns come last, of a wide parent the lowest
      // super-block: the first row past those is ready before them.
      const int32_t *r = S.srows.data() + S.srowptr[J];
      const int64_t  p = S.sparent[J], p0 = S.sfirst[p];
      int64_t        end = S.sfirst[p + 1];
      if (S.w(p) > kFlowNarrow) end = std::min(end, p0 + ((r[w] - p0) / kFlowSB + 1) * kFlowSB);
      const int32_t *q = std::lower_bound(r + w, r + h, static_cast<int32_t>(end));
      if (q != r + h) f.gate = *q;
    }
    if (warp_solved(J)) {
      f.inv = flow_wpanel_total;
      flow_wpanel_total += flow_wpanel_elems(f.w, f.h);
      if (top[J]) flow_warp_top = true;
      continue;
    }
    f.inv = flow_inv_elems;
    flow_inv_elems += flow_inv_blocks(w) * kFlowBlk;
    for (int64_t s = 0; s * kFlowSB < w; s++) {
      const int32_t n = static_cast<int32_t>(std::min<int64_t>(kFlowSB, w - s * kFlowSB));
      for (int32_t c = 0; c < n; c += 16)
        (top[J] ? inv_top : inv)
            .push_back(FlowInvDesc{f.panel + s * kFlowSB * (h + 1), f.inv + s * kFlowTriSB * kFlowBlk, f.h,
                                   n, c, 0});
    }
    // The rows below a narrow block that fit one chunk are taken by the item
    // that solves the block.
    if (w > kFlowNarrow || h - w > kFlowChunk) {
      f.chunks = static_cast<int32_t>((h - w + kFlowChunk - 1) / kFlowChunk);
      f.part   = flow_part_elems;
      flow_part_elems += static_cast<int64_t>(f.chunks) * w;
    }
  }
  // Long strips first (a strip's work grows with the rows below it).
  for (auto *v : {&inv, &inv_top})
    std::stable_sort(v->begin(), v->end(), [](const FlowInvDesc &a, const FlowInvDesc &b) {
      return a.n - a.c0 > b.n - b.c0;
    });
  nflow_inv_low = static_cast<int32_t>(inv.size());
  inv.insert(inv.end(), inv_top.begin(), inv_top.end());
  // A level's warp-solved fronts, in groups that spread over the SMs and
  // whose panels fit the shared memory.
  auto warps = [&](std::vector<FlowItem> &out, size_t first, size_t count) {
    const size_t per = std::min<size_t>(kFlowWarpsPerItem, std::max<size_t>(1, (count + kSMs - 1) / kSMs));
    for (size_t q = first; q < first + count;) {
      int64_t used = 0;
      size_t  e   = q;
      while (e < first + count && e - q < per) {
        const int64_t b = flow_wpanel_elems(warp[e].w, warp[e].h) * 8;
        if (used + b > kFlowPanelSmem) break;
        warp[e].part = used;
        used += b;
        e++;
      }
      out.push_back(FlowItem{FlowFront{}, kFlowWarps, static_cast<int32_t>(q),
                             static_cast<int32_t>(e - q), 0});
      q = e;
    }
  };
  // Leaves of at most 64 rows, where there are many of them.
  nflow_leaf = nflow_leaf_fwd = nflow_leaf_bwd = 0;
  std::vector<FlowFront> leaf;
  size_t                 leaf_warps = 0;  // the first of the warp-solved fronts
  if (S.nlevels > 0) {
    int64_t nw = 0, nn = 0;
    for (int64_t q = S.level_ptr[0]; q < S.level_ptr[1]; q++) {
      const int64_t J = S.level_sup[q];
      if (!is_large(J)) (warp_solved(J) ? nw : nn)++;
    }
    if (nw / kFlowWarpsPerItem + nn >= kFlowLeafItems)
      for (int64_t q = S.level_ptr[0]; q < S.level_ptr[1]; q++) {
        const int64_t J = S.level_sup[q];
        if (is_large(J)) continue;
        leaf.push_back(fr[J]);
        if (warp_solved(J))
          warp.push_back(fr[J]);
        else
          fwd.push_back(FlowItem{fr[J], kFwdNarrow, fr[J].w, fr[J].h - fr[J].w, 0});
      }
    leaf_warps = warp.size();
    warps(fwd, 0, leaf_warps);
    nflow_leaf     = static_cast<int32_t>(leaf.size());
    nflow_leaf_fwd = static_cast<int32_t>(fwd.size());
  }
  auto taken = [&](int64_t J, int32_t t) { return t == 0 && nflow_leaf > 0 && !is_large(J); };
  struct Range {
    size_t first, count;
  };
  std::vector<Range> wr(S.nlevels);
  // Forward, leaves first.  Within a level: the sums of its rows with many
  // contributions (a sum's sources first), the slabs of the wide fronts'
  // diagonal blocks (their chains start together), the narrow fronts, the
  // warp-solved fronts, then the rows below the wide blocks, which wait on
  // the slabs.  An item waits only on items before it.
  for (int32_t t = 0; t < S.nlevels; t++) {
    wr[t].first = warp.size();
    for (const auto &s : sums[t]) fwd.insert(fwd.end(), s.begin(), s.end());
    std::vector<FlowItem> rows, narrow;
    // Rows of a narrow front's items: 512, less where the level would leave
    // SMs idle (w <= 32: always 512, a thread a row).
    int64_t below = 0;
    for (int64_t q = S.level_ptr[t]; q < S.level_ptr[t + 1]; q++) {
      const FlowFront &f = fr[S.level_sup[q]];
      if (f.w > 32 && f.w <= kFlowNarrow) below += f.h - f.w;
    }
    int32_t step4 = kFlowRows;
    while (step4 > 128 && below / step4 < kSMs) step4 /= 2;
    for (int64_t q = S.level_ptr[t]; q < S.level_ptr[t + 1]; q++) {
      const int64_t    J = S.level_sup[q];
      const FlowFront &f = fr[J];
      if (taken(J, t)) continue;
      if (warp_solved(J)) {
        warp.push_back(f);
      } else if (f.w <= kFlowNarrow) {
        const int32_t step = f.w <= 32 ? kFlowRows : step4;
        int32_t       r    = f.w;
        do {
          narrow.push_back(FlowItem{f, kFwdNarrow, r, std::min(step, f.h - r), 0});
          r += step;
        } while (r < f.h);
      } else {
        for (int32_t r = 0; r < f.w; r += 32)
          fwd.push_back(FlowItem{f, kFwdSlab, r, std::min(32, f.w - r), 0});
        for (int32_t r = f.w; r < f.h; r += kFlowRowsW)
          rows.push_back(FlowItem{f, kFwdRows, r, std::min(kFlowRowsW, f.h - r), 0});
      }
    }
    wr[t].count = warp.size() - wr[t].first;
    fwd.insert(fwd.end(), narrow.begin(), narrow.end());
    warps(fwd, wr[t].first, wr[t].count);
    fwd.insert(fwd.end(), rows.begin(), rows.end());
  }
  // Backward, roots first: the chunks of the rows below the blocks, the
  // blocks (the slabs of a wide one last first), the warp-solved fronts.
  for (int32_t t = S.nlevels - 1; t >= 0; t--) {
    std::vector<FlowItem> own;
    for (int64_t q = S.level_ptr[t]; q < S.level_ptr[t + 1]; q++) {
      const int64_t    J = S.level_sup[q];
      const FlowFront &f = fr[J];
      if (warp_solved(J) || taken(J, t)) continue;
      for (int32_t c = 0; c < f.chunks; c++)
        for (int32_t k = 0; k < f.w; k += kFlowChunkC)
          bwd.push_back(FlowItem{f, kBwdChunk, k, std::min(kFlowChunkC, f.w - k), c});
      if (f.w <= kFlowNarrow)
        own.push_back(FlowItem{f, kBwdNarrow, 0, f.w, 0});
      else
        for (int32_t k = (f.w - 1) / 32 * 32; k >= 0; k -= 32)
          own.push_back(FlowItem{f, kBwdSlab, k, std::min(32, f.w - k), 0});
    }
    bwd.insert(bwd.end(), own.begin(), own.end());
    warps(bwd, wr[t].first, wr[t].count);
  }
  const size_t others = bwd.size();
  for (const FlowFront &f : leaf)
    if (!(f.w <= kWarpSolveW && f.h <= kWarpSolveH)) bwd.push_back(FlowItem{f, kBwdNarrow, 0, f.w, 0});
  warps(bwd, 0, leaf_warps);
  nflow_leaf_bwd    = static_cast<int32_t>(bwd.size() - others);
  nflow_fwd         = static_cast<int32_t>(fwd.size());
  nflow_bwd         = static_cast<int32_t>(bwd.size());
  nflow_inv         = static_cast<int32_t>(inv.size());
  host_.flow_warp   = std::move(warp);
  host_.flow_leaf   = std::move(leaf);
  host_.flow_fwd    = std::move(fwd);
  host_.flow_bwd    = std::move(bwd);
  host_.flow_inv    = std::move(inv);
}

}  // namespace mpir
