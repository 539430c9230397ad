// chain_plan.cpp -- the packer's placement of a region's single-pass reads in
// chain items (chain_plan.h).  Replaces the reference's SIMD grouping
// (greedy_grouping, src/core/pairhmm_schedule.cpp:46-105) for the warp
// wavefront's geometry.
#include "chain_plan.h"

#include <algorithm>

namespace rodv {

namespace {

// Time per computed cell (lane rows x columns, padding included) of the chain
// kernels by rows per lane R, relative to R = 8: the autotuner's per-class
// batches (reads of 32R - 5 bases, one read pair per item) on B200 with each
// class's fastest variant (per-row R = 8 takes 1.62 times uniform R = 8).
// R <= 3, and R = 4 with per-row gaps, run as two 16-lane items per warp with
// 2R rows per lane, hence their closeness to R = 8.
constexpr double kChainCellCost[2][kMaxRowsPerLane + 1] = {
    {0.0, 1.41, 1.15, 1.14, 1.02, 1.08, 1.035, 1.05, 1.0},   // per-row gaps
    {0.0, 1.64, 1.28, 1.17, 1.11, 1.11, 1.02, 1.04, 1.0}};   // uniform gaps

// Whether a region's uniform pairs stack decides which read of an odd count is
// left over, and a leftover's result is rounded differently from a pair's
// (the two-haplotype kernel scales row 0 by its own haplotype).  So the
// decision takes fixed costs and a fixed geometry (two items per warp for R <=
// 2), and no kernel variant or later measurement moves a result's last bits.
constexpr double kDecisionCost[kMaxRowsPerLane + 1] = {0.0,   1.53,  1.20,  1.09, 1.024,
                                                       1.093, 1.047, 1.031, 1.0};
constexpr int kDecisionItemsPerWarp[kMaxRowsPerLane + 1] = {0, 2, 2, 1, 1, 1, 1, 1, 1};

// The cheapest class of one gap form whose items hold n pairs with longer
// reads of lengths lens (the R = 8 class always does).
const ChainGeom& cheapest(const ChainGeom (&geom)[kMaxRowsPerLane + 1], bool uniform,
                          const uint32_t* lens, size_t n) {
  const ChainGeom* best = &geom[kMaxRowsPerLane];
  for (int R = 1; R < kMaxRowsPerLane; ++R) {
    if (geom[R].cost >= best->cost) continue;
    uint32_t lanes = 0;
    for (size_t i = 0; i < n; ++i) lanes += pair_lanes(lens[i], geom[R].rows, uniform);
    if (lanes <= geom[R].lanes) best = &geom[R];
  }
  return *best;
}

// Stacks np read pairs of one gap form -- the reads desc[0 .. 2 np) in
// decreasing length, neighbours pair up -- into items: the pairs go by best
// fit in that order into items of the R = 8 class (a pair takes the item with
// the fewest free lanes that still holds its pair_lanes), and each item then
// goes to the cheapest class that holds its pairs.  Appends the items to rc
// and returns true if they cost less than `limit` (uniform gaps: by the
// decision's costs).
bool stack_pairs(const uint32_t* read_lengths, const ChainGeoms& geoms, bool uniform,
                 const std::vector<uint32_t>& desc, size_t np, double limit, RegionChains& rc) {
  const ChainGeom& stack_geom = geoms.g[uniform][kMaxRowsPerLane];
  rc.pair_item.assign(np, 0);
  rc.item_free.clear();
  for (auto& v : rc.bucket) v.clear();
  for (size_t q = 0; q < np; ++q) {
    const uint32_t lanes = pair_lanes(read_lengths[desc[2 * q]], stack_geom.rows, uniform);
    uint32_t it = kNoPair;
    for (uint32_t f = lanes; f <= stack_geom.lanes && it == kNoPair; ++f)
      if (!rc.bucket[f].empty()) {
        it = rc.bucket[f].back();
        rc.bucket[f].pop_back();
      }
    if (it == kNoPair) {
      it = (uint32_t)rc.item_free.size();
      rc.item_free.push_back(stack_geom.lanes);
    }
    rc.item_free[it] -= lanes;
    rc.bucket[rc.item_free[it]].push_back(it);
    rc.pair_item[q] = it;
  }
  // the items' pairs, item after item, each item's in placement order
  const uint32_t nit = (uint32_t)rc.item_free.size();
  rc.item_fill.assign(nit + 1, 0);
  for (uint32_t it : rc.pair_item) rc.item_fill[it + 1] += 2;
  for (uint32_t it = 0; it < nit; ++it) rc.item_fill[it + 1] += rc.item_fill[it];
  rc.item_lens.resize(np);
  rc.item_cls.resize(nit);
  {
    std::vector<uint32_t>& at = rc.item_free;  // reused: next pair slot per item
    for (uint32_t it = 0; it < nit; ++it) at[it] = rc.item_fill[it] / 2;
    for (size_t q = 0; q < np; ++q)
      rc.item_lens[at[rc.pair_item[q]]++] = read_lengths[desc[2 * q]];
  }
  double cost = 0.0;
  for (uint32_t it = 0; it < nit; ++it) {
    const uint32_t p0 = rc.item_fill[it] / 2, p1 = rc.item_fill[it + 1] / 2;
    const uint32_t* lens = rc.item_lens.data() + p0;
    rc.item_cls[it] = cheapest(geoms.g[uniform], uniform, lens, p1 - p0).cls;
    cost += cheapest(uniform ? geoms.decide : geoms.g[0], uniform, lens, p1 - p0).cost;
  }
  if (!(cost < limit)) return false;
  const uint32_t base = (uint32_t)rc.reads.size();
  rc.reads.resize(base + 2 * np);
  for (uint32_t it = 0; it < nit; ++it)
    rc.items.push_back(ChainPairs{rc.item_cls[it], base + rc.item_fill[it],
                                  (rc.item_fill[it + 1] - rc.item_fill[it]) / 2});
  for (size_t q = 0; q < np; ++q) {
    uint32_t& at = rc.item_fill[rc.pair_item[q]];
    rc.reads[base + at] = desc[2 * q];
    rc.reads[base + at + 1] = desc[2 * q + 1];
    at += 2;
  }
  return true;
}

}  // namespace

void chain_geometry(const int (&items_per_warp)[2][kMaxRowsPerLane + 1], ChainGeoms& geoms) {
  for (int u = 0; u < 2; ++u) {
    geoms.g[u][0] = ChainGeom{};
    for (int R = 1; R <= kMaxRowsPerLane; ++R) {
      const int ipw = items_per_warp[u][R] > 1 ? items_per_warp[u][R] : 1;
      geoms.g[u][R] = ChainGeom{single_pass_class(R, u != 0), (uint32_t)(kWarp / ipw),
                                (uint32_t)(R * ipw), R * kChainCellCost[u][R]};
    }
  }
  geoms.decide[0] = ChainGeom{};
  for (int R = 1; R <= kMaxRowsPerLane; ++R) {
    const int ipw = kDecisionItemsPerWarp[R];
    geoms.decide[R] = ChainGeom{single_pass_class(R, true), (uint32_t)(kWarp / ipw),
                                (uint32_t)(R * ipw), R * kDecisionCost[R]};
  }
}

void sort_single_pass(const uint32_t* read_lengths, const uint8_t* read_class,
                      uint32_t read_start, uint32_t num_reads, std::vector<uint32_t>& out) {
  out.clear();
  for (uint32_t r = 0; r < num_reads; ++r) {
    const uint32_t read = read_start + r;
    if (!class_multi(read_class[read])) out.push_back(read);
  }
  std::stable_sort(out.begin(), out.end(), [&](uint32_t x, uint32_t y) {
    const uint32_t kx = ((read_class[x] & 1u) << 20) | read_lengths[x];
    const uint32_t ky = ((read_class[y] & 1u) << 20) | read_lengths[y];
    return kx < ky;
  });
}

void plan_region_chains(const uint32_t* read_lengths, const uint8_t* read_class,
                        const ChainGeoms& geoms, ChainStacking stacking,
                        const std::vector<uint32_t>& sr, RegionChains& rc) {
  auto pair_class = [&](uint32_t x, uint32_t y) {
    const uint32_t len = std::max(read_lengths[x], read_lengths[y]);
    return class_of(len, (read_class[x] & 1) && (read_class[y] & 1));
  };
  rc.reads.clear();
  rc.items.clear();
  rc.leftover = kNoPair;
  size_t nu = 0;  // reads with per-row gap priors come first
  while (nu < sr.size() && !(read_class[sr[nu]] & 1)) ++nu;
  auto add_pair = [&](uint32_t x, uint32_t y) {
    rc.items.push_back(ChainPairs{pair_class(x, y), (uint32_t)rc.reads.size(), 1});
    rc.reads.push_back(x);
    rc.reads.push_back(y);
  };
  // cost of the one-pair item of a pair whose longer read has `len` bases
  auto pair_cost = [&](uint32_t len, bool uniform) {
    return cheapest(uniform ? geoms.decide : geoms.g[0], uniform, &len, 1).cost;
  };
  // Reads computed with per-row gap priors: sr[0, m).
  const size_t m = ((nu & 1) && nu < sr.size()) ? nu + 1 : nu;
  const size_t np_row = m / 2;
  bool stacked = false;
  if (stacking == ChainStacking::kAll && np_row >= 2) {
    double one = 0.0;
    for (size_t k = 0; k < np_row; ++k)
      one += pair_cost(std::max(read_lengths[sr[2 * k]], read_lengths[sr[2 * k + 1]]), false);
    // decreasing length (the uniform read of an odd count comes last in sr)
    rc.desc.assign(sr.begin(), sr.begin() + 2 * np_row);
    std::stable_sort(rc.desc.begin(), rc.desc.end(), [&](uint32_t x, uint32_t y) {
      return read_lengths[x] > read_lengths[y];
    });
    stacked = stack_pairs(read_lengths, geoms, false, rc.desc, np_row, one, rc);
  }
  for (size_t k = 0; k < np_row && !stacked; ++k) add_pair(sr[2 * k], sr[2 * k + 1]);
  if (m & 1) {  // odd per-row reads and no uniform one
    rc.leftover = sr[m - 1];
    return;
  }
  const size_t nU = sr.size() - m;  // uniform reads sr[m..), increasing length
  if (nU == 0) return;
  const size_t np = nU / 2;
  stacked = false;
  if (stacking != ChainStacking::kNone && np >= 2) {
    // (an odd count's leftover costs half a one-pair item: the longest read's
    // without stacking, the shortest one's with it)
    double one = 0.0;
    for (size_t i = m; i + 1 < sr.size(); i += 2) one += pair_cost(read_lengths[sr[i + 1]], true);
    if (nU & 1)
      one += 0.5 * (pair_cost(read_lengths[sr.back()], true) - pair_cost(read_lengths[sr[m]], true));
    rc.desc.assign(sr.rbegin(), sr.rend() - m);
    stacked = stack_pairs(read_lengths, geoms, true, rc.desc, np, one, rc);
  }
  if (stacked) {
    if (nU & 1) rc.leftover = sr[m];
    return;
  }
  size_t i = m;
  for (; i + 1 < sr.size(); i += 2) add_pair(sr[i], sr[i + 1]);
  if (i < sr.size()) rc.leftover = sr[i];
}

}  // namespace rodv
