// chain_plan.h -- how the packer turns a region's single-pass reads into
// chain items (host only, no device calls): which reads pair up, which pairs
// share an item's lanes, and which work class each item runs in.
#pragma once
#include <cstdint>
#include <vector>

#include "engine.h"

namespace rodv {

// A class's chain kernel as packed: an item holds `lanes` lanes
// of `rows` rows each (two items of 16 lanes with 2R rows per warp for the
// lane-grouped variants); `cost` is the relative time of one item.
struct ChainGeom {
  int cls;
  uint32_t lanes, rows;
  double cost;
};

// g[uniform][R], R = 1..8, and the uniform classes' as the stacking decision
// takes them.
struct ChainGeoms {
  ChainGeom g[2][kMaxRowsPerLane + 1];
  ChainGeom decide[kMaxRowsPerLane + 1];
};

// Which read pairs may share an item's lanes: none, uniform-gap ones, or all.
enum class ChainStacking { kNone, kUniform, kAll };

// One chain item: its class and read pairs, reads[first, first + 2 * pairs)
// of the region's RegionChains (x, then y or kNoPair).
struct ChainPairs {
  int cls;
  uint32_t first, pairs;
};

// The chain items of one region, its leftover read (kNoPair: none) and the
// planner's scratch (reused across regions by one thread).
struct RegionChains {
  std::vector<uint32_t> reads;
  std::vector<ChainPairs> items;
  uint32_t leftover = kNoPair;
  std::vector<uint32_t> desc, pair_item, item_free, item_fill, item_lens;
  std::vector<int> item_cls;
  std::vector<uint32_t> bucket[kWarp + 1];
};

// The geometry from the chain items per warp of each class's packed kernel
// variant (items_per_warp[uniform][R]: 1, or 2 for the lane-grouped ones).
void chain_geometry(const int (&items_per_warp)[2][kMaxRowsPerLane + 1], ChainGeoms& geoms);

// Lanes of `rows` rows that a read pair takes whose longer read has len
// bases: its rows, a pass-through row and, in the uniform-gap form, the sum
// row.
inline uint32_t pair_lanes(uint32_t len, uint32_t rows, bool uniform) {
  return (len + (uniform ? 1u : 0u)) / rows + 1;
}

// The single-pass reads read_start .. read_start + num_reads - 1 (read_class[r]
// of each, multi-pass ones left out), in increasing (uniform gaps, length).
void sort_single_pass(const uint32_t* read_lengths, const uint8_t* read_class,
                      uint32_t read_start, uint32_t num_reads, std::vector<uint32_t>& out);

// The chain items of a region's sorted single-pass reads sr (sort_single_pass).
// Reads with per-row gap priors -- and, where their count is odd, the shortest
// uniform read, which then takes per-row priors too -- pair up; so do the
// uniform-gap reads.  Without stacking, neighbours in increasing length pair
// up, one pair per item, in the class of the pair's longer read, and an odd
// last read is the region's leftover.  Stacked (stack_pairs), where the cost
// table finds it cheaper: neighbours in decreasing length pair up and several
// pairs share an item; the leftover is the shortest uniform read, or the
// longest per-row one (a leftover's result is rounded differently from a
// pair's, so which read it is must not depend on the stacking of per-row
// reads).  Depends on the region's reads only.
void plan_region_chains(const uint32_t* read_lengths, const uint8_t* read_class,
                        const ChainGeoms& geoms, ChainStacking stacking,
                        const std::vector<uint32_t>& sr, RegionChains& rc);

}  // namespace rodv
