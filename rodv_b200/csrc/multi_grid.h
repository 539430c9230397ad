// multi_grid.h -- grids of the multi-pass launches (host only).
#pragma once
#include <algorithm>

namespace rodv {

// Blocks of a launch of `items` items where `resident` blocks fit the GPU.  Up to
// max_rounds items a block, every block gets as many.
inline int even_blocks(int resident, int items, int max_rounds) {
  const int blocks = std::max(1, std::min(resident, items));
  const int rounds = (items + blocks - 1) / blocks;
  return rounds > 1 && rounds <= max_rounds ? (items + rounds - 1) / rounds : blocks;
}

// FP32 items have two passes in flight, so a block of four warps sweeps two items
// at a time (540 pairs of reads of 850 x 4,300 bases: 1.68 ms on 444 blocks,
// 1.38 on 270 of two items each).
constexpr int kEvenRoundsF32 = 3;
// FP64 items have every pass in flight that a warp is free for: grids are even
// as long as a block's warps hold all passes of all its items, the longest
// having `passes` (460 items of 300-500 bases, two passes: 0.90 ms on 444 blocks
// of four warps, 0.68 on 230).  Beyond that one item fills its block, and fewer
// blocks leave warps of the GPU idle (600 items of 1,000-2,000 bases: 2.45 ms on
// 300 blocks, 2.09 on 444; per-row gaps, 300 items: 2.54 on 150, 1.94 on 296).
inline int even_rounds_f64(int passes, int warps) {
  return warps / std::max(1, std::min(passes, warps));
}

// Whether FP32 uniform-gap launches whose grids have `warps` warps, all launches
// that run beside one another together, take the kernels built for few blocks:
// where they fit at 8 warps per SM, their items' sweeps are shorter (pairs of
// reads of about 1,500 x 4,350 bases, 18 items 1.08 -> 1.04 ms, 540 in 270 blocks
// 2.70 -> 2.59).  Above that, the resident warps count for more (2,160 such
// items 7.78 ms at 12 warps per SM, 8.64 at 8).
inline bool takes_few(long warps, int sms) { return warps <= 8L * sms; }

}  // namespace rodv
