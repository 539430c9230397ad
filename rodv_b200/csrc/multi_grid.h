// multi_grid.h -- grids of the multi-pass launches (host only).
#pragma once
#include <algorithm>

namespace rodv {

// Blocks of a launch of `items` items where `resident` blocks fit the GPU.  Up to
// three items a block, every block gets as many (540 pairs of reads of 850 x
// 4,300 bases: 1.68 ms on 444 blocks, 1.38 on 270 of two items each).
inline int even_blocks(int resident, int items) {
  const int blocks = std::max(1, std::min(resident, items));
  const int rounds = (items + blocks - 1) / blocks;
  return rounds > 1 && rounds <= 3 ? (items + rounds - 1) / rounds : blocks;
}

// Whether FP32 uniform-gap launches whose grids have `warps` warps, all launches
// that run beside one another together, take the kernels built for few blocks:
// where they fit at 8 warps per SM, their items' sweeps are shorter (pairs of
// reads of about 1,500 x 4,350 bases, 18 items 1.08 -> 1.04 ms, 540 in 270 blocks
// 2.70 -> 2.59).  Above that, the resident warps count for more (2,160 such
// items 7.78 ms at 12 warps per SM, 8.64 at 8).
inline bool takes_few(long warps, int sms) { return warps <= 8L * sms; }

}  // namespace rodv
