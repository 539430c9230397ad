// kernel_table.cuh -- KernelInfo of every forward-kernel instantiation.
//
// Each rows-per-lane value R is instantiated in its own translation unit
// (kernels_r<R>.cu; multi-pass strip heights in kernels_multi_r<R>.cu) so the
// ~150 kernels compile in parallel.
#pragma once
#include <type_traits>

#include "kernels.h"
#include "pairhmm_fwd.cuh"
#include "pairhmm_pipe.cuh"

namespace rodv {

template <class P, int R, int GAPS, bool MU, bool SAME, int MINB, int GROUP = 32>
KernelInfo make_info(int variant) {
  using F = Forward<P, R, GAPS, MU, SAME, MINB, GROUP>;
  KernelInfo k;
  k.fn = reinterpret_cast<const void*>(&forward_kernel<P, R, GAPS, MU, SAME, MINB, GROUP>);
  k.threads = F::kWarpsPerBlock * kWarp;
  k.warps_per_block = F::kWarpsPerBlock;
  k.smem_bytes = F::kWarpsPerBlock * F::kSmemPerWarp;
  k.rows_per_lane = R;
  k.uniform = GAPS != kGapsPerRow;
  k.multi = MU;
  k.same_hap = SAME || P::kSlots == 1;
  k.chain = F::kChain;
  k.items_per_warp = F::kGroups;
  k.items_per_block = F::kWarpsPerBlock * F::kGroups;
  k.min_blocks = MINB;
  k.variant = variant;
  return k;
}

// Multi-pass kernels: a pool of passes on the W warps of a block.
template <class P, int R, int GAPS, bool SAME, int W, int WARPS = 12>
KernelInfo make_pipe_info(int variant) {
  // 168 registers (12 warps per SM) in the scaled form, 8 warps for launches
  // of few blocks; per-row kernels keep five coefficients a row
  constexpr int kMinBlocks = GAPS == kGapsPerRow ? 1 : WARPS / W;
  using F = PipeForward<P, R, GAPS, SAME, kMinBlocks, W>;
  KernelInfo k;
  k.fn = reinterpret_cast<const void*>(&forward_pipe_kernel<P, R, GAPS, SAME, kMinBlocks, W>);
  k.threads = W * kWarp;
  k.warps_per_block = W;
  k.smem_bytes = W * F::kSmemPerWarp;
  k.rows_per_lane = R;
  k.uniform = GAPS != kGapsPerRow;
  k.multi = true;
  k.same_hap = SAME || P::kSlots == 1;
  k.chain = false;
  k.items_per_warp = 1;
  k.items_per_block = 1;
  k.min_blocks = kMinBlocks;
  k.boundary_rows = F::kRows;
  k.variant = variant;
  return k;
}

// The FP64 kernel of the single-pass classes of up to HI rows per lane.
template <int GAPS, int HI>
KernelInfo make_rescue_info() {
  using F = Forward<F64, HI, GAPS, false, false, 1>;
  KernelInfo k;
  k.fn = reinterpret_cast<const void*>(&rescue_kernel<GAPS, HI>);
  k.threads = F::kWarpsPerBlock * kWarp;
  k.warps_per_block = F::kWarpsPerBlock;
  k.smem_bytes = F::kWarpsPerBlock * F::kSmemPerWarp;
  k.rows_per_lane = HI;
  k.uniform = GAPS != kGapsPerRow;
  k.same_hap = true;
  k.items_per_block = F::kWarpsPerBlock;
  return k;
}
// The one with the fewest rows that has the class of `rows` rows per lane.
template <int GAPS>
KernelInfo rescue_info_for(int rows) {
  if constexpr (GAPS == kGapsPerRow) {
    if (rows <= kRescueRows[0]) return make_rescue_info<GAPS, kRescueRows[0]>();
    if (rows <= kRescueRows[1]) return make_rescue_info<GAPS, kRescueRows[1]>();
    if (rows <= kRescueRows[2]) return make_rescue_info<GAPS, kRescueRows[2]>();
  }
  return make_rescue_info<GAPS, kMaxRowsPerLane>();
}

// The multi-pass variants of strip height R (pipe_variant_rows) for one
// precision, gap form and item kind: W = 2 or 4 warps per block.
template <int R, int GAPS>
KernelInfo pipe_gap_info(Precision prec, bool same, int variant) {
  const bool w4 = pipe_variant_warps(variant) == 4;
  if (prec == Precision::kF64)
    return w4 ? make_pipe_info<F64, R, GAPS, false, 4>(variant)
              : make_pipe_info<F64, R, GAPS, false, 2>(variant);
  if constexpr (GAPS != kGapsPerRow) {
    if (variant & kPipeFew) {
      if (same)
        return w4 ? make_pipe_info<F32x2, R, GAPS, true, 4, 8>(variant)
                  : make_pipe_info<F32x2, R, GAPS, true, 2, 8>(variant);
      return w4 ? make_pipe_info<F32x2, R, GAPS, false, 4, 8>(variant)
                : make_pipe_info<F32x2, R, GAPS, false, 2, 8>(variant);
    }
  }
  if (same)
    return w4 ? make_pipe_info<F32x2, R, GAPS, true, 4>(variant)
              : make_pipe_info<F32x2, R, GAPS, true, 2>(variant);
  return w4 ? make_pipe_info<F32x2, R, GAPS, false, 4>(variant)
            : make_pipe_info<F32x2, R, GAPS, false, 2>(variant);
}

template <int R>
KernelInfo pipe_info_for(Precision prec, GapForm gaps, bool same, int variant) {
  switch (gaps) {
    case kGapsPerRow: return pipe_gap_info<R, kGapsPerRow>(prec, same, variant);
    case kGapsUniform: return pipe_gap_info<R, kGapsUniform>(prec, same, variant);
    default: return pipe_gap_info<R, kGapsConst>(prec, same, variant);
  }
}

// Same-haplotype FP32 kernels come in occupancy targets (variant_min_blocks);
// the chain kernels of reads up to 128 bases (R <= 4) also in a lane-grouped
// form: two 16-lane groups per warp, each sweeping its own chain item with
// 2R rows per lane, so that each lane's per-step overhead (shuffles, code and
// table loads, row-0 selects) covers twice the rows (faster on B200 at R <= 3
// and, with per-row gaps, R = 4; slower at uniform R = 4, where the longer
// per-step dependency chain shows; the autotuner picks).  Every other kernel has one variant.
template <class P, int R, int GAPS, bool MU, bool SAME>
KernelInfo variant_info(int variant) {
  if constexpr (!(std::is_same<P, F32x2>::value && SAME)) {
    (void)variant;
    return make_info<P, R, GAPS, MU, SAME, 1>(0);
  } else {
    constexpr bool kRow = GAPS == kGapsPerRow;
    if constexpr (!MU && R <= kMaxGroupedRows) {
      switch (variant) {
        case 4: return make_info<P, 2 * R, GAPS, MU, SAME, variant_min_blocks(4, 2 * R, kRow), 16>(4);
        case 5: return make_info<P, 2 * R, GAPS, MU, SAME, variant_min_blocks(5, 2 * R, kRow), 16>(5);
        case 6: return make_info<P, 2 * R, GAPS, MU, SAME, variant_min_blocks(6, 2 * R, kRow), 16>(6);
        case 7: return make_info<P, 2 * R, GAPS, MU, SAME, variant_min_blocks(7, 2 * R, kRow), 16>(7);
        default: break;
      }
    }
    switch (variant) {
      case 0: return make_info<P, R, GAPS, MU, SAME, variant_min_blocks(0, R, kRow)>(0);
      case 1: return make_info<P, R, GAPS, MU, SAME, variant_min_blocks(1, R, kRow)>(1);
      case 2: return make_info<P, R, GAPS, MU, SAME, variant_min_blocks(2, R, kRow)>(2);
      default: return make_info<P, R, GAPS, MU, SAME, variant_min_blocks(3, R, kRow)>(3);
    }
  }
}

template <int R, bool MU, int GAPS>
KernelInfo gap_info(bool same, int variant) {
  if (same) return variant_info<F32x2, R, GAPS, MU, true>(variant);
  // Two-haplotype items: multi-pass leftovers, and the odd single-pass read
  // of a region against each of its haplotypes.
  return variant_info<F32x2, R, GAPS, MU, false>(0);
}

template <int R, bool MU>
KernelInfo info_for(GapForm gaps, bool same, int variant) {
  switch (gaps) {
    case kGapsPerRow: return gap_info<R, MU, kGapsPerRow>(same, variant);
    case kGapsUniform: return gap_info<R, MU, kGapsUniform>(same, variant);
    default: return gap_info<R, MU, kGapsConst>(same, variant);
  }
}

}  // namespace rodv
