// pairhmm_pipe.cuh -- multi-pass sweeps of long reads: the passes of a block's
// work items run concurrently on the warps of the block.
//
// A read longer than one pass (32 lanes x R rows) is swept in passes of 32R
// rows; pass p needs the last row of pass p-1 (its boundary row) column by
// column.  Swept one pass after the other by one warp, a pair of a 2,000-base
// read and a 5,000-base haplotype takes 8 x 5,031 steps in sequence, and the
// longest pairs of a batch set the length of the whole launch.  Here lane 31 of
// the warp on pass p writes the pass's last row into a boundary row in global
// memory and publishes, after every 32 steps, how far it has come; lane 0 of the
// warp on pass p+1 reads that row through a shared-memory ring (cp.async, 32
// columns ahead), waiting for the publication before each chunk.  Pass p+1 can
// thus trail pass p by about 100 steps instead of a whole pass.
//
// Tasks.  A block's W warps take passes one by one (acquire): a warp that ends
// one takes the next, of the same item or of another, with no barrier between
// items.  (With a team of W warps per item, warp w on passes w, w+W, ..., and a
// block barrier at its end, six passes kept four warps busy three quarters of
// the time, and a rejected item's W passes in flight were all swept.)  An open
// item -- one with a pass started and not all ended -- occupies one of W slots.
// The choice, in this order: the oldest open item's next pass, if fewer than
// kWindow of its started passes have yet to end; a new item from the queue, up
// to the block's even share of the queue; any open item's next pass; a new
// item.  A block's first item is the one of its own number, so that blocks which
// open two leave every block one (540 items on 444 blocks: 2.0 ms when 270
// blocks took two each, 1.7 so).  FP32 items are held to two passes in flight, so that an item rejected
// after a pass (below) has swept at most one pass more; a queue too short to
// fill the block lifts that.  FP64 items take every pass as soon as a warp is
// free: the longest item comes first and ends soonest.  Measured with the team
// of four warps before: 1,500 pairs of 1,500 x 3,500 bases 2.87 -> 2.55 ms in
// FP32, 1.70 -> 1.31 where every pair is rejected, 4.83 -> 4.28 in FP64.
//
// What crosses a pass boundary is what the lanes of a warp hand each other.
// In the scaled form (uniform gaps) that is two values per column: the M term
// of the row below, t = (mm/c) M~ + I^ + D^ (used one column later), and the
// row below's I^ = ii' I^ + M~ (ii' of the row below), both computed by the
// lane above with the operations the lane below would apply, so the results
// are bitwise those of a three-value hand-over of (M~, I^, D^).  Other forms
// hand over (M, I, D).  A boundary cell is 16 or 24 bytes.
//
// Boundary rows.  A block owns 2W rows; a started pass but the last owns one
// until both it and the pass that reads it have ended (an item that is closed
// early keeps its rows until its last pass in flight has ended).  W-1 other
// warps are in passes, each with two rows at most, and an item between passes
// keeps one, so a row is free for every pass; only while a closed item's last
// pass leaves may a warp have to look again.  Every
// wait is a pass waiting for the item's previous pass, which was started before
// it: waits cannot form a cycle.  Each wait also gives up after a bounded number
// of polls, sets kErrWaitTimeout and stops the block's warps, so a kernel always
// ends.  A row starts with kPad cells before its column 0: lane 31 stores its
// hand-over every step, the first of which are columns <= 0 (zeros, never read),
// so no store needs a column test.
//
// Progress words live in shared memory: (pass << 17) | column, written with a
// CTA-scope release by the producing lane after its row stores, read with a CTA-scope acquire by every lane of the consumer before
// it copies the chunk.  The warps are in one block, so they share the SM's
// L1 and the CTA scope suffices.  The rest of the block's state (Ctl) is
// changed by one lane at a time under a lock.
//
// FP32 items stop early as in the single-warp sweep: after each pass but the
// last, the warp that swept it bounds the likelihood by the sum over the row
// it wrote (rejects(), the bound of Forward::row_bound_rejects restated for
// the hand-over cells); once both slots are below the acceptance bound the
// item is closed and both pairs go to FP64.  The bound is exact, so the
// rescued pairs and every result are those of the full sweep.
//
// The per-cell arithmetic is the single-warp sweeps' (Forward::cells_scaled,
// Forward::cells for per-row gaps), and the pass count (pipe_passes, layout.h) leaves at least one pass-through row at
// the end, so a result is always the column sum of the I of a pass-through
// row (its M is 0): it depends neither on W nor on the strip height R nor on
// the item's other read.
#pragma once
#include <type_traits>

#include "pairhmm_fwd.cuh"

namespace rodv {

__device__ __forceinline__ uint32_t ld_acquire_cta(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.cta.shared.u32 %0, [%1];"
               : "=r"(v)
               : "r"((unsigned)__cvta_generic_to_shared(p))
               : "memory");
  return v;
}
__device__ __forceinline__ void st_release_cta(uint32_t* p, uint32_t v) {
  asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(p)),
               "r"(v)
               : "memory");
}
// cp.async of 16 bytes global -> shared (L2 only); both addresses 16-byte aligned
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem) : "memory");
}

// Stores of boundary cells where `on` is set, as predicated instructions: a
// branch in every step would split the unrolled steps (as the separator test
// does in the chain sweeps).  No "memory" clobber: the loads of the following
// steps (codes, emissions, the ring) never read what they write and may move
// ahead of them.  The release that publishes the cells (st_release_cta) is a
// volatile asm too and stays behind them.
__device__ __forceinline__ void st_cell(bool on, void* p, float2 a, float2 b) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
      "@q st.global.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(p),
      "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "r"((uint32_t)on));
}
__device__ __forceinline__ void st_cell(bool on, void* p, double a, double b) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t"
      "@q st.global.v2.f64 [%0], {%1, %2};\n\t}" ::"l"(p),
      "d"(a), "d"(b), "r"((uint32_t)on));
}
__device__ __forceinline__ void st_cell(bool on, void* p, float2 a) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t"
      "@q st.global.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(p),
      "f"(a.x), "f"(a.y), "r"((uint32_t)on));
}
__device__ __forceinline__ void st_cell(bool on, void* p, double a) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
      "@q st.global.f64 [%0], %1;\n\t}" ::"l"(p),
      "d"(a), "r"((uint32_t)on));
}

template <class P, int R, int GAPS, bool SAME, int MINB, int W>
struct PipeForward {
  using F = Forward<P, R, GAPS, true, SAME, MINB>;
  using V = typename P::V;
  using S = typename P::S;
  static constexpr bool kTwo = F::kScaled;  // two-value hand-over (t, i)
  struct HandCell {
    V t, i;
  };
  using Cell = typename std::conditional<kTwo, HandCell, typename F::BoundaryCell>::type;
  static_assert(sizeof(Cell) <= 24, "the engine sizes boundary rows at 24 bytes a cell");
  static constexpr int kRows = 2 * W;                   // boundary rows per block
  // Chunks between two looks at the stop word.
  static constexpr int kStopChunks = 4;
  // started passes of an item that may be in flight before it has to wait
  static constexpr uint32_t kWindow = P::kSlots == 2 ? 2u : ~0u;
  // Columns a lane runs behind its left neighbour.  FP64 (two-value form): two,
  // so a value shuffled in one step is used in the next (Forward::run_single).
  static constexpr int kLag = kTwo && P::kSlots == 1 ? 2 : 1;
  static constexpr int kPad = kLag * kWarp;             // cells before column 0 of a row
  static_assert(kPad + 8 <= kBoundaryPad, "the engine sizes boundary rows");
  // Steps per loop iteration of a whole chunk: eight at 168 registers (12 warps
  // per SM).  4,440 pairs of 1,500 x 3,500 bases: FP32 6.48 ms, FP64 11.2 (four
  // steps 6.46 and 11.3, sixteen 6.34 and 11.5); at 128 registers and 16 warps,
  // with spills, 6.80 and 11.2 (four steps 6.78 and 12.1), and a lone item takes
  // 0.92 and 0.78 ms instead of 0.81 and 0.72.
  // The kernels for few blocks (FP32, 8 warps per SM) take four: a lone item of
  // two reads of 850 (1,500) x 4,300 bases 0.458 (0.875) ms, with eight 0.477
  // (0.908), at 12 warps 0.489 (0.932), four steps at 12 warps 0.483 (0.921).
  static constexpr bool kFew = P::kSlots == 2 && kTwo && MINB * W <= 8;
  static constexpr int kUnroll = kFew ? 4 : 8;
  // Where lane 0 alone reads its row above from the ring, in the step itself:
  // in FP64 the three-value form's cells (24 bytes) cost the other lanes more
  // than the load's latency costs lane 0.  20 pairs of 1,000-2,000 bases
  // 1.33 -> 1.24 ms, 100 pairs 1.41 -> 1.31, 1,500 pairs 6.45 -> 6.30 (four steps
  // an iteration, all lanes reading: 1.31, 1.38, 6.6).
  static constexpr bool kLoneRead = !kTwo && P::kSlots == 1;
  static constexpr int kSmemPerWarp = F::kSmemPerWarp;  // emission table + cell ring
  // polls of a progress word (about 100 ns each) before a wait gives up
  static constexpr uint32_t kWaitPolls = 1u << 24;
  static constexpr uint32_t kLockPolls = 1u << 22;

  enum : uint32_t { kFree = 0, kOpen = 1, kClosed = 2 };  // Open::state
  struct Open {
    uint32_t state;
    uint32_t item, passes;
    uint32_t next;       // first pass not started
    uint32_t done;       // passes ended
    uint32_t running;    // passes in flight
    uint32_t rows;       // boundary rows held (bits)
    uint32_t wrote, read;  // of these: the pass that writes it, that reads it, has ended
    uint32_t last_row;   // of the last pass started
  };
  // A warp's pass.
  struct Task {
    uint32_t slot, item, pass, passes, in_row, out_row;
    bool last;
  };
  struct Ctl {
    uint32_t ticket, serving;  // the lock: next ticket, the ticket that holds it
    uint32_t broken;     // a warp gave up its ticket: the lock serves nobody any more
    uint32_t fail;       // a wait expired: every warp stops
    uint32_t started;    // the block's first item is taken
    uint32_t scanning;   // a warp is taking the queue's next item
    uint32_t exhausted;  // the queue is empty
    uint32_t num_open;
    uint32_t free_rows;  // bits
    uint32_t stop[W];    // per warp: its item is closed
    Task task[W];        // per warp
    Open open[W];
    uint32_t prog[kRows];  // per boundary row: (pass << 17) | last column published
  };

  __device__ __forceinline__ static uint32_t enc(uint32_t pass, uint32_t col) {
    return (pass << 17) | col;
  }

  // Whether this warp has to leave its pass (its item is closed, or a wait
  // expired), the same in every lane.
  __device__ __forceinline__ static bool stopped(Ctl& ctl, int warp) {
    return __any_sync(kFullMask, (*reinterpret_cast<volatile uint32_t*>(&ctl.stop[warp]) |
                                  *reinterpret_cast<volatile uint32_t*>(&ctl.fail)) != 0u);
  }

  // The block's lock, taken by one lane; false if it was not to be had (which
  // stops the block).  Tickets are served in order: with a test-and-set word,
  // warps that look again and again (acquire) can keep one that ends its pass
  // from ever finding the lock free, since their sleeps end in step.
  __device__ static bool lock(Ctl& ctl, const ClassLaunch& c) {
    const uint32_t polls = c.wait_polls ? c.wait_polls : kLockPolls;
    const uint32_t mine = atomicAdd(&ctl.ticket, 1u);
    for (uint32_t k = 0; *reinterpret_cast<volatile uint32_t*>(&ctl.serving) != mine; ++k) {
      if (*reinterpret_cast<volatile uint32_t*>(&ctl.broken)) return false;
      if (k >= polls) {
        atomicOr(c.error_flags, kErrWaitTimeout);
        atomicExch(&ctl.broken, 1u);
        atomicExch(&ctl.fail, 1u);
        return false;
      }
      __nanosleep(32);
    }
    __threadfence_block();
    return true;
  }
  __device__ static void unlock(Ctl& ctl) {
    __threadfence_block();
    atomicAdd(&ctl.serving, 1u);
  }

  // The queue's next valid item and its passes; kNoPair when the queue is empty.
  __device__ static uint32_t next_item(const BatchView& b, const ClassLaunch& c, uint32_t n,
                                       Ctl& ctl, uint32_t& passes) {
    for (;;) {
      // the block's first item is its own: another block that opens two at once
      // must not leave it without
      const uint32_t item = ctl.started ? gridDim.x + atomicAdd(c.counter, 1u) : blockIdx.x;
      ctl.started = 1u;
      if (item >= n) return kNoPair;
      PairRef refs[2];
      F::load_refs(c, item, refs);
      // an FP64 list position that no rescue filled (kLaunchRescueByItem lists)
      if (P::kSlots == 1 && refs[0].read == kNoPair) continue;
      if (refs[1].read == kNoPair) refs[1] = refs[0];
      const HapDesc hx = b.haps[refs[0].hap], hy = b.haps[refs[1].hap];
      const uint32_t lx = b.reads[refs[0].read].len, ly = b.reads[refs[1].read].len;
      // slot x has the longer haplotype
      if (hx.len == 0 || hy.len == 0 || lx == 0 || ly == 0 ||
          (F::kSameHap && hx.code_off != hy.code_off) || hy.len > hx.len ||
          (uint64_t)hx.len + kPad + 8 > c.scratch_cols) {
        atomicOr(c.error_flags, kErrBadLength);
        continue;
      }
      passes = pipe_passes(lx > ly ? lx : ly, R);
      return item;
    }
  }

  // The same out of line, for the kernel whose sweep is a hundredth slower with it
  // in line (kLoneRead; the others' are with the call).
  __device__ __noinline__ static uint32_t next_item_call(const BatchView& b, const ClassLaunch& c,
                                                         uint32_t n, Ctl& ctl, uint32_t& passes) {
    return next_item(b, c, n, ctl, passes);
  }

  // Opens `item` (next_item) in a free slot, of which there is one; its slot, or -1
  // if the queue was empty.  Under the lock.
  __device__ static int open_item(Ctl& ctl, uint32_t item, uint32_t passes) {
    if (item == kNoPair) {
      ctl.exhausted = 1u;
      return -1;
    }
    int slot = 0;
    while (slot < W - 1 && ctl.open[slot].state != kFree) ++slot;
    ctl.open[slot] = Open{kOpen, item, passes, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
    ++ctl.num_open;
    return slot;
  }

  // Takes the queue's next item for the lane whose try_acquire returned kScan (and
  // set ctl.scanning, so that no other takes one meanwhile), outside the lock: an
  // FP64 list of 1e8 positions that no rescue filled keeps a block looking for
  // half a second.  False if the lock was not to be had.
  __device__ static bool scan(const BatchView& b, const ClassLaunch& c, uint32_t n, Ctl& ctl) {
    uint32_t passes = 0;
    const uint32_t item = kLoneRead ? next_item_call(b, c, n, ctl, passes)
                                    : next_item(b, c, n, ctl, passes);
    if (!lock(ctl, c)) return false;
    ctl.scanning = 0u;
    open_item(ctl, item, passes);
    unlock(ctl);
    return true;
  }

  // The next pass for this warp, in ctl.task[warp]; false (in every lane) when
  // there is none.  max_open: the block's even share of the queue.
  __device__ static bool acquire(const BatchView& b, const ClassLaunch& c, uint32_t n,
                                 uint32_t max_open, int warp, int lane, Ctl& ctl) {
    int got = kNone;
    for (uint32_t tries = 0;; ++tries) {
      if (lane == 0) {
        while ((got = try_acquire(b, c, n, max_open, warp, ctl)) == kScan)
          if (!scan(b, c, n, ctl)) {
            got = kNone;
            break;
          }
        // a scan ends by itself, however long the list
        if (*reinterpret_cast<volatile uint32_t*>(&ctl.scanning)) tries = 0;
      }
      got = __shfl_sync(kFullMask, got, 0);
      __syncwarp();  // ctl.task[warp] is visible to the whole warp
      if (got != kLater) return got == kPass;
      if (__shfl_sync(kFullMask, tries, 0) >= kLockPolls) {
        if (lane == 0) {
          atomicOr(c.error_flags, kErrWaitTimeout);
          atomicExch(&ctl.fail, 1u);
        }
        return false;
      }
      __nanosleep(200);
    }
  }

  // One try, by one lane.  kNone: no pass is left to start.  kLater: another
  // warp is taking an item off the queue, or every row or slot is held by items
  // that are being closed (their last passes end within kStopChunks chunks).
  // kScan: a new item is wanted, and this lane is to take it (scan).  FP32 lists
  // have no empty positions: their next item is taken under the lock.
  enum : int { kNone, kPass, kLater, kScan };
  __device__ static int try_acquire(const BatchView& b, const ClassLaunch& c, uint32_t n,
                                    uint32_t max_open, int warp, Ctl& ctl) {
    if (!lock(ctl, c)) return kNone;
    auto oldest = [&](uint32_t window) {
      int best = -1;
      for (int k = 0; k < W; ++k) {
        const Open& o = ctl.open[k];
        if (o.state == kOpen && o.next < o.passes && o.next - o.done < window &&
            (best < 0 || o.item < ctl.open[best].item))
          best = k;
      }
      return best;
    };
    int k = -1, got = kNone;
    if (!ctl.fail) {
      const bool can_open = !ctl.exhausted && !ctl.scanning && ctl.num_open < W;
      k = oldest(kWindow);
      if (P::kSlots == 2) {
        uint32_t passes = 0;
        if (k < 0 && can_open && ctl.num_open < max_open)
          k = open_item(ctl, next_item(b, c, n, ctl, passes), passes);
        if (k < 0) k = oldest(~0u);
        if (k < 0 && can_open && !ctl.exhausted)
          k = open_item(ctl, next_item(b, c, n, ctl, passes), passes);
      } else if (k < 0 && can_open) {  // (kWindow takes every pass that can start)
        // kLoneRead, up to two items a block: the further one waits until half the
        // block's warps are free for it.  Begun by one warp, it ends a whole pass
        // later than in a block whose item ends next (400 pairs of 1,000-2,000
        // bases on 296 blocks: 2.37 -> 2.22 ms; 1,500 pairs 6.37 -> 6.52).
        uint32_t running = 0;
        for (int w = 0; w < W && kLoneRead && max_open <= 2u; ++w)
          running += ctl.open[w].state != kFree ? ctl.open[w].running : 0u;
        if (running <= W / 2) {
          got = kScan;
          ctl.scanning = 1u;
        }
      }
      if (k < 0 && got == kNone && !ctl.exhausted) got = kLater;
    }
    if (k >= 0) {
      Open& o = ctl.open[k];
      Task t;
      t.slot = (uint32_t)k;
      t.item = o.item;
      t.pass = o.next;
      t.passes = o.passes;
      t.last = t.pass + 1 == o.passes;
      t.in_row = o.last_row;
      t.out_row = 0;
      if (!t.last && ctl.free_rows == 0u) {
        got = kLater;
      } else {
        if (!t.last) {
          t.out_row = (uint32_t)__ffs((int)ctl.free_rows) - 1u;
          ctl.free_rows &= ~(1u << t.out_row);
          ctl.prog[t.out_row] = 0u;
          o.rows |= 1u << t.out_row;
          o.last_row = t.out_row;
        }
        ++o.next;
        ++o.running;
        ctl.stop[warp] = 0u;
        ctl.task[warp] = t;
        got = kPass;
      }
    }
    unlock(ctl);
    return got;
  }

  // Closes this warp's item, if it is still open, and stops the other warps on
  // it; whether this warp closed it (the same in every lane): it then writes the
  // item's results or rescues.
  __device__ static bool close(const ClassLaunch& c, int warp, int lane, Ctl& ctl) {
    bool won = false;
    if (lane == 0 && lock(ctl, c)) {
      const uint32_t slot = ctl.task[warp].slot;
      if (ctl.open[slot].state == kOpen && !ctl.stop[warp] && !ctl.fail) {
        ctl.open[slot].state = kClosed;
        for (int w = 0; w < W; ++w)
          if (w != warp && ctl.task[w].slot == slot) ctl.stop[w] = 1u;
        won = true;
      }
      unlock(ctl);
    }
    return __shfl_sync(kFullMask, (int)won, 0) != 0;
  }

  // The end of this warp's pass; swept: to its last column.
  __device__ static void release(const ClassLaunch& c, int warp, int lane, Ctl& ctl, bool swept) {
    __syncwarp();
    if (lane == 0 && lock(ctl, c)) {
      const Task t = ctl.task[warp];
      Open& o = ctl.open[t.slot];
      auto give_back = [&](uint32_t bits) {
        o.rows &= ~bits;
        o.wrote &= ~bits;
        o.read &= ~bits;
        ctl.free_rows |= bits;
      };
      --o.running;
      if (swept) {
        // a row is free once its writer has ended (it may still be summing the
        // row) and its reader has read it all
        if (t.pass > 0) o.read |= 1u << t.in_row;
        if (!t.last) o.wrote |= 1u << t.out_row;
        give_back(o.read & o.wrote);
        o.done = o.done > t.pass + 1 ? o.done : t.pass + 1;
      }
      if (o.state == kClosed && o.running == 0) {
        give_back(o.rows);
        o.state = kFree;
        --ctl.num_open;
      }
      ctl.task[warp].slot = W;  // none
      unlock(ctl);
    }
    __syncwarp();
  }

  // The whole warp waits until *word >= want; false (in every lane) when its
  // item was closed meanwhile or the wait expired (which stops the block).
  __device__ static bool wait_word(Ctl& ctl, int warp, const uint32_t* word, uint32_t want,
                                   uint32_t* err, uint32_t polls) {
    for (uint32_t k = 0;; ++k) {
      if (__all_sync(kFullMask, ld_acquire_cta(word) >= want)) return true;
      if (stopped(ctl, warp)) return false;
      if (k >= polls) {
        if ((threadIdx.x & (kWarp - 1)) == 0) {
          atomicOr(err, kErrWaitTimeout);
          atomicExch(&ctl.fail, 1u);
        }
        __syncwarp();
        return false;
      }
      __nanosleep(64);
    }
  }

  // The FP32 early-rejection decision after a pass (the same value in every
  // lane), from the hand-over cells of the pass's last row r.  With c = mi
  // gapm, t = (mm/gapm) M~/mi + I^ + D^ >= min(1, mm/gapm) (M~/mi + I^), so
  // max(1, gapm/mm) sum_j t bounds the sum Forward::row_bound_rejects bounds
  // the likelihood by (sum M~/mi + sum I^, rows r < L); a pass-through row
  // (r >= L) has M~ = D^ = 0 and t = I^, and its bound is sum t / mi.  The
  // acceptance test and its 1e-6 margin are the same.
  __device__ static bool rejects(const BatchView& b, const ClassLaunch& c, const Cell* row0,
                                 const uint32_t (&H)[2], const uint32_t (&L)[2], uint32_t row,
                                 int lane, uint32_t item) {
    if constexpr (!kTwo) {
      return F::row_bound_rejects(c, row0, H, lane, item);
    } else {
      V st = P::zero();
      for (uint32_t col = 1 + (uint32_t)lane; col <= H[0]; col += kWarp) {
        const V t = row0[col].t;
        st = P::add(st, P::make(P::sx(t), col <= H[1] ? P::sy(t) : S(0)));
      }
      double sum[2] = {(double)P::sx(st), (double)P::sy(st)};
#pragma unroll
      for (int d = 16; d >= 1; d /= 2) {
        sum[0] += __shfl_xor_sync(kFullMask, sum[0], d);
        sum[1] += __shfl_xor_sync(kFullMask, sum[1], d);
      }
      PairRef refs[2];
      F::load_refs(c, item, refs);
      bool rejected = true;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (s == 1 && refs[1].read == kNoPair) continue;
        const uint32_t w = b.read_rows[b.reads[refs[s].read].row_off];
        double mi, gapm;
        F::read_gaps(b, c.gaps, refs[s].read, &mi, &gapm);
        const double mm = (double)row_priors<S>(w, b.tab).mm;
        const double bound = row < L[s] ? (gapm > mm ? gapm / mm : 1.0) * sum[s] : sum[s] / mi;
        const double amin = (double)kMinAcceptedF / (mi * gapm);  // as scaled_result's
        rejected = rejected && mm > 0.0 && bound >= 0.0 && bound < amin * 1e-6;
      }
      return rejected;
    }
  }

  // Sweeps this warp's pass (ctl.task[warp]) and, as the warp that ends or
  // rejects its item, writes the item's results or rescues.
  __device__ static void run(const BatchView& b, const ClassLaunch& c, int warp, int lane,
                             uint4* table, Ctl& ctl, Cell* rows) {
    const uint32_t item = ctl.task[warp].item;
    const uint32_t p = ctl.task[warp].pass;
    PairRef refs[2];
    F::load_refs(c, item, refs);
    SlotInfo sl[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const bool valid = (s == 0) || refs[1].read != kNoPair;
      const PairRef r = valid ? refs[s] : refs[0];
      const HapDesc hd = b.haps[r.hap];
      const ReadDesc rd = b.reads[r.read];
      sl[s].hap = b.hap_codes + hd.code_off;
      sl[s].H = hd.len;
      sl[s].L = rd.len;
      sl[s].row_off = rd.row_off;
    }
    const uint32_t H = sl[0].H;
    const int nsteps = (int)H + kLag * (kWarp - 1);  // slot x has the longer haplotype
    // slot y's last accumulated step + 1
    const int nfreeze = (int)sl[1].H + kLag * (kWarp - 1);
    const V init = P::make(P::init_const() / (S)sl[0].H, P::init_const() / (S)sl[1].H);
    const uint32_t L[2] = {sl[0].L, sl[1].L};
    const uint64_t row_off[2] = {sl[0].row_off, sl[1].row_off};
    Cell* ring = reinterpret_cast<Cell*>(table + F::Shape::kBytesPerWarp / 16);
    const uint32_t polls = c.wait_polls ? c.wait_polls : kWaitPolls;
    const bool publish = (c.flags & kLaunchNoPublish) == 0;

    V acc = P::zero();  // column sum of the I of the last row
    S frozen = 0;       // slot y's, at its own last column (two-haplotype items)
    bool alive = true;
    {
      const bool store = !ctl.task[warp].last && lane == kWarp - 1;
      const int out_row = (int)ctl.task[warp].out_row;
      const int in_row = (int)ctl.task[warp].in_row;
      Cell* const out_cells = rows + (size_t)out_row * c.scratch_cols + kPad;  // column 0
      // lane 31's step s holds column s - 31 kLag + 1 after the step
      constexpr int kLastCol = kLag * (kWarp - 1) - 1;
      Cell* const dst = out_cells - kLastCol;
      const Cell* const src = rows + (size_t)in_row * c.scratch_cols + kPad;
      // cells of steps [32 k, 32 k + 32) from the previous pass's row
      // (columns 32 k + 1 .. 32 k + 32), copied once they are published
      auto fetch_chunk = [&](int k) -> bool {
        const uint32_t first = (uint32_t)k * kWarp + 1u;
        if (first <= H) {
          const uint32_t upto = first + kWarp - 1 < H ? first + kWarp - 1 : H;
          if (!wait_word(ctl, warp, &ctl.prog[in_row], enc(p - 1, upto), c.error_flags, polls))
            return false;
        }
        const uint32_t idx = first + (uint32_t)lane;
        if (idx + kPad < c.scratch_cols) {
          Cell* d = ring + (k & 1) * kWarp + lane;
          const Cell* s = src + idx;
          if constexpr (kTwo) {
            cp_async16(d, s);
          } else {
            cp_async8(&d->m, &s->m);
            cp_async8(&d->i, &s->i);
            cp_async8(&d->d, &s->d);
          }
        }
        cp_async_commit();
        return true;
      };

      typename F::Priors pr;
      const uint32_t fr = p * (kWarp * R) + lane * R;
      F::load_rows(b, c.gaps, L, row_off, {fr, fr}, lane, table, pr);
      V M[R], I[R], D[R];
#pragma unroll
      for (int k = 0; k < R; ++k) M[k] = I[k] = D[k] = P::zero();
      const bool from_ring = p > 0;
      if (from_ring) {
        alive = fetch_chunk(0);
      } else {
        // pass 0: lane 0's row above is row 0 of the DP at every column
        Cell top;
        if constexpr (kTwo) {
          top.t = init; top.i = P::zero();
        } else {
          top.m = P::zero(); top.i = P::zero(); top.d = init;
        }
        ring[lane] = top;
        ring[kWarp + lane] = top;
      }
      __syncwarp();
      uint32_t cx_next = sl[0].hap[-kLag * lane];
      uint32_t cy_next = F::kSameHap ? 0u : (uint32_t)sl[1].hap[-kLag * lane];
      const uint8_t* hx = sl[0].hap - kLag * lane + 1;  // code of the step after s: hx[s]
      const uint8_t* hy = sl[1].hap - kLag * lane + 1;
      // two-value form: this lane's hand-over for the lane below, and the M
      // term of its first row carried to the next column
      V h_t = P::zero(), h_i = P::zero();
      V next_t = P::zero(), next_i = P::zero();  // kLag 2: shuffled in the previous step
      V dg_t = (lane == 0 && p == 0) ? init : P::zero();
      // three-value form: the row above at the previous column
      V dg_m = P::zero(), dg_i = P::zero(), dg_d = (lane == 0 && p == 0) ? init : P::zero();

      // One step; i: the step of its chunk.  The sum of the last row is kept
      // in every pass (only the last pass's is used): a test in each step
      // cost more than the add.
      Cell cell_next;  // lane 0's row above in the next step, loaded a step ahead
      auto step = [&](int s, const Cell* now, const Cell* next) {
        const uint32_t cx = cx_next, cy = cy_next;
        cx_next = hx[s];
        if (!F::kSameHap) cy_next = hy[s];
        V e[R], t_last;
        Cell cl = cell_next;
        if (!kLoneRead) cell_next = *next;
        if constexpr (kTwo) {
          V in_t = P::shfl_up(h_t), in_i = P::shfl_up(h_i);
          if (kLag == 2) {
            const V t = in_t, i = in_i;
            in_t = next_t; in_i = next_i;
            next_t = t; next_i = i;
          }
          if (lane == 0) {
            in_t = cl.t; in_i = cl.i;
          }
          F::load_emission(table, lane, cx, cy, e);
          F::cells_scaled(e, dg_t, in_i, M, I, D, pr, t_last);
          dg_t = in_t;
          h_t = P::fma(pr.mmU, M[R - 1], P::add(I[R - 1], D[R - 1]));
          h_i = P::fma(pr.iiN, I[R - 1], M[R - 1]);
          st_cell(store, dst + s, h_t, h_i);
        } else {
          V up_m = P::shfl_up(M[R - 1]);
          V up_i = P::shfl_up(I[R - 1]);
          V up_d = P::shfl_up(D[R - 1]);
          if (lane == 0) {
            if (kLoneRead) cl = *now;
            up_m = cl.m; up_i = cl.i; up_d = cl.d;
          }
          F::load_emission(table, lane, cx, cy, e);
          F::cells(e, up_m, up_i, up_d, dg_m, dg_i, dg_d, M, I, D, pr, t_last);
          st_cell(store, &dst[s].m, M[R - 1]);
          st_cell(store, &dst[s].i, I[R - 1]);
          st_cell(store, &dst[s].d, D[R - 1]);
        }
        (void)t_last;
        acc = P::add(acc, I[R - 1]);
      };

      const int nchunks = (nsteps + kWarp - 1) / kWarp;
      for (int k = 0; k < nchunks; ++k) {
        if ((k & (kStopChunks - 1)) == 0 && stopped(ctl, warp)) {
          alive = false;
          break;
        }
        if (from_ring) {
          cp_async_wait_all();  // this chunk's cells
          __syncwarp();
          if (!fetch_chunk(k + 1)) {
            alive = false;
            break;
          }
        }
        const Cell* rc = ring + (k & 1) * kWarp;
        cell_next = rc[0];
        const int s0 = k * kWarp;
        const int cnt = nsteps - s0 < kWarp ? nsteps - s0 : kWarp;
        // slot y of a two-haplotype item ends within this chunk
        const bool freeze = P::kSlots == 2 && !F::kSameHap && nfreeze > s0 && nfreeze <= s0 + cnt;
        if (cnt == kWarp && !freeze) {
#pragma unroll 1
          for (int i = 0; i < kWarp; i += kUnroll) {
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
              step(s0 + i + u, rc + i + u, rc + ((i + u + 1) & (kWarp - 1)));
          }
        } else {
#pragma unroll 1
          for (int i = 0; i < cnt; ++i) {
            step(s0 + i, rc + i, rc + ((i + 1) & (kWarp - 1)));
            if (freeze && s0 + i == nfreeze - 1) frozen = P::sy(acc);
          }
        }
        if (store && publish) {
          const int col = s0 + cnt - 1 - kLastCol;  // the last column stored
          if (col >= 1) {
            // (orders this lane's row stores before it)
            st_release_cta(&ctl.prog[out_row], enc(p, (uint32_t)col));
          }
        }
      }
      if (from_ring) {
        cp_async_wait_all();  // the prefetch past the last step lands before the ring is reused
        __syncwarp();
      }
    }
    if (alive) {
      if (ctl.task[warp].last) {
        if (close(c, warp, lane, ctl) && lane == kWarp - 1) {
          if constexpr (kTwo) results_call(b, c, item, acc, frozen);
          else results(b, c, item, acc, frozen);
        }
      } else if constexpr (P::kSlots == 2) {
        __syncwarp();  // lane 31's row stores are visible to the whole warp
        const uint32_t Hs[2] = {sl[0].H, sl[1].H};
        const Cell* out_cells = rows + (size_t)ctl.task[warp].out_row * c.scratch_cols + kPad;
        if (rejects(b, c, out_cells, Hs, L, (p + 1) * (kWarp * R) - 1, lane, item) &&
            close(c, warp, lane, ctl) && lane == 0) {
          F::load_refs(c, item, refs);
          const uint32_t pos = c.rescue_base + 2u * item;  // kLaunchRescueByItem positions
          F::finish(b, c, refs[0], 0.0, (double)kMinAcceptedF, pos);
          if (refs[1].read != kNoPair)
            F::finish(b, c, refs[1], 0.0, (double)kMinAcceptedF, pos + 1);
        }
      }
    }
    release(c, warp, lane, ctl, alive);
  }

  // The results of an item from the sums of its last pass (one lane).
  __device__ static void results(const BatchView& b, const ClassLaunch& c, uint32_t item, V acc,
                                 S frozen) {
    PairRef fr[2];
    F::load_refs(c, item, fr);
    const bool valid_y = P::kSlots == 2 && fr[1].read != kNoPair;
    const uint32_t pos = c.rescue_base + 2u * item;  // kLaunchRescueByItem positions
    // both slots of a same-haplotype item ran exactly their own columns
    const S fy = (P::kSlots == 2 && F::kSameHap) ? P::sy(acc) : frozen;
    double res[2] = {0.0, 0.0};
    double amin[2] = {(double)kMinAcceptedF, (double)kMinAcceptedF};
    if (F::kScaled) {
      res[0] = F::scaled_result(b, c.gaps, fr[0].read, P::sx(acc), &amin[0]);
      if (valid_y) res[1] = F::scaled_result(b, c.gaps, fr[1].read, fy, &amin[1]);
    } else {
      // the pass-through row holds M_L + I_L in its I (non-uniform form)
      res[0] = P::sx(acc);
      res[1] = fy;
    }
    F::finish(b, c, fr[0], res[0], amin[0], pos);
    if (valid_y) F::finish(b, c, fr[1], res[1], amin[1], pos + 1);
  }
  // Out of line for the scaled form, whose sweep is 2% faster without this code
  // beside it (20 pairs of 1,000-2,000 bases 1.005 -> 0.98 ms in FP64, 0.571 ->
  // 0.553 in FP32; the three-value form's FP32 sweep is 2 to 6% slower so).
  __device__ __noinline__ static void results_call(const BatchView& b, const ClassLaunch& c,
                                                   uint32_t item, V acc, S frozen) {
    results(b, c, item, acc, frozen);
  }
};

// c.scratch holds kRows boundary rows of c.scratch_cols cells for every block of
// the grid.
template <class P, int R, int GAPS, bool SAME, int MINB, int W>
__global__ void __launch_bounds__(W * kWarp, MINB)
    forward_pipe_kernel(BatchView b, ClassLaunch c) {
  using F = PipeForward<P, R, GAPS, SAME, MINB, W>;
  extern __shared__ uint4 smem[];
  __shared__ typename F::Ctl ctl;
  const int lane = threadIdx.x & (kWarp - 1);
  const int warp = threadIdx.x / kWarp;
  uint4* table = smem + warp * (F::kSmemPerWarp / 16);
  typename F::Cell* rows = reinterpret_cast<typename F::Cell*>(c.scratch) +
                           (size_t)blockIdx.x * F::kRows * c.scratch_cols;
  const uint32_t n = c.work_count ? *c.work_count : c.static_count;
  const uint32_t max_open = (n + gridDim.x - 1) / gridDim.x;
  if (threadIdx.x == 0) {
    ctl.ticket = ctl.serving = ctl.broken = ctl.fail = 0u;
    ctl.started = ctl.scanning = ctl.exhausted = ctl.num_open = 0u;
    ctl.free_rows = (1u << F::kRows) - 1u;
    for (int w = 0; w < W; ++w) {
      ctl.stop[w] = 0u;
      ctl.task[w].slot = W;
      ctl.open[w].state = F::kFree;
    }
  }
  __syncthreads();
  while (F::acquire(b, c, n, max_open, warp, lane, ctl)) F::run(b, c, warp, lane, table, ctl, rows);
}

}  // namespace rodv
