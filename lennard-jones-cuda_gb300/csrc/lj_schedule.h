// lj_schedule.h -- stream-K work split of the all-pairs loop (host side).
//
// The (i-block, j-chunk) pairs of every box are laid out in one sequence
// (box-major, then i-block, then j) and cut into G contiguous ranges of
// equal cost, one per persistent CTA.  Cuts fall on j-chunks of `grain`
// records, not only on whole j-tiles: the persistent grid holds every CTA at
// once, the hardware spreads consecutive CTAs over the SMs, and whole-tile
// ranges (some CTAs one tile more than others) leave SMs with up to one tile
// per resident CTA more work than others.  A CTA emits one partial segment
// per i-block it touches; the integrator sums each block's segments in CTA
// order.
#pragma once

#include <vector>

#include "lj_internal.h"

namespace ljgb {

struct Schedule {
  int G = 0;         // CTAs (persistent grid)
  int BI = 0;        // i-block length (= CTA threads of the pair kernel)
  int TILE = 0;      // j-tile length
  int ntiles = 0;    // total tiles
  int nseg = 0;      // partial segments
  std::vector<BlockInfo> blocks;
  int grain = 0;     // j records per work chunk (cut granularity)
  std::vector<int> cta_tile_begin;  // G + 1: flattened tile holding each CTA's first j
  std::vector<int> cta_lo;          // G + 1: offset of that j within its tile (entry G: 0)
  std::vector<int> cta_block;       // G
  std::vector<int> cta_jt;          // G
  std::vector<int> sys_block_first; // nsys + 1
};

// Builds the schedule for boxes of sizes n[0..nsys).  `tile_overhead` is the
// fixed cost of a tile in units of one j-record (barrier, compensation).
// CTA g covers j from (cta_tile_begin[g], cta_lo[g]) up to, not including,
// (cta_tile_begin[g+1], cta_lo[g+1]): cta_tile_begin[g+1] - cta_tile_begin[g]
// tiles, plus the head of tile cta_tile_begin[g+1] when cta_lo[g+1] > 0.
// Returns false on invalid input (n < 1, BI/TILE < 1, G < 1, TILE not a
// multiple of grain).
constexpr int kSplitGrain = 32;
bool build_schedule(const int* n, int nsys, int BI, int TILE, int G, int tile_overhead, Schedule* out,
                    int grain = kSplitGrain);

// Work split of the pair histogram of one box: i-blocks of kRdfBlock particles,
// each against the j's from the block's own first particle on, in chunks of
// kRdfChunk (pairs j <= i inside the block's own square are skipped by the
// kernel), cut into G contiguous ranges of equal chunk counts.
constexpr int kRdfBlock = 256;
constexpr int kRdfChunk = 32;
struct RdfRanges {
  int G = 0;
  std::vector<int> cta_block, cta_chunk, cta_units;  // G each
};
bool build_rdf_ranges(int n, int ctas, RdfRanges* out);

// Squares and tasks of the FP64 pair pass for boxes of sizes n (Pair64Task).
// The square side grows while there are still about 80 tasks an SM: a tile
// then has at most ~256 slots, so the sums stay at 10 KB a particle whatever
// N is.  Squares of one tile are split into 2 or 4 tasks where that takes 2% off
// the SM with the most work, at `turn_ops` FP64 instructions a turn and
// `slot_ops` for adding one more slot of a tile: N = 200 gives 28 squares for 152
// SMs or 98 quarters, N = 1000 528 squares, 4 on some SMs, or 1024 halves, 7 at
// most.  us for 20 steps, whole -> split: FP64 EVN N = 200 480 -> 358, N = 600
// 648 -> 608, N = 1250 1343 -> 1271; adjoint N = 200 1045 -> 656, N = 600 1680
// -> 1349, N = 1000 2788 -> 2636.  With fewer than 8 tasks an SM the turns of a
// task are shared by 2, 4 or 8 warps, two turns each at least: N = 512 gives 136
// tasks.
struct Pair64Plan {
  int group = 1, parts = 1, split = 1;
  long long slots = 0;
  std::vector<Pair64Task> tasks;
  std::vector<Pair64Box> boxes;
};
// `group` > 1: at least that side, for sums that have to take less memory.
Pair64Plan plan_pairs64(const std::vector<int>& n, int sms, int turn_ops = 28, int slot_ops = 5, int group = 1);
// The plan of the smallest side for which take(plan) has cudaSuccess, given that
// only a lack of memory is worth another try; a plan whose sums (`values` a
// particle and slot) would leave less memory free than they take is not tried
// while a larger side is left.
template <typename Take>
cudaError_t plan_pairs64_within(const std::vector<int>& n, int sms, int turn_ops, int slot_ops, int values,
                                Pair64Plan* p, Take take) {
  for (int group = 1;; group = 2 * p->group) {
    *p = plan_pairs64(n, sms, turn_ops, slot_ops, group);
    bool last = true;
    for (const Pair64Box& b : p->boxes) last &= b.groups == 1;
    if (!last && !leaves_room(sizeof(double) * 32 * values * (size_t)p->slots)) continue;
    const cudaError_t e = take(*p);
    if (e != cudaErrorMemoryAllocation || last) return e;
  }
}

// Tasks of the unordered-pair kernel for n particles and `warps` warps: equal
// shares (+-1) of the (block, tile) sequence.  The i sums of (task, block) are
// part task + block, so a block's parts are consecutive: block_part holds the
// first and the count.
struct NewtonPlan {
  std::vector<NewtonTask> tasks;
  std::vector<int> block_part;
  long long jparts = 0;  // parts of the j sums
  int iparts = 0;
  size_t bytes() const { return sizeof(float) * 5 * (32 * (size_t)jparts + kNewtonBlock * (size_t)iparts); }
};
NewtonPlan plan_newton(int n, int warps);

}  // namespace ljgb
