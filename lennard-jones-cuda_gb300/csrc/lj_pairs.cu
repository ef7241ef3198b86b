// lj_pairs.cu -- all-pairs Lennard-Jones force / energy / virial kernels.
//
// Replaces calculateForces + RDFmerger of the reference
// (src/library/MDSystem.cu:21-153) and the O(N^2) CPU loop of
// MDSystem::CalculateForces (src/library/MDSystem.cpp:253-310).  Same pair set
// (ordered pairs j != i, minimum image for periodic boxes, no cutoff), same
// physics (MDSystem.cu:44-53), redesigned for sm_103a:
//
//  * persistent stream-K grid: every CTA receives an equal share of the
//    (i-block, j-tile) sequence of all boxes, so the single wave fills all
//    SMs regardless of N (the reference launches ceil(N/256) CTAs);
//  * j-tiles of 16-byte records staged in shared memory by cp.async.bulk
//    (TMA bulk copies) into a STAGES-deep mbarrier ring, read back as
//    broadcast 128-bit shared loads;
//  * MIXED precision: positions as 32-bit fixed-point fractions of the box
//    whose wrapping integer difference is the minimum image (no rounding
//    instructions per pair), FP32 pair math, per-tile FP32 sums folded into
//    TwoSum-compensated accumulators;
//  * no per-pair global atomics: partial sums of each (CTA, i-block) segment
//    go to a partial buffer reduced deterministically in FP64 by the
//    integrator kernels (pair histograms are lj_rdf.cu's).
#include <cuda_runtime.h>

#include <cstdint>

#include "lj_device.cuh"
#include "lj_kernels.h"
#include "lj_mixed.cuh"
#include "lj_schedule.h"
#include "lj_stepdev.cuh"

namespace ljgb {

namespace {

#ifndef LJ_CHUNK
#define LJ_CHUNK 32
#endif
constexpr int kChunk = LJ_CHUNK;  // pairs per compensated force partial sum
// CTA ranges start and end on multiples of kSplitGrain j records inside a
// tile; the unrolled chunk loop needs those to be whole chunks.
static_assert(kSplitGrain % kChunk == 0, "schedule cuts must fall on chunk boundaries");

}  // namespace

// ---------------------------------------------------------------------------
// MIXED-precision persistent pair kernel.
// THREADS threads, one i-particle each; TILE j-records per stage.
// ---------------------------------------------------------------------------
// EPI = 0: partial segments only.  EPI = MODE_EVN / MODE_TVN: the CTA that
// writes the last segment of an i-block also runs the second half of the
// Verlet step for that block (fused_block_step), and the CTA that finishes
// the last block runs the per-box observables (EVN) or the TVN scale (TVN).
// Completion is detected with atomic counters only; no CTA waits on another.
template <int THREADS, int TILE, int STAGES, int EPI>
__device__ __forceinline__ void pairs_body(const PairArgs& a, const StateArgs& st, unsigned char* smem_raw) {
  int4* sq = reinterpret_cast<int4*>(smem_raw);
  __shared__ uint64_t bars[STAGES];
  __shared__ double shd[EPI ? 4 * 32 : 1];
  __shared__ int sflag;
  __shared__ int4 sirec[THREADS];  // i records on their way to slots 1..3

  const int g = blockIdx.x;
  const int tid = threadIdx.x;
  if (EPI && g == 0) {
    if (tid == 0) st.glob_cnt[st.ticket ^ 1] = 0;  // the other parity's ticket counter
    if (EPI == MODE_EVN) {
      // This step's observables are pending once the launch completes: its
      // parity's entry is read only after that (the next step's pair kernel,
      // a read-back), and this launch reads only the other parity's.
      const int par = st.ticket - 2;
      for (int sys = tid; sys < st.nsys; sys += THREADS) {
        st.sc[sys].obs_slot[par] = st.obs_slot;
        st.sc[sys].obs_nblk[par] = 0;
        st.sc[sys].obs_pending[par] = MODE_EVN;
      }
    }
  }
  // This CTA's j range: from offset lo0 of its first tile to offset lo1 of
  // tile t1 (lo1 = 0: up to the end of tile t1 - 1).
  const int t0 = a.cta_tile_begin[g], t1 = a.cta_tile_begin[g + 1];
  const int lo0 = a.cta_lo ? a.cta_lo[g] : 0, lo1 = a.cta_lo ? a.cta_lo[g + 1] : 0;
  const int ntiles = t1 - t0 + (lo1 > 0 ? 1 : 0);
  if (ntiles <= 0) return;

  // Barrier-free j-tile pipeline: warps wait only for the data of the stage
  // they read (its mbarrier) and count themselves done with it in shared
  // memory; the last warp to finish a stage refills it with the tile STAGES
  // ahead (its lane 0 issues the bulk copy).  Warps therefore drift freely by
  // up to STAGES-1 tiles instead of meeting at a CTA barrier every tile.
  constexpr int NW = THREADS / 32;
  __shared__ int done_cnt[STAGES];
  __shared__ int prod[3];  // producer cursor: i-block, j-tile, tiles issued
  __shared__ volatile int sfail;
  const int lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars[s], 1);
      done_cnt[s] = 0;
    }
    sfail = 0;
    fence_mbar_init();
  }
  __syncthreads();
  if (tid == 0) {
    int pB = a.cta_block[g], pjt = a.cta_jt[g], issued = 0;
    const int pre = ntiles < STAGES ? ntiles : STAGES;
    for (; issued < pre; ++issued) {
      const BlockInfo bi = a.blocks[pB];
      const int j0 = pjt * TILE;
      const int cnt = min(TILE, bi.n_sys - j0);
      const int s = issued % STAGES;
      mbar_arrive_expect_tx(&bars[s], (uint32_t)cnt * 16u);
      bulk_g2s(sq + s * TILE, a.q + bi.p0 + j0, (uint32_t)cnt * 16u, &bars[s]);
      if (++pjt == bi.njt) { ++pB; pjt = 0; }
    }
    prod[0] = pB;
    prod[1] = pjt;
    prod[2] = issued;
  }
  __syncthreads();

  int B = a.cta_block[g], jt = a.cta_jt[g];
  BlockInfo bi = a.blocks[B];
  int i_local = bi.i0 + tid;
  bool valid_i = tid < bi.n_i;
  int4 qi = i_record_slots123(a.q[bi.p0 + (valid_i ? i_local : bi.i0)], &sirec[tid]);
  float k2inv = a.sc[bi.sys].k2inv;
  FloatAcc acc[5];
#pragma unroll
  for (int c = 0; c < 5; ++c) acc[c] = FloatAcc{0.f, 0.f};

  // A warp whose wait times out (or that sees another warp's timeout) keeps
  // walking the tile sequence without computing, so every CTA-wide barrier
  // below is still reached by all warps; results of the launch are void.
  bool failed = false;
  for (int k = 0; k < ntiles; ++k) {
    const int s = k % STAGES;
    if (!failed) {
      const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bars[s], (uint32_t)((k / STAGES) & 1)));
      if (!ok) {
        failed = true;
        if (lane == 0) sfail = 1;
      } else if (sfail) {
        failed = true;
      }
    }
    const int j0 = jt * TILE;
    const int cnt = min(TILE, bi.n_sys - j0);
    const int jlo = k == 0 ? lo0 : 0;                        // multiples of kChunk
    const int jhi = (k == ntiles - 1 && lo1 > 0) ? lo1 : cnt;
    if (!failed) {
      const int4* st = sq + s * TILE;
      const bool masked = j0 < bi.i0 + bi.n_i && j0 + cnt > bi.i0;  // tile holds this block's own i's
      // Force sums are folded into the TwoSum accumulators every kChunk
      // pairs, so a large near-neighbour term rounds at most kChunk-1 later
      // additions.  Energy sums go chunk -> tile (plain FP32) -> TwoSum: a
      // chunk partial is never small next to the tile sum, so the far-field
      // (s/r)^6 tail is not truncated.
      float ta = 0.f, tb = 0.f;
      if (cnt == TILE) {
        // Full tile: unrolled chunks.  Only the diagonal tile (the j-range
        // holding this CTA's own i's) needs the self-pair excluded; it
        // keeps the unrolled loop and pays one compare + select per pair.
        const bool diag = masked;
#pragma unroll 1
        for (int c0 = jlo; c0 < jhi; c0 += kChunk) {
          const f32x2 k2i2 = pk2(k2inv, k2inv);
          f32x2 FX = 0ull, FY = 0ull, FZ = 0ull, PA = 0ull, PB = 0ull;
          if (!diag) {
#pragma unroll
            for (int jj = c0; jj < c0 + kChunk; jj += 2)
              pair_mixed2<false>(qi, st[jj], st[jj + 1], k2i2, false, false, FX, FY, FZ, PA, PB);
          } else {
            const int self = i_local - j0;  // tile-local index of this thread's i
#pragma unroll
            for (int jj = c0; jj < c0 + kChunk; jj += 2)
              pair_mixed2<true>(qi, st[jj], st[jj + 1], k2i2, jj == self, jj + 1 == self, FX, FY, FZ, PA, PB);
          }
          const float fx = lane_sum(FX), fy = lane_sum(FY), fz = lane_sum(FZ), pa = lane_sum(PA),
                      pb = lane_sum(PB);
          two_sum_add(acc[0], fx);
          two_sum_add(acc[1], fy);
          two_sum_add(acc[2], fz);
          ta += pa;
          tb += pb;
        }
      } else {
        // Ragged last tile of a box: packed pairs with the self pair
        // excluded, an odd last record on its own.
        const int self = i_local - j0;
        for (int c0 = jlo; c0 < jhi; c0 += kChunk) {
          const int c1 = min(jhi, c0 + kChunk);
          const f32x2 k2i2 = pk2(k2inv, k2inv);
          f32x2 FX = 0ull, FY = 0ull, FZ = 0ull, PA = 0ull, PB = 0ull;
          int jj = c0;
          for (; jj + 1 < c1; jj += 2)
            pair_mixed2<true>(qi, st[jj], st[jj + 1], k2i2, jj == self, jj + 1 == self, FX, FY, FZ, PA, PB);
          float fx = lane_sum(FX), fy = lane_sum(FY), fz = lane_sum(FZ), pa = lane_sum(PA), pb = lane_sum(PB);
          if (jj < c1) pair_mixed<true>(qi, st[jj], k2inv, jj == self, fx, fy, fz, pa, pb);
          two_sum_add(acc[0], fx);
          two_sum_add(acc[1], fy);
          two_sum_add(acc[2], fz);
          ta += pa;
          tb += pb;
        }
      }
      two_sum_add(acc[3], ta);
      two_sum_add(acc[4], tb);
    }
    // This warp is done reading stage s; the last warp done refills it.
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      if (atomicAdd(&done_cnt[s], 1) == NW - 1) {
        done_cnt[s] = 0;
        const int issued = prod[2];
        if (issued < ntiles) {
          const int pB = prod[0], pjt = prod[1];
          const BlockInfo pbi = a.blocks[pB];
          const int pj0 = pjt * TILE;
          const int pcnt = min(TILE, pbi.n_sys - pj0);
          mbar_arrive_expect_tx(&bars[s], (uint32_t)pcnt * 16u);
          bulk_g2s(sq + s * TILE, a.q + pbi.p0 + pj0, (uint32_t)pcnt * 16u, &bars[s]);
          const bool wrap = (pjt + 1 == pbi.njt);
          prod[0] = wrap ? pB + 1 : pB;
          prod[1] = wrap ? 0 : pjt + 1;
          prod[2] = issued + 1;
        }
        __threadfence_block();
      }
    }
    const bool last = (k == ntiles - 1);
    const bool block_end = (jt + 1 == bi.njt);
    if (block_end || last) {
      if (valid_i && !failed) {
        const int seg = bi.seg_first + (g - bi.g_first);
        float* out = a.partial + (size_t)seg * 5 * THREADS;
#pragma unroll
        for (int c = 0; c < 5; ++c) out[c * THREADS + tid] = acc[c].hi + acc[c].lo;
      }
#pragma unroll
      for (int c = 0; c < 5; ++c) acc[c] = FloatAcc{0.f, 0.f};
      if (EPI) {
        // Last segment of block B?  (fence, then count; the CTA that
        // completes the count owns the block's epilogue)
        __threadfence();
        __syncthreads();
        if (tid == 0) sflag = !sfail && (atomicAdd(st.blk_cnt + B, 1) == bi.seg_count - 1);
        __syncthreads();
        if (sflag) {
          __threadfence();
          fused_block_step<EPI>(st, B, shd);
          __syncthreads();
          // No per-box stage here: TVN's chi is formed by k_tvn_close from
          // the blocks' sums, and EVN's observables were marked pending at
          // the launch's start.
          if (tid == 0) st.blk_cnt[B] = 0;
        }
      }
      if (block_end && !last) {
        ++B;
        bi = a.blocks[B];
        i_local = bi.i0 + tid;
        valid_i = tid < bi.n_i;
        qi = i_record_slots123(a.q[bi.p0 + (valid_i ? i_local : bi.i0)], &sirec[tid]);
        k2inv = a.sc[bi.sys].k2inv;
        jt = 0;
      }
    } else {
      ++jt;
    }
  }

  if (EPI) {
    // This CTA's pair work is done: the first CTAs to get here compute the
    // observables the previous step left pending (one box per ticket), in
    // time the SM would otherwise leave to the CTAs still busy.  The ticket
    // counters alternate by step parity; CTA 0 clears the other one at its
    // start, after the previous step's kernels have completed.
    __shared__ int ticket;
    __syncthreads();
    if (tid == 0) ticket = atomicAdd(st.glob_cnt + st.ticket, 1);
    __syncthreads();
    if (ticket < st.nsys && !sfail) pending_observables(st, ticket, gridDim.x, shd);
    // The dependent kernel of a fused TVN step (k_tvn_close) may be scheduled
    // from here on; it waits for this grid's completion before reading.
    if (EPI == MODE_TVN) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  __syncthreads();
  if (sfail) {
    // Drain the copies still in flight before the CTA's shared memory goes away.
    if (tid == 0) {
      const int issued = prod[2];
      for (int kk = issued - STAGES < 0 ? 0 : issued - STAGES; kk < issued; ++kk)
        mbar_wait_bounded(&bars[kk % STAGES], (uint32_t)((kk / STAGES) & 1));
      atomicOr(a.status, LJ_DEVFLAG_TIMEOUT);
    }
    return;
  }
}

template <int THREADS, int TILE, int STAGES, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) k_pairs_mixed(PairArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  pairs_body<THREADS, TILE, STAGES, 0>(a, StateArgs{}, smem_raw);
}

template <int THREADS, int TILE, int STAGES, int MINB, int EPI>
__global__ void __launch_bounds__(THREADS, MINB) k_pairs_mixed_fused(FusedPairArgs f) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  pairs_body<THREADS, TILE, STAGES, EPI>(f.pair, f.st, smem_raw);
}

// ---------------------------------------------------------------------------
// Shape table and launchers.
// ---------------------------------------------------------------------------
namespace {

template <int THREADS, int TILE, int STAGES, int MINB>
cudaError_t launch_mixed_t(const PairArgs& a, int grid, cudaStream_t st) {
  // <= 48 KB: 16 B x STAGES x TILE staging, no opt-in needed.
  const size_t smem = sizeof(int4) * STAGES * TILE;
  return launch_dependent(k_pairs_mixed<THREADS, TILE, STAGES, MINB>, grid, THREADS, smem, st, a);
}

template <int THREADS, int TILE, int STAGES, int MINB>
cudaError_t launch_fused_t(int mode, const FusedPairArgs& f, int grid, cudaStream_t st) {
  const size_t smem = sizeof(int4) * STAGES * TILE;
  auto* k = mode == MODE_EVN ? k_pairs_mixed_fused<THREADS, TILE, STAGES, MINB, MODE_EVN>
                             : k_pairs_mixed_fused<THREADS, TILE, STAGES, MINB, MODE_TVN>;
  return launch_dependent(k, grid, THREADS, smem, st, f);
}

template <int THREADS, int TILE, int STAGES, int MINB>
cudaError_t occupancy_mixed_t(int* blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      blocks_per_sm, k_pairs_mixed<THREADS, TILE, STAGES, MINB>, THREADS,
      sizeof(int4) * STAGES * TILE);
}

}  // namespace

// Kernel shapes the autotuner chooses among (threads = i-block size; MINB =
// resident CTAs per SM the register allocation must allow).
#define LJ_SHAPES(X)   \
  X(0, 128, 256, 3, 6)  \
  X(1, 128, 512, 3, 6)  \
  X(2, 256, 256, 3, 3)  \
  X(3, 256, 512, 3, 3)  \
  X(4, 384, 512, 3, 2)  \
  X(5, 64, 256, 3, 12)

const PairShape kShapes[] = {
#define LJ_SHAPE_ROW(i, T, TL, S, M) {T, TL, S},
    LJ_SHAPES(LJ_SHAPE_ROW)
#undef LJ_SHAPE_ROW
};
const int kNumShapes = sizeof(kShapes) / sizeof(kShapes[0]);

cudaError_t pair_occupancy(int shape, int* blocks_per_sm) {
  switch (shape) {
#define LJ_OCC_CASE(i, T, TL, S, M) \
  case i:                           \
    return occupancy_mixed_t<T, TL, S, M>(blocks_per_sm);
    LJ_SHAPES(LJ_OCC_CASE)
#undef LJ_OCC_CASE
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_pairs(int shape, const PairArgs& a, int grid, cudaStream_t st) {
  switch (shape) {
#define LJ_LAUNCH_CASE(i, T, TL, S, M) \
  case i:                              \
    return launch_mixed_t<T, TL, S, M>(a, grid, st);
    LJ_SHAPES(LJ_LAUNCH_CASE)
#undef LJ_LAUNCH_CASE
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_pairs_fused(int shape, int mode, const FusedPairArgs& f, int grid, cudaStream_t st) {
  switch (shape) {
#define LJ_FUSED_CASE(i, T, TL, S, M) \
  case i:                             \
    return launch_fused_t<T, TL, S, M>(mode, f, grid, st);
    LJ_SHAPES(LJ_FUSED_CASE)
#undef LJ_FUSED_CASE
  }
  return cudaErrorInvalidValue;
}

}  // namespace ljgb
