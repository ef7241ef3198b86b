// lj_rdf.cu -- pair histograms (RDF) of one box.
//
// Replaces the per-pair global atomics and RDFmerger of the reference
// (src/library/MDSystem.cu:36-42, 140-153) and the bin counting of its CPU
// loop (src/library/MDSystem.cpp:281-285).  Counts are those of all ordered
// pairs j != i, as the reference's.
#include <cuda_runtime.h>

#include <cstdint>

#include "lj_device.cuh"
#include "lj_kernels.h"
#include "lj_schedule.h"
#include "lj_stepdev.cuh"

namespace ljgb {
namespace {

// floor(x) for 0 <= x < 2^23: 2^23 + x rounded down is 2^23 + floor(x)
// exactly, read back from the float's bits (an FP32 add and an integer
// subtract instead of a round and a float -> int conversion).
__device__ __forceinline__ int floor_small(float x) {
  return __float_as_int(__fadd_rd(x, 8388608.0f)) - 0x4B000000;
}

constexpr int kTile = 256;  // j records staged in shared memory

// Bin position of a squared fixed-point separation x, before floor, in the
// separately rounded products that the oracle's emu_rdf_* repeats on the CPU:
// r^2 bins (modes 0, 1) x k2 inv_w; linear bins (mode 2) only x k2, compared
// with rmax^2 before the root.
template <int MODE>
__device__ __forceinline__ float bin_pos(float x, float k2, float inv_w) {
  const float r2 = __fmul_rn(x, k2);
  return MODE == 2 ? r2 : __fmul_rn(r2, inv_w);
}

// Smallest x >= 0 whose bin position reaches `limit`, by bisection on the
// bits: rounded products by positive constants are monotonic in x, so `x <
// bound` decides as comparing the position itself would, without forming it.
// 0, so that no pair lies below it, where a factor is infinite (widths below
// 2^-128, say): separation 0 then has no position, and the others are past every
// bin.
template <int MODE>
__device__ float bin_bound(float k2, float inv_w, float limit) {
  if (bin_pos<MODE>(0.0f, k2, inv_w) != 0.0f) return 0.0f;
  int lo = 0, hi = 0x7f800000;
  auto reaches = [&](int bits) { return bin_pos<MODE>(__int_as_float(bits), k2, inv_w) >= limit; };
  // the real quotient is a few ulps away from it, unless a product over- or
  // underflows: a few tests instead of 31, which every CTA would wait for
  // (N = 16384, 256 linear bins: 121 us a call without, 113 with)
  const int near = __float_as_int(MODE == 2 ? limit / k2 : limit / inv_w / k2);
  if (near > 64 && near < 0x7f000000) {
    if (reaches(near + 16)) hi = near + 16;
    if (!reaches(near - 16)) lo = near - 16;
  }
  while (lo < hi) {
    const int mid = lo + (hi - lo) / 2;
    if (reaches(mid)) hi = mid;
    else lo = mid + 1;
  }
  return __int_as_float(lo);
}

// One pair into the CTA's histogram, from its fixed-point separation (qi in
// slots 1..3, see i_record_slots123).  Pairs at or past the bound are not
// counted here: dropped (modes 1, 2), or the last bin's (mode 0), which gets
// all pairs less the counted ones at the end.
template <int MODE>
__device__ __forceinline__ void bin_pair(const int4 qi, const int4 qj, float bound, float k2, float inv_w, int last,
                                         unsigned* shist) {
  const float dx = __int2float_rn(fixed_diff(qj.x, qi.y));
  const float dy = __int2float_rn(fixed_diff(qj.y, qi.z));
  const float dz = __int2float_rn(fixed_diff(qj.z, qi.w));
  const float x = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
  if (x < bound) {
    const float b = bin_pos<MODE>(x, k2, inv_w);
    atomicAdd(&shist[MODE == 2 ? min(floor_small(__fmul_rn(__fsqrt_rn(b), inv_w)), last) : floor_small(b)], 1u);
  }
}

// The pass's end: its last CTA hands counts and status words to the host.
__device__ __forceinline__ void mail_counts(const RdfPass& a, int* flag) {
  const int tid = threadIdx.x;
  __threadfence();
  __syncthreads();
  if (tid == 0) *flag = atomicAdd(a.mail.grid_ticket, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!*flag) return;
  __threadfence();
  for (int b = tid; b < a.hist.nb; b += kRdfBlock) a.counts_out[b] = __ldcg(a.hist.counts + b);
  if (tid == 0) {
    *a.mail.grid_ticket = 0;
    mail_status(a.mail);
  }
  __threadfence_system();
  __syncthreads();
  if (tid == 0) *(volatile int*)(a.mail.words_out + 2) = a.mail.seq;
}

// Each unordered pair once: block b of 256 i's (one per thread) runs over the
// j's from its own first particle on and skips j <= i inside its own square;
// the wrapping difference is antisymmetric, so (j, i) falls into the bin of
// (i, j) exactly and the flush adds every count twice.  The loop is bound by
// issue (no memory traffic: the shadow stays in L2): 11 instructions for a pair
// past the bound, which most are.  N = 16384, 256 clamped bins, us a call: 234
// over ordered pairs, 131 over unordered ones, 119 with the bound in place of
// the products and a counter, 113 with bin_bound's bracket.  A CTA owns a
// contiguous range of (block, 32-j chunk) units (build_rdf_ranges), flushing its
// shared histogram once: a grid of single tiles would flush 256 bins thousands
// of times.
// MAIL: the last CTA hands the counts to the host (rdf_counts of 500 particles
// 42 -> 30 us, of 16384 113 -> 102, against two copies behind the pass).
template <int MODE, bool MAIL>
__global__ void __launch_bounds__(kRdfBlock, 6) k_rdf(RdfPass a) {
  extern __shared__ unsigned shist[];
  __shared__ int4 tile[kTile];
  __shared__ int4 sirec[kRdfBlock];
  const int tid = threadIdx.x, lane = tid & 31;
  const HistArgs h = a.hist;
  const int last = h.nb - 1;
  for (int b = tid; b < h.nb; b += kRdfBlock) shist[b] = 0u;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const float k2 = a.sc->k2;
  const float bound = bin_bound<MODE>(k2, h.inv_w, MODE == 2 ? h.rmax2 : (float)(MODE == 1 ? h.nb : last));
  unsigned npairs = 0;  // of this thread's i, since the last flush
  auto flush = [&]() {
    __syncthreads();
    unsigned counted = 0;
    for (int b = tid; b < h.nb; b += kRdfBlock)
      if (shist[b]) {
        counted += shist[b];
        atomicAdd(h.counts + b, 2ull * shist[b]);
      }
    if (MODE == 0) {
      // (sums of a CTA stay below 2^32; the difference may be negative for a warp)
      const unsigned all = __reduce_add_sync(0xffffffffu, npairs), binned = __reduce_add_sync(0xffffffffu, counted);
      if (lane == 0) atomicAdd(h.counts + last, 2ull * all - 2ull * binned);
    }
    npairs = 0;
  };
  int B = a.cta_block[blockIdx.x], c = a.cta_chunk[blockIdx.x], left = a.cta_units[blockIdx.x];
  const int nchunks = (a.n + kRdfChunk - 1) / kRdfChunk;
  int counted = 0;  // units since the last flush
  for (; left > 0; ++B, c = 0) {
    const int i0 = B * kRdfBlock, i = i0 + tid;
    const int4 qi = i_record_slots123(a.q[min(i, a.n - 1)], &sirec[tid]);
    int take = min(left, nchunks - B * (kRdfBlock / kRdfChunk) - c);
    left -= take;
    // 2^19 units are 2^32 pairs, what a 32-bit bin can hold
    for (; take > 0;) {
      const int part = min(take, (1 << 18));
      if (counted + part > (1 << 18)) {
        flush();
        __syncthreads();
        for (int b = tid; b < h.nb; b += kRdfBlock) shist[b] = 0u;
        counted = 0;
      }
      counted += part;
      const int j1 = min(a.n, i0 + (c + part) * kRdfChunk);
      for (int j0 = i0 + c * kRdfChunk; j0 < j1; j0 += kTile) {
        const int cnt = min(kTile, j1 - j0);
        __syncthreads();
        if (tid < cnt) tile[tid] = a.q[j0 + tid];
        __syncthreads();
        if (i >= a.n) continue;
        if (j0 >= i0 + kRdfBlock) {
#pragma unroll 8
          for (int jj = 0; jj < cnt; ++jj) bin_pair<MODE>(qi, tile[jj], bound, k2, h.inv_w, last, shist);
          npairs += cnt;
        } else {
          for (int jj = 0; jj < cnt; ++jj)
            if (j0 + jj > i) bin_pair<MODE>(qi, tile[jj], bound, k2, h.inv_w, last, shist);
          npairs += max(0, j0 + cnt - max(j0, i + 1));
        }
      }
      take -= part;
      c += part;
    }
  }
  flush();
  if (MAIL) mail_counts(a, &sirec[0].x);
}

// ---------------------------------------------------------------------------
// Short-ranged histograms of large boxes: the particles are sorted into cells
// of 1/16 of the frame in Morton order, so 32 consecutive ones (a tile) lie
// together, and pairs of tiles that are too far apart are left out.  The test
// is exact: the gap of two tiles' bounds, circular as the wrapping difference
// is, goes through the pairs' own roundings, which are monotonic.
// ---------------------------------------------------------------------------
constexpr int kCells = kRdfCells;

// shift: 28 where the frame is the whole 32-bit circle (periodic), 27 where
// the positions lie in its lower half.
__device__ __forceinline__ int cell_of(const int4 q, int shift) {
  auto spread = [](unsigned c) { return (c & 1u) | (c & 2u) << 2 | (c & 4u) << 4 | (c & 8u) << 6; };
  return (int)(spread((unsigned)q.x >> shift & 15u) | spread((unsigned)q.y >> shift & 15u) << 1 |
               spread((unsigned)q.z >> shift & 15u) << 2);
}

__global__ void __launch_bounds__(kRdfBlock) k_rdf_cells(const int4* q, int n, int shift, RdfNear s) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int i = blockIdx.x * kRdfBlock + threadIdx.x;
  if (i < n) s.rank[i] = atomicAdd(&s.cells[cell_of(q[i], shift)], 1);
}

// Every CTA forms the cells' first places itself (a launch less).
__global__ void __launch_bounds__(kRdfBlock) k_rdf_scatter(const int4* q, int n, int shift, RdfNear s) {
  __shared__ int first[kCells];
  __shared__ int wsum[kRdfBlock / 32];
  constexpr int kPer = kCells / kRdfBlock;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int c[kPer], sum = 0;
#pragma unroll
  for (int k = 0; k < kPer; k += 4) {
    const int4 v = *reinterpret_cast<const int4*>(s.cells + tid * kPer + k);
    c[k] = v.x;
    c[k + 1] = v.y;
    c[k + 2] = v.z;
    c[k + 3] = v.w;
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) sum += c[k];
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  int at = incl - sum;
  for (int k = 0; k < w; ++k) at += wsum[k];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    first[tid * kPer + k] = at;
    at += c[k];
  }
  __syncthreads();
  const int i = blockIdx.x * kRdfBlock + tid;
  if (i >= n) return;
  const int4 r = q[i];
  s.sorted[first[cell_of(r, shift)] + s.rank[i]] = r;
}

// Bounds of each tile: a warp a tile.
__global__ void __launch_bounds__(kRdfBlock) k_rdf_boxes(int n, RdfNear s) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int t = (blockIdx.x * kRdfBlock + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t * 32 >= n) return;
  const int4 r = s.sorted[min(t * 32 + lane, n - 1)];
  const unsigned v[3] = {(unsigned)r.x, (unsigned)r.y, (unsigned)r.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const uint2 b = make_uint2(__reduce_min_sync(0xffffffffu, v[c]), __reduce_max_sync(0xffffffffu, v[c]));
    if (lane == 0) s.box[t * 3 + c] = b;
  }
}

// Least circular distance of two intervals.
__device__ __forceinline__ unsigned gap(uint2 a, uint2 b) {
  const unsigned lo = max(a.x, b.x), hi = min(a.y, b.y);
  if (lo <= hi) return 0u;
  return min(lo - hi, 0u - (max(a.y, b.y) - min(a.x, b.x)));
}

// A unit is a tile of i's (one a lane) against a group of 8 tiles of j's, from
// its own tile on; units go round the warps of the grid.  Bound by issue as
// k_rdf where the reach is long, by the tiles' loads where it is short.
template <int MODE, bool MAIL>
__global__ void __launch_bounds__(kRdfBlock, 6) k_rdf_near(RdfPass a, RdfNear s) {
  extern __shared__ unsigned shist[];
  __shared__ int4 tile[kRdfBlock / 32][32];
  __shared__ int4 sirec[kRdfBlock];
  constexpr int kGroup = 8;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const HistArgs h = a.hist;
  const int last = h.nb - 1;
  for (int b = tid; b < h.nb; b += kRdfBlock) shist[b] = 0u;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const float k2 = a.sc->k2;
  const float bound = bin_bound<MODE>(k2, h.inv_w, MODE == 2 ? h.rmax2 : (float)(MODE == 1 ? h.nb : last));
  __syncthreads();
  const int tiles = (a.n + 31) / 32, groups = (tiles + kGroup - 1) / kGroup;
  for (long long u = (long long)w * gridDim.x + blockIdx.x; u < (long long)tiles * groups;
       u += (long long)gridDim.x * (kRdfBlock / 32)) {
    const int I = (int)(u / groups), g = (int)(u - (long long)I * groups);
    if ((g + 1) * kGroup <= I) continue;
    const int mine = g * kGroup + lane;
    bool near = false;
    if (lane < kGroup && mine >= I && mine < tiles) {
      const float gx = __uint2float_rn(gap(s.box[I * 3], s.box[mine * 3]));
      const float gy = __uint2float_rn(gap(s.box[I * 3 + 1], s.box[mine * 3 + 1]));
      const float gz = __uint2float_rn(gap(s.box[I * 3 + 2], s.box[mine * 3 + 2]));
      near = __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, __fmul_rn(gx, gx))) < bound;
    }
    unsigned todo = __ballot_sync(0xffffffffu, near);
    if (!todo) continue;
    const int i = I * 32 + lane;
    const int4 qi = i_record_slots123(s.sorted[min(i, a.n - 1)], &sirec[tid]);
    for (; todo; todo &= todo - 1) {
      const int J = g * kGroup + __ffs(todo) - 1, cnt = min(32, a.n - J * 32);
      __syncwarp();
      tile[w][lane] = s.sorted[min(J * 32 + lane, a.n - 1)];
      __syncwarp();
      if (i >= a.n) continue;
      if (J > I && cnt == 32) {
#pragma unroll 8
        for (int jj = 0; jj < 32; ++jj) bin_pair<MODE>(qi, tile[w][jj], bound, k2, h.inv_w, last, shist);
      } else {
        for (int jj = 0; jj < cnt; ++jj)
          if (J > I || jj > lane) bin_pair<MODE>(qi, tile[w][jj], bound, k2, h.inv_w, last, shist);
      }
    }
  }
  __syncthreads();
  unsigned counted = 0;
  for (int b = tid; b < h.nb; b += kRdfBlock)
    if (shist[b]) {
      counted += shist[b];
      atomicAdd(h.counts + b, 2ull * shist[b]);
    }
  if (MODE == 0) {  // the last bin's are all pairs less the counted ones
    const unsigned binned = __reduce_add_sync(0xffffffffu, counted);
    if (lane == 0 && binned) atomicAdd(h.counts + last, 0ull - 2ull * binned);
    if (tid == 0 && blockIdx.x == 0) atomicAdd(h.counts + last, (unsigned long long)a.n * (a.n - 1));
  }
  if (MAIL) mail_counts(a, &sirec[0].x);
}

}  // namespace

// 6 CTAs of 256 threads an SM at 40 registers; their shared memory (4 + 4 KB
// and at most 16 KB of bins each) fits beside each other for any bin count.
int rdf_ctas_per_sm() { return 6; }

cudaError_t launch_rdf(const RdfPass& a, int grid, cudaStream_t st) {
  const size_t smem = sizeof(unsigned) * (size_t)a.hist.nb;
  const bool mail = a.mail.seq != 0;
  auto* k = a.hist.mode == 0   ? (mail ? k_rdf<0, true> : k_rdf<0, false>)
            : a.hist.mode == 1 ? (mail ? k_rdf<1, true> : k_rdf<1, false>)
                               : (mail ? k_rdf<2, true> : k_rdf<2, false>);
  return launch_dependent(k, grid, kRdfBlock, smem, st, a);
}

cudaError_t launch_rdf_near(const RdfPass& a, const RdfNear& s, bool periodic, int grid, cudaStream_t st) {
  const int shift = periodic ? 28 : 27, nb = (a.n + kRdfBlock - 1) / kRdfBlock;
  cudaError_t e = launch_dependent(k_rdf_cells, nb, kRdfBlock, 0, st, a.q, a.n, shift, s);
  if (e == cudaSuccess) e = launch_dependent(k_rdf_scatter, nb, kRdfBlock, 0, st, a.q, a.n, shift, s);
  if (e == cudaSuccess) e = launch_dependent(k_rdf_boxes, nb, kRdfBlock, 0, st, a.n, s);
  if (e != cudaSuccess) return e;
  // (a pass that leaves its counts on the device is calculateNForces', mode 0)
  auto* k = a.mail.seq == 0     ? k_rdf_near<0, false>
            : a.hist.mode == 0 ? k_rdf_near<0, true>
            : a.hist.mode == 1 ? k_rdf_near<1, true>
                               : k_rdf_near<2, true>;
  if (a.mail.seq == 0 && a.hist.mode != 0) return cudaErrorInvalidValue;
  return launch_dependent(k, grid, kRdfBlock, sizeof(unsigned) * (size_t)a.hist.nb, st, a, s);
}

}  // namespace ljgb
