// lj_newton.cu -- the MIXED step of one box of 8192 particles or more, every
// unordered pair evaluated once.
//
// The stream-K and row kernels evaluate ordered pairs, as the reference does
// (src/library/MDSystem.cu:74-111), at the rate of the packed pair loop: per
// two pairs 14 FP32x2 operations and as many differences, conversions and
// reciprocals.  Applied to both particles, a pair needs five FP32x2
// operations more and saves the other evaluation.  What it costs is a place
// for the second particle's sums; here they travel:
//   * a warp holds a block of 256 i's, eight a lane in the halves of FP32x2
//     registers, and meets one tile of 32 j's after another;
//   * lane l meets j = l + s in turn s of 32, and the j's five sums move on to
//     lane l - 1 by shuffles, so after 32 turns every i of the block has met
//     every j of the tile, and no sum was reduced across lanes;
//   * the j sums of each (block, tile) and the i sums of each (warp, block)
//     are written once, and k_newton_sum adds a particle's parts in FP32
//     TwoSum and takes the step's second half.
// Arithmetic per pair is that of lj_mixed.cuh, sums are folded into TwoSum
// pairs every 32 pairs of an i, and a j's forces every 32 with each half of the
// i's, its energies every 64.
#include <cuda_runtime.h>

#include <cstdint>

#include "lj_device.cuh"
#include "lj_kernels.h"
#include "lj_mixed.cuh"
#include "lj_stepdev.cuh"

namespace ljgb {
namespace {

constexpr int kWarps = kNewtonWarps;   // tasks are per warp, no barrier
constexpr int kI = 8;                  // i's a lane holds
constexpr int kFold = 8;               // turns between folds of the j sums
static_assert(kNewtonBlock == 32 * kI, "block of a warp");

struct NewtonShared {
  int4 tile[kWarps][2][32];
  f32x2 hi[kWarps][kI / 2][5][32], lo[kWarps][kI / 2][5][32];  // the i's TwoSum pairs
  FloatAcc j[kWarps][5][32];                                   // the tile's j's
};

// One turn for two of the lane's i's (slots 1..3) and its current j.
template <bool MASKED>
__device__ __forceinline__ void pair_both(const int4 qa, const int4 qb, const int4 qj, f32x2 k2inv2, bool exa,
                                          bool exb, f32x2 (&f)[5], f32x2 (&g)[5]) {
  const f32x2 dx = pk2(__int2float_rn(fixed_diff(qa.y, qj.x)), __int2float_rn(fixed_diff(qb.y, qj.x)));
  const f32x2 dy = pk2(__int2float_rn(fixed_diff(qa.z, qj.y)), __int2float_rn(fixed_diff(qb.z, qj.y)));
  const f32x2 dz = pk2(__int2float_rn(fixed_diff(qa.w, qj.z)), __int2float_rn(fixed_diff(qb.w, qj.z)));
  const f32x2 r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
  float r2a, r2b;
  upk2(r2, r2a, r2b);
  float ra = rcp_approx(r2a), rb = rcp_approx(r2b);
  if (MASKED) {
    ra = exa ? 0.0f : ra;
    rb = exb ? 0.0f : rb;
  }
  const f32x2 ri = mul2(pk2(ra, rb), k2inv2);
  const f32x2 r6 = mul2(mul2(ri, ri), ri);
  const f32x2 t = fma2(r6, pk2(12.0f, 12.0f), pk2(-6.0f, -6.0f));
  const f32x2 sf = mul2(mul2(r6, ri), t);
  f[0] = fma2(sf, dx, f[0]);
  f[1] = fma2(sf, dy, f[1]);
  f[2] = fma2(sf, dz, f[2]);
  f[3] = fma2(r6, r6, f[3]);
  f[4] = add2(f[4], r6);
  g[0] = fma2(sf, dx, g[0]);  // the j's force with the i's sign
  g[1] = fma2(sf, dy, g[1]);
  g[2] = fma2(sf, dz, g[2]);
  g[3] = fma2(r6, r6, g[3]);
  g[4] = add2(g[4], r6);
}

__device__ __forceinline__ f32x2 shfl2(f32x2 v, int from) { return __shfl_sync(0xffffffffu, v, from); }

// A tile of j's against the lane's i's; i0: index of the block's first i, j0
// of the tile's first j.  Leaves the i sums of the tile in f, the j sums in J
// (by j).
template <bool MASKED>
__device__ __forceinline__ void newton_tile(const int4 (&q)[kI], const int4* tile, f32x2 k2i2, int i0, int j0, int n,
                                            f32x2 (&f)[kI / 2][5], FloatAcc (*J)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 5; ++k) J[k][lane] = FloatAcc{0.f, 0.f};
  __syncwarp();
#pragma unroll 1
  for (int s0 = 0; s0 < 32; s0 += kFold) {
    f32x2 g[5] = {0ull, 0ull, 0ull, 0ull, 0ull};
#pragma unroll 4
    for (int s = s0; s < s0 + kFold; ++s) {
      const int jl = (lane + s) & 31;
      const int4 qj = tile[jl];
#pragma unroll
      for (int m = 0; m < kI / 2; ++m) {
        bool exa = false, exb = false;
        if (MASKED) {
          const int j = j0 + jl, ia = i0 + 64 * m + lane;
          exa = j <= ia || j >= n;
          exb = j <= ia + 32 || j >= n;
        }
        pair_both<MASKED>(q[2 * m], q[2 * m + 1], qj, k2i2, exa, exb, f[m], g);
      }
#pragma unroll
      for (int k = 0; k < 5; ++k) g[k] = shfl2(g[k], (lane + 1) & 31);
    }
    const int jl = (lane + s0 + kFold) & 31;  // the j whose sums are at this lane now
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      FloatAcc acc = J[k][jl];
      if (k < 3) {  // forces: the halves (32 pairs each) meet exactly too
        FloatAcc both;
        float other;
        upk2(g[k], both.hi, other);
        both.lo = 0.f;
        two_sum_add(both, other);
        two_sum_add(acc, both.hi);
        acc.lo = __fadd_rn(acc.lo, both.lo);
      } else {
        two_sum_add(acc, lane_sum(g[k]));
      }
      J[k][jl] = acc;
    }
    __syncwarp();
  }
}

}  // namespace

// Bound: issue and register reads of the turns (33 instructions of them 19
// FP32x2 a packed evaluation, so per 4 ordered pairs, where the stream-K loop
// spends 28 and 14 per 2).  12 warps an SM at 168 registers: with 16 warps at
// 128 the loop spilled and ran 7% slower; unrolled 4 turns (1: 25% slower, 8:
// 1% faster on the largest boxes and 7% slower at N = 16384).  us a TVN step,
// stream-K -> this kernel and its sums: N = 16384 185 -> 154, N = 65536 2700
// -> 2080, N = 262144 42.9 -> 31.9 ms.
__global__ void __launch_bounds__(32 * kWarps, 3) k_newton(NewtonArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  NewtonShared& sh = *reinterpret_cast<NewtonShared*>(smem_raw);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, task = blockIdx.x * kWarps + w;
  const bool active = task < a.ntasks;
  NewtonTask tk{};
  if (active) tk = a.tasks[task];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!active) return;
  const int n = a.n, tiles = (n + 31) / 32;
  const float k2inv = a.sc->k2inv;
  const f32x2 k2i2 = pk2(k2inv, k2inv);
  int I = tk.block, t = tk.tile, left = tk.count;
  while (left > 0) {
    const int i0 = I * kNewtonBlock, t1 = min(tiles, t + left);
    // Each i record passes through this lane's own entry of a tile buffer: the
    // other lanes' last reads of it lie before newton_tile's closing
    // __syncwarp, and their next ones after the one that follows the tile's own
    // records.  (Every other array here has lanes reach into each other's.)
    int4 q[kI];
#pragma unroll
    for (int k = 0; k < kI; ++k) {
      const int4 r = a.q[min(i0 + 32 * k + lane, n - 1)];
      q[k] = i_record_slots123(r, &sh.tile[w][0][lane]);
    }
#pragma unroll
    for (int m = 0; m < kI / 2; ++m)
#pragma unroll
      for (int k = 0; k < 5; ++k) sh.hi[w][m][k][lane] = sh.lo[w][m][k][lane] = 0ull;
    int4 next = a.q[min(t * 32 + lane, n - 1)];
    left -= t1 - t;
    for (; t < t1; ++t) {
      int4* const tile = sh.tile[w][t & 1];
      tile[lane] = next;
      __syncwarp();
      if (t + 1 < t1) next = a.q[min((t + 1) * 32 + lane, n - 1)];
      f32x2 f[kI / 2][5];
#pragma unroll
      for (int m = 0; m < kI / 2; ++m)
#pragma unroll
        for (int k = 0; k < 5; ++k) f[m][k] = 0ull;
      FloatAcc(*const J)[32] = sh.j[w];
      // the block's own tiles, and a last tile with fewer than 32 particles
      if (t < (I + 1) * kI || (t + 1) * 32 > n) newton_tile<true>(q, tile, k2i2, i0, t * 32, n, f, J);
      else newton_tile<false>(q, tile, k2i2, i0, t * 32, n, f, J);
      // tile t's sums from block I: triangular packing, tile-major
      const int tb = t / kI;  // t's own block
      float* const out = a.jpart + ((size_t)kI * ((size_t)tb * (tb + 1) / 2) + (size_t)(t - tb * kI) * (tb + 1) + I) * 160;
#pragma unroll
      for (int k = 0; k < 5; ++k) out[k * 32 + lane] = (k < 3 ? -1.0f : 1.0f) * (J[k][lane].hi + J[k][lane].lo);
#pragma unroll
      for (int m = 0; m < kI / 2; ++m)
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          Float2Acc acc{sh.hi[w][m][k][lane], sh.lo[w][m][k][lane]};
          two_sum_add2(acc, f[m][k]);
          sh.hi[w][m][k][lane] = acc.hi;
          sh.lo[w][m][k][lane] = acc.lo;
        }
    }
    float* const out = a.ipart + (size_t)(task + I) * 5 * kNewtonBlock;
#pragma unroll
    for (int m = 0; m < kI / 2; ++m)
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        float x, y;
        upk2(add2(sh.hi[w][m][k][lane], sh.lo[w][m][k][lane]), x, y);
        out[k * kNewtonBlock + 64 * m + lane] = x;
        out[k * kNewtonBlock + 64 * m + 32 + lane] = y;
      }
    ++I;
    t = I * kI;
  }
}

// One tile of 32 particles: its parts added in FP32 TwoSum (value c by kSum
// warps, every kSum-th part each; fixed order), then the step's second half
// with a thread per particle and component, as in k_rows.  One more CTA forms
// the observables the previous step left pending.  4 CTAs an SM: N = 16384
// fits into one wave (12.0 us; at 60 registers and 3 an SM 15.8).
namespace {
constexpr int kSum = 2;
}
template <int MODE>
__global__ void __launch_bounds__(160 * kSum, 4) k_newton_sum(StateArgs s, NewtonArgs a) {
  __shared__ FloatAcc part[kSum][5][32];
  __shared__ double red[5];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = warp % 5, u = warp / 5;
  const int n = a.n, t = blockIdx.x, i = t * 32 + lane;
  if (MODE != MODE_FORCES_ONLY && t == (n + 31) / 32) {
    extern __shared__ double shd[];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    pending_observables(s, 0, 1, shd);
    return;
  }
  const BoxArgs box = MODE == MODE_FORCES_ONLY ? BoxArgs{} : s.boxes[0];
  const int tb = t / kI, first = a.block_part[2 * tb], count = a.block_part[2 * tb + 1];
  const float* jp = a.jpart + ((size_t)kI * ((size_t)tb * (tb + 1) / 2) + (size_t)(t - tb * kI) * (tb + 1)) * 160 + c * 32 + lane;
  const float* ip = a.ipart + (size_t)first * 5 * kNewtonBlock + c * kNewtonBlock + (t - tb * kI) * 32 + lane;
  const int total = tb + 1 + count;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool mine = u == 0 && i < n;
  const size_t k3 = (size_t)min(c, 2) * s.npad + min(i, n - 1);
  double x = 0.0, v = 0.0, fn = 0.0;
  if (MODE != MODE_FORCES_ONLY && mine && c < 3) {
    x = s.x[k3];
    v = s.v[k3];
    fn = s.f[k3];
  }
  FloatAcc acc{0.f, 0.f};
  for (int k = u; k < total; k += 8 * kSum) {
    float val[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int p = k + m * kSum;
      val[m] = p >= total ? 0.0f : (p <= tb ? jp[(size_t)p * 160] : ip[(size_t)(p - tb - 1) * 5 * kNewtonBlock]);
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) two_sum_add(acc, val[m]);
  }
  part[u][c][lane] = acc;
  __syncthreads();
  auto value = [&](int k) {
    FloatAcc r = part[0][k][lane];
#pragma unroll
    for (int m = 1; m < kSum; ++m) {
      two_sum_add(r, part[m][k][lane].hi);
      r.lo += part[m][k][lane].lo;
    }
    return widen(r.hi) + widen(r.lo);
  };
  DevScalars& sc = s.sc[0];
  double p0 = 0.0, p1 = 0.0;
  if (mine && c < 3) {
    const double F = sc.fscale * value(c);
    if (MODE == MODE_EVN) {
      x = drift_pos(box, x, v, fn);
      v = fma(box.hdt, F, fma(box.hdt, fn, v));
      apply_bc1(box.bc, box.L, x, v);
      s.f[k3] = F;
      s.x[k3] = x;
      s.v[k3] = v;
      predict_coord(s, sc, box, c, i, drift_pos(box, x, v, F));
      p0 = v * v;
    } else if (MODE == MODE_TVN) {
      const double tv = fma(box.qdt, fn + F, v);
      s.tf[k3] = F;
      p0 = tv * tv;
    } else {
      reinterpret_cast<float*>(s.force4 + i)[c] = (float)F;
    }
  } else if (MODE == MODE_FORCES_ONLY && mine && c == 3) {
    const double A = value(3), B = value(4);
    s.force4[i].w = (float)(A - B);
    p0 = fma(12.0, A, -6.0 * B);
  } else if (mine && c == 3) {
    const double A = value(3), B = value(4);
    p0 = box.eps4 * (A - B);
    p1 = box.eps4 * fma(12.0, A, -6.0 * B);
    s.e[i] = p0;
    s.w[i] = p1;
  }
  if (u == 0 && c < 3) {
    p0 = warp_sum(p0);
    if (lane == 0) red[c] = p0;
  } else if (u == 0 && c == 3) {
    const double r = warp_sums<2>({p0, p1});
    if (lane == sums_lane(0)) red[3] = r;
    if (lane == sums_lane(1)) red[4] = r;
  }
  __syncthreads();
  if (MODE == MODE_FORCES_ONLY) {
    forces_only_finish(s, red[3]);
    return;
  }
  if (threadIdx.x != 0) return;
  double* const o = s.row_part + (size_t)t * 8;
  if (MODE == MODE_EVN) {
    o[s.obs_slot + 0] = 0.5 * (red[0] + red[1] + red[2]);
    o[s.obs_slot + 1] = 0.5 * red[3];
    o[s.obs_slot + 2] = red[4];
    if (t == 0) {
      const int par = s.ticket - 2;
      sc.obs_slot[par] = s.obs_slot;
      sc.obs_nblk[par] = gridDim.x - 1;
      sc.obs_pending[par] = MODE_EVN;
    }
  } else {
    o[3] = red[0] + red[1] + red[2];
  }
}

cudaError_t newton_setup(int* ctas_per_sm) {
  cudaError_t e = cudaFuncSetAttribute(k_newton, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(NewtonShared));
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, k_newton, 32 * kWarps, sizeof(NewtonShared));
}

cudaError_t launch_newton(const NewtonArgs& a, cudaStream_t st) {
  return launch_dependent(k_newton, (a.ntasks + kWarps - 1) / kWarps, 32 * kWarps, sizeof(NewtonShared), st, a);
}

cudaError_t launch_newton_sum(const StateArgs& s, const NewtonArgs& a, int mode, cudaStream_t st) {
  auto* k = mode == MODE_EVN   ? k_newton_sum<MODE_EVN>
            : mode == MODE_TVN ? k_newton_sum<MODE_TVN>
                               : k_newton_sum<MODE_FORCES_ONLY>;
  return launch_dependent(k, (a.n + 31) / 32 + (mode == MODE_FORCES_ONLY ? 0 : 1), 160 * kSum, sizeof(double) * 3 * 32,
                          st, s, a);
}

}  // namespace ljgb
