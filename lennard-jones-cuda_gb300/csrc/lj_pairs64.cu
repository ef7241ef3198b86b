// lj_pairs64.cu -- all-FP64 pair kernel (LJ_PREC_FP64): forces and energy
// sums of every unordered pair evaluated once, and the second half of the
// kernel-per-phase step that sums its parts.
//
// Same pair set and physics as the reference's loop over ordered pairs
// (src/library/MDSystem.cu:21-56, src/library/MDSystem.cpp:260-310).
#include <cuda_runtime.h>

#include <cstdint>

#include "lj_device.cuh"
#include "lj_kernels.h"
#include "lj_pair64.cuh"
#include "lj_stepdev.cuh"

namespace ljgb {
namespace {

// A task is a square of `group` x `group` tiles of 32 particles.  Each lane
// holds one i and one j; the j positions and sums move to the next lane after
// every pair, so in 32 turns all 32 x 32 pairs of two tiles meet and both
// particles' sums grow without any reduction across lanes.  A tile against
// itself takes turns 1..16 (turn 16 meets every pair from both ends: the
// lower half of the warp keeps it).
//
// A task has one CTA: of one warp, or, for small boxes (squares of one tile),
// of `parts` warps that share the square's turns and add their sums in shared
// memory.  One-warp CTAs spread evenly: N = 2048 has 2080 tasks for 152 SMs.
//
// Bound: the FP64 pipe, 85% of whose rate it reaches.  28 operations an
// unordered pair with sigma = 1 (3 differences, 3 images, 3 r^2, 3 reciprocal,
// 5 powers and force factor, 6 force sums, 4 energy sums), against 2 x 36 of
// the loop over ordered pairs that this kernel replaced (IEEE division,
// product-round-fma images).  N = 2048: 355 -> 114 us; N = 512: 103 -> 13 us.
struct Sums64 {
  double x, y, z, a, b;  // s d, (s/r)^12, (s/r)^6
};

// Turns r0 .. r1-1 of tiles ta and tb (positions xi, x_tb); J enters with the
// sums of the lane's first j and leaves with those of the returned one.
template <bool PERIODIC, bool UNIT>
__device__ __forceinline__ int pairs64_turns(const double4_32a* xd, const BoxArgs& box, int n, int ta, int tb, int r0,
                                             int r1, double4_32a xi, Sums64& I, Sums64& J) {
  const int lane = threadIdx.x & 31;
  const bool vi = ta * 32 + lane < n, diag = ta == tb;
  const double s2 = box.sigma * box.sigma;
  const ImageBounds ib{box.image_lo, box.image_hi};
  int jl = (lane + r0) & 31;
  const double4_32a xj4 = xd[min(tb * 32 + jl, n - 1)];
  double xj = xj4.x, yj = xj4.y, zj = xj4.z;
  __builtin_assume((r1 - r0) % 2 == 0);  // Pair64Plan::parts sees to it
#pragma unroll 2
  for (int r = r0; r < r1; ++r) {
    double d[3] = {xi.x - xj, xi.y - yj, xi.z - zj};
    if (PERIODIC) nearest_image<true>(d, box.L, box.invL, ib);
    double r2 = fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0]));
    double y = rcp_seed(r2);
    const bool meets = vi && tb * 32 + jl < n && !(diag && r == 16 && lane >= 16);
    if (!meets || beyond_seed(r2)) {  // a seed of 0 makes the pair's terms 0
      r2 = 1.0;
      y = 0.0;
    }
    const double ri = UNIT ? rcp_from_seed(r2, y) : div_from_seed(s2, r2, y);
    const double r6 = ri * ri * ri;
    const double sf = r6 * ri * fma(12.0, r6, -6.0);
    I.x = fma(sf, d[0], I.x);
    I.y = fma(sf, d[1], I.y);
    I.z = fma(sf, d[2], I.z);
    I.a = fma(r6, r6, I.a);
    I.b += r6;
    J.x = shfl_next(fma(-sf, d[0], J.x), lane);
    J.y = shfl_next(fma(-sf, d[1], J.y), lane);
    J.z = shfl_next(fma(-sf, d[2], J.z), lane);
    J.a = shfl_next(fma(r6, r6, J.a), lane);
    J.b = shfl_next(J.b + r6, lane);
    jl = (jl + 1) & 31;
    xj = shfl_next(xj, lane);
    yj = shfl_next(yj, lane);
    zj = shfl_next(zj, lane);
  }
  return jl;
}

__device__ __forceinline__ void store_sums(double* to, int at, const Sums64& s) {
  to[at] = s.x;
  to[32 + at] = s.y;
  to[64 + at] = s.z;
  to[96 + at] = s.a;
  to[128 + at] = s.b;
}

template <bool PERIODIC, bool UNIT>
__device__ __forceinline__ void pairs64_task(const Pair64Args& a, const Pair64Task tk, const Pair64Box& bt,
                                             const BoxArgs& box, double* sh) {
  const int lane = threadIdx.x & 31;
  const double4_32a* xd = a.xd + bt.p0;
  const int slots = (bt.groups + 1) * a.split;  // of one tile
  double* const part = a.part + (size_t)bt.tile0_slot * 160;
  if (a.parts > 1) {
    const int w = threadIdx.x >> 5, ta = tk.ga, tb = tk.gb;
    const int turns = (ta == tb ? min(16, a.turns) : a.turns) / a.parts;
    const int first = (ta == tb ? 1 : 0) + a.turns * tk.slot;
    Sums64 I{}, J{};
    const int jl = pairs64_turns<PERIODIC, UNIT>(xd, box, bt.n, ta, tb, first + w * turns, first + (w + 1) * turns,
                                                 xd[min(ta * 32 + lane, bt.n - 1)], I, J);
    store_sums(sh + w * 320, lane, I);
    store_sums(sh + w * 320 + 160, jl, J);
    __syncthreads();
    for (int k = threadIdx.x; k < 320; k += blockDim.x) {
      double v = 0.0;
      for (int p = 0; p < a.parts; ++p) v += sh[p * 320 + k];
      // i sums: tile ta, slot of the square's column; j sums: tile tb, slot of its row
      if (k < 160) part[((size_t)ta * slots + (tb + 1) * a.split + tk.slot) * 160 + k] = v;
      else part[((size_t)tb * slots + ta * a.split + tk.slot) * 160 + k - 160] = v;
    }
    return;
  }
  const int a0 = tk.ga * a.group, a1 = min(bt.tiles, a0 + a.group);
  const int b0 = tk.gb * a.group, b1 = min(bt.tiles, b0 + a.group);
  for (int ta = a0; ta < a1; ++ta) {
    const double4_32a xi = xd[min(ta * 32 + lane, bt.n - 1)];
    Sums64 I{};
    for (int tb = max(ta, b0); tb < b1; ++tb) {
      const int r0 = (ta == tb ? 1 : 0) + a.turns * tk.slot, r1 = r0 + (ta == tb ? min(16, a.turns) : a.turns);
      double* const jslot = part + ((size_t)tb * slots + tk.ga * a.split + tk.slot) * 160;
      const int at = (lane + r0) & 31;
      Sums64 J{};
      if (ta > a0)  // earlier rows' sums
        J = Sums64{jslot[at], jslot[32 + at], jslot[64 + at], jslot[96 + at], jslot[128 + at]};
      const int jl = pairs64_turns<PERIODIC, UNIT>(xd, box, bt.n, ta, tb, r0, r1, xi, I, J);
      store_sums(jslot, jl, J);
      __syncwarp();  // the next row's lanes read each other's sums
    }
    store_sums(part + ((size_t)ta * slots + (tk.gb + 1) * a.split + tk.slot) * 160, lane, I);
  }
}

__global__ void __launch_bounds__(256) k_pairs64(Pair64Args a) {
  extern __shared__ double sh[];  // parts > 1: parts x 2 x 5 x 32
  const Pair64Task tk = a.tasks[blockIdx.x];
  const int sys = a.nsys == 1 ? 0 : tk.sys;  // one box: its tables load beside the task's
  const Pair64Box bt = a.boxes64[sys];
  const BoxArgs box = a.boxes[sys];
  // A programmatic dependent of the kernel that wrote the shadow; its own
  // dependent (k_reduce64) may be scheduled as the last tasks end.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool unit = box.sigma == 1.0;
  if (box.bc == 0) {
    if (unit) pairs64_task<true, true>(a, tk, bt, box, sh);
    else pairs64_task<true, false>(a, tk, bt, box, sh);
  } else {
    if (unit) pairs64_task<false, true>(a, tk, bt, box, sh);
    else pairs64_task<false, false>(a, tk, bt, box, sh);
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// End of a kernel with a CTA per tile: the CTA that finishes a box's last tile
// goes on to the box's observables (a launch of their own took 5 us).
// Block-wide call.
template <int MODE>
__device__ __forceinline__ void finish_box(const StateArgs& s, const BlockInfo& bi, int tiles, const BoxArgs& box) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  const int b0 = blockIdx.x - bi.i0 / 32, lane = threadIdx.x & 31;  // b0: the box's first block
  if (threadIdx.x == 0) last = atomicAdd(s.blk_cnt + b0, 1) == tiles - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) s.blk_cnt[b0] = 0;
  if (threadIdx.x >= 32) return;
  double kvw[3] = {0.0, 0.0, 0.0};
  for (int k = lane; k < tiles; k += 32)
#pragma unroll
    for (int m = 0; m < 3; ++m) kvw[m] += __ldcg(s.blk_part + (size_t)(b0 + k) * 8 + m);
#pragma unroll
  for (int m = 0; m < 3; ++m) kvw[m] = warp_sum(kvw[m]);
  if (lane == 0) write_observables<MODE>(s, bi.sys, box, kvw[0], kvw[1], kvw[2], -1);
}

// What a finished step leaves of component c for the next pair pass, the next
// step's drift, and for the histogram (periodic boxes), the position's
// fixed-point shadow.
__device__ __forceinline__ void carry64(const StateArgs& s, const BoxArgs& box, int sys, int4* qhist, int c, int at,
                                        double x, double v, double F) {
  reinterpret_cast<double*>(s.xd + at)[c] = drift_pos(box, x, v, F);
  if (qhist) reinterpret_cast<int*>(qhist + at)[c] = fixed_coord_scaled(x, frame_scale(s.sc[sys]));
}

// One tile of 32 particles: the sums over its slots (value c of a particle by
// four warps, a quarter of the slots each; fixed order), then, a component
// per warp, what k_reduce does for the mixed path: (EVN) the second half-kick
// and boundaries, (TVN) the averaged force and the half-kicked velocity whose
// kinetic temperature sets chi.  Block partials [0] K, [1] V, [2] W, [3]
// sum tv^2.
// CARRIED: x, v and F are those of the step's start and the shadow held the
// drift; the drift is taken here, and the next one's shadow left behind (a
// launch for the drift: 4.5 us a step).
// Latency is what bounds it: the slots' loads, then a serial chain of FP64
// operations (a warp's takes 16 clocks of the SM's pipe alone).
constexpr int kSumWarps = 4;  // warps per value
template <int MODE, bool CARRIED>
__global__ void __launch_bounds__(160 * kSumWarps) k_reduce64(StateArgs s, Pair64Args a, int4* qhist) {
  __shared__ double sum[kSumWarps][5][32];
  __shared__ double ksum[3], tsum[3];
  const int B = blockIdx.x, warp = threadIdx.x >> 5, c = warp % 5, u = warp / 5, lane = threadIdx.x & 31;
  const BlockInfo bi = s.blocks[B];
  const Pair64Box bt = a.boxes64[bi.sys];
  const BoxArgs box = s.boxes[bi.sys];
  const int slots = (bt.groups + 1) * a.split;
  const double* p = a.part + ((size_t)bt.tile0_slot + (size_t)(bi.i0 / 32) * slots) * 160 + c * 32 + lane;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool valid = lane < bi.n_i;
  const int at = bi.p0 + bi.i0 + lane;
  const size_t k3 = (size_t)min(c, 2) * s.npad + (valid ? at : bi.p0 + bi.i0);
  double x = 0.0, v = 0.0, fn = 0.0;
  if (u == 0 && c < 3) {
    x = s.x[k3];
    v = s.v[k3];
    if (CARRIED) fn = s.f[k3];
    else if (MODE == MODE_TVN) fn = s.tf[k3];  // F_n / 2
  }
  double q0 = 0., q1 = 0.;
  for (int k = u; k < slots; k += 8 * kSumWarps) {
    double val[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) val[m] = k + m * kSumWarps < slots ? p[(size_t)(k + m * kSumWarps) * 160] : 0.0;
    q0 += (val[0] + val[2]) + (val[4] + val[6]);
    q1 += (val[1] + val[3]) + (val[5] + val[7]);
  }
  sum[u][c][lane] = q0 + q1;
  __syncthreads();
  auto total = [&](int k) { return (sum[0][k][lane] + sum[1][k][lane]) + (sum[2][k][lane] + sum[3][k][lane]); };
  double vv = 0.0, tv2 = 0.0;
  if (u == 0 && c < 3) {
    if (valid) {
      const double F = box.fscale64 * total(c);
      s.f[k3] = F;
      if (CARRIED) x = drift_pos(box, x, v, fn);
      if (MODE == MODE_FORCES_ONLY) {
        vv = v * v;
      } else if (MODE == MODE_EVN) {
        if (CARRIED) v = fma(box.hdt, fn, v);
        v = fma(box.hdt, F, v);
        apply_bc1(box.bc, box.L, x, v);
        s.v[k3] = v;
        if (CARRIED || box.bc == 0) s.x[k3] = x;
        if (CARRIED) carry64(s, box, bi.sys, qhist, c, at, x, v, F);
        vv = v * v;
      } else {  // TVN
        const double tf = (CARRIED ? 0.5 * fn : fn) + 0.5 * F;
        s.tf[k3] = tf;
        if (CARRIED) s.x[k3] = x;
        const double tv = fma(box.hdt, tf, v);
        tv2 = tv * tv;
      }
    }
    vv = warp_sum(MODE == MODE_TVN ? tv2 : vv);
    if (lane == 0) (MODE == MODE_TVN ? tsum : ksum)[c] = vv;
  } else if (u == 0 && c == 3) {
    double e = 0.0, w = 0.0;
    if (valid) {
      const double A = total(3), Bs = total(4);
      e = box.eps4 * (A - Bs);
      w = box.eps4 * fma(12.0, A, -6.0 * Bs);
      s.e[at] = e;
      s.w[at] = w;
    }
    const double r = warp_sums<2>({e, w});
    if (lane == sums_lane(0)) s.blk_part[(size_t)B * 8 + 1] = 0.5 * r;
    if (lane == sums_lane(1)) s.blk_part[(size_t)B * 8 + 2] = r;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (MODE == MODE_TVN) s.blk_part[(size_t)B * 8 + 3] = tsum[0] + tsum[1] + tsum[2];
    else s.blk_part[(size_t)B * 8 + 0] = 0.5 * (ksum[0] + ksum[1] + ksum[2]);
  }
  if (MODE != MODE_TVN) finish_box<MODE>(s, bi, bt.tiles, box);  // (TVN: K follows from chi)
}

// TVN velocity update (MDSystem.cpp:498-506) of a tile, a component per warp:
// chi = sqrt(T0 / Tkin(tv)) by the fourth warp, v = (2 chi - 1) v + chi dt tF,
// boundaries, K, the box's observables, and what is carried to the next step.
// (Two launches before, a thread per particle and then the observables.)
template <bool CARRIED>
__global__ void __launch_bounds__(128) k_close64(StateArgs s, Pair64Args a, int4* qhist) {
  __shared__ double chi_sh, ksum[3];
  const int B = blockIdx.x, c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const BlockInfo bi = s.blocks[B];
  const BoxArgs box = s.boxes[bi.sys];
  const int tiles = a.boxes64[bi.sys].tiles, b0 = B - bi.i0 / 32;
  const bool valid = lane < bi.n_i;
  const int at = bi.p0 + bi.i0 + lane;
  const size_t k3 = (size_t)min(c, 2) * s.npad + (valid ? at : bi.p0 + bi.i0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  double x = 0.0, v = 0.0, tf = 0.0, F = 0.0;
  if (c < 3) {
    x = s.x[k3];
    v = s.v[k3];
    tf = s.tf[k3];
    if (CARRIED) F = s.f[k3];
  } else {
    double tv2 = 0.0;
    for (int k = lane; k < tiles; k += 32) tv2 += __ldcg(s.blk_part + (size_t)(b0 + k) * 8 + 3);
    tv2 = warp_sum(tv2);
    if (lane == 0) {
      double Tkin;
      chi_sh = tvn_chi(box, tv2, &Tkin);
      if (B == b0) {
        s.sc[bi.sys].Tkin = Tkin;
        s.sc[bi.sys].chi = chi_sh;
      }
    }
  }
  __syncthreads();
  if (c < 3) {
    const double chi = chi_sh;
    v = fma(2. * chi - 1., v, chi * box.dt * tf);
    apply_bc1(box.bc, box.L, x, v);
    if (valid) {
      s.v[k3] = v;
      if (box.bc == 0) s.x[k3] = x;
      if (CARRIED) carry64(s, box, bi.sys, qhist, c, at, x, v, F);
    }
    const double vv = warp_sum(valid ? v * v : 0.0);
    if (lane == 0) ksum[c] = vv;
  }
  __syncthreads();
  if (threadIdx.x == 0) s.blk_part[(size_t)B * 8 + 0] = 0.5 * (ksum[0] + ksum[1] + ksum[2]);
  finish_box<MODE_TVN>(s, bi, tiles, box);
}

}  // namespace

void fp64_image_bounds(double L, double invL, long long* lo, long long* hi) {
  const ImageBounds b = image_bounds(L, invL, true);  // ties away from zero (fast_round, MDSystem.cpp:732-739)
  *lo = b.lo;
  *hi = b.hi;
}

cudaError_t launch_pairs64(const Pair64Args& a, cudaStream_t st) {
  return launch_dependent(k_pairs64, a.ntasks, 32 * a.parts, a.parts > 1 ? sizeof(double) * 320 * a.parts : 0, st, a);
}

cudaError_t launch_reduce64(const StateArgs& s, const Pair64Args& a, int nblocks, int mode, bool carried, int4* qhist,
                            cudaStream_t st) {
  auto* k = mode == MODE_FORCES_ONLY ? k_reduce64<MODE_FORCES_ONLY, false>
            : mode == MODE_EVN       ? (carried ? k_reduce64<MODE_EVN, true> : k_reduce64<MODE_EVN, false>)
                                     : (carried ? k_reduce64<MODE_TVN, true> : k_reduce64<MODE_TVN, false>);
  cudaError_t e = launch_dependent(k, nblocks, 160 * kSumWarps, 0, st, s, a, qhist);
  if (e != cudaSuccess || mode != MODE_TVN) return e;
  return launch_dependent(carried ? k_close64<true> : k_close64<false>, nblocks, 128, 0, st, s, a, qhist);
}

}  // namespace ljgb
