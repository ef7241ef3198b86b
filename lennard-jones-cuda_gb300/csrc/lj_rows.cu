// lj_rows.cu -- the MIXED step of one box of fewer than 8192 particles,
// a CTA per SM, each owning its rows (i's) outright.
//
// The stream-K kernel (lj_pairs.cu) cuts every i-block's j range over several
// CTAs, writes partial segments, and lets the last CTA of a block sum them
// and advance its particles, a thread per particle.  On a box of a few
// thousand particles that leaves most schedulers with one warp or none, and
// the step is a chain of round trips and of FP64 operations (64 clocks each
// when nothing else uses the pipe).  Here a CTA evaluates all pairs of its
// rows, so nothing leaves the SM: lanes take the j's, two rows a lane in the
// halves of the FP32x2 instructions, sums cross the lanes by shuffles and the
// warps through shared memory, and the step's second half has a thread per
// particle and component.  Equations and arithmetic per pair are those of
// lj_pairs.cu and fused_block_step.
#include <cuda_runtime.h>

#include <cstdint>

#include "lj_device.cuh"
#include "lj_kernels.h"
#include "lj_mixed.cuh"
#include "lj_stepdev.cuh"

namespace ljgb {
namespace {

constexpr int kRowWarps = 16;    // 12 to 20 warps measure alike (N = 400 to 8000)
constexpr int kRowThreads = 32 * kRowWarps;
constexpr int kRowFold = 32;     // j's a lane sums in plain FP32 before the compensated sum takes them
constexpr int kMaxRows = 64;     // rows of a CTA: 4 threads each in the second half

__device__ __forceinline__ int4 load_slots(const int4* rec) {
  int4 r;  // volatile: kept a 128-bit load into an aligned register quadruple
  asm volatile("ld.volatile.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "r"(smem_addr(rec)));
  return r;
}

// Pairs of two rows with chunks c0 .. c1-1 (32 j's each, one a lane) of the n
// records st; the lanes' sums added up into out[row * 5 + value].  self: the
// first row's index (even).
// UNROLL: chunks in flight.  The registers that the second half holds meanwhile
// decide: us a step, 4 / 8, TVN N = 4000 19.3 / 19.7, N = 8000 49.7 / 51.0; EVN N =
// 2001 7.9 / 8.1, N = 4000 16.3 / 16.0, N = 8000 49.0 / 47.5.
template <int UNROLL>
__device__ __forceinline__ void row_portion(const int4* rowq, const int4* st, int n, int c0, int c1, int self,
                                            f32x2 k2i2, float* out) {
  const int lane = threadIdx.x & 31;
  const int4 qa = load_slots(rowq), qb = load_slots(rowq + 1);
  Float2Acc acc[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) acc[k] = Float2Acc{0ull, 0ull};
  const int ragged = (n & 31) ? n >> 5 : -1;  // chunk that ends before its 32nd record
  const int cself = self >> 5;                    // chunk that holds the rows themselves
  for (int c = c0; c < c1;) {
    const int special = cself >= c && cself < c1 ? cself : (ragged >= c && ragged < c1 ? ragged : c1);
    f32x2 f[5] = {0ull, 0ull, 0ull, 0ull, 0ull};
    if (c < special) {
      const int ce = min(special, c + kRowFold);
#pragma unroll UNROLL
      for (; c < ce; ++c)
        pair_mixed_rows<false>(qa, qb, st[c * 32 + lane], k2i2, false, false, f[0], f[1], f[2], f[3], f[4]);
    } else {
      const int j = c * 32 + lane;
      const bool out_of = j >= n;
      pair_mixed_rows<true>(qa, qb, st[out_of ? 0 : j], k2i2, out_of || j == self, out_of || j == self + 1, f[0], f[1],
                            f[2], f[3], f[4]);
      ++c;
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) two_sum_add2(acc[k], f[k]);
  }
  // The lanes' forces meet as TwoSum pairs too, their energies (compensated so
  // far) in plain FP32, five additions where the stream-K kernel has one a chunk
  // over a tile.  Row 0 goes to the lower half of the warp and row 1 to the
  // upper; then value 0 or 1 (3 or 4) is kept by every other eight lanes, and
  // that or value 2 by every other four (fixed order).  All five values plain,
  // 0.3 us of an EVN step faster at N = 2001 (20 steps: 185 us, so 191), lose a
  // force that meets a larger one in another lane.
  const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
  FloatAcc f[3];
  float ke[2];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    FloatAcc a, b;
    upk2(acc[k].hi, a.hi, b.hi);
    upk2(acc[k].lo, a.lo, b.lo);
    f[k] = exchange1(a, b, h16, 16);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    float a, b;
    upk2(add2(acc[3 + k].hi, acc[3 + k].lo), a, b);
    ke[k] = (h16 ? b : a) + __shfl_xor_sync(0xffffffffu, h16 ? a : b, 16);
  }
  FloatAcc v = exchange1(f[0], f[1], h8, 8);
  const FloatAcc v2 = exchange1(f[2], f[2], false, 8);
  float e = (h8 ? ke[1] : ke[0]) + __shfl_xor_sync(0xffffffffu, h8 ? ke[0] : ke[1], 8);
  v = exchange1(v, v2, h4, 4);
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) v = exchange1(v, v, false, o);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  float* const row = out + (h16 ? 5 : 0);
  if ((lane & 3) == 0 && !(h4 && h8)) row[h4 ? 2 : h8 ? 1 : 0] = v.hi + v.lo;
  if ((lane & 7) == 0) row[h8 ? 4 : 3] = e;
}

// The warp that works on unit u when U units are cut evenly over the warps.
__device__ __forceinline__ int warp_of_unit(int u, int U) { return ((u + 1) * kRowWarps - 1) / U; }

}  // namespace

// One step of one box: CTA b owns rows [b * rows, (b + 1) * rows); the last
// CTA computes the observables the previous step left pending.  MODE_EVN: the
// whole step; MODE_TVN: up to sum tv^2 (k_rows_close follows).
//
// The work is groups x chunks units (two rows x 32 j's) in one sequence, cut
// evenly over the warps; the portion of group g by warp w has slot w + g (the
// sequence visits (w, g) monotonically, so no two portions share a slot), and
// the second half adds a row's slots in a fixed order.
//
// Bound: from N ~ 8000 the pair loop's issue and register reads as in
// lj_pairs.cu; below ~2000 the fixed parts (launch, first copy, reductions, a
// chain of ~15 FP64 operations), ~5 us.  us a step, stream-K kernel -> this
// one, on GB300: EVN N = 400 14.4 -> 5.5, N = 1000 16.4 -> 6.2, N = 2001 20.5
// -> 8.1; TVN N = 256 18.4 -> 8.3, N = 4000 30.8 -> 19.3, N = 8000 70 -> 49.7.
template <int MODE>
__global__ void __launch_bounds__(kRowThreads, 1) k_rows(StateArgs s, int n, int rows, int ctas) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t bar;
  __shared__ volatile int sfail;
  __shared__ int4 srow[kMaxRows];
  __shared__ double red[5][2];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int4* const sq = reinterpret_cast<int4*>(smem_raw);              // all n records
  float* const part = reinterpret_cast<float*>(smem_raw + sizeof(int4) * (size_t)n);

  if (MODE != MODE_FORCES_ONLY && (int)blockIdx.x == ctas) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (MODE == MODE_EVN) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    pending_observables(s, 0, 1, reinterpret_cast<double*>(smem_raw));
    return;
  }
  const int i0 = blockIdx.x * rows, nr = min(rows, n - i0), groups = (nr + 1) / 2;
  const int slots = kRowWarps + groups;
  if (tid == 0) {
    mbar_init(&bar, 1);
    sfail = 0;
    fence_mbar_init();
  }
  for (int k = tid; k < slots * 10; k += kRowThreads) part[k] = 0.0f;
  const BoxArgs box = MODE == MODE_FORCES_ONLY ? BoxArgs{} : s.boxes[0];
  __syncthreads();
  // What the previous step's kernels write is read from here on.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // The next step's CTAs (a whole SM each) may queue up behind these.  TVN's
  // close is only launched as these end: its small CTAs would all crowd onto
  // the few SMs left free and take turns at their FP64 pipes (N = 2001: the
  // close added 8.1 us to the step, and 4 us so).
  if (MODE == MODE_EVN) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) {
    mbar_arrive_expect_tx(&bar, (uint32_t)n * 16u);
    bulk_g2s(sq, s.q, (uint32_t)n * 16u, &bar);
  }
  if (tid < 2 * groups) {
    const int4 q = s.q[min(i0 + tid, n - 1)];
    srow[tid] = make_int4(0, q.x, q.y, q.z);
  }
  DevScalars& sc = s.sc[0];
  const float k2inv = sc.k2inv;
  if (MODE == MODE_EVN && blockIdx.x == 0 && tid == 0) {
    // pending once the launch completes; this launch reads the other parity's
    const int par = s.ticket - 2;
    sc.obs_slot[par] = s.obs_slot;
    sc.obs_nblk[par] = ctas;
    sc.obs_pending[par] = MODE_EVN;
  }
  // second half: threads [c * rpad, (c + 1) * rpad) hold component c of the
  // rows, those of c = 3 the energies
  const int rpad = (nr + 31) / 32 * 32, c = tid / rpad, r = tid - c * rpad;
  const bool mine = c < 4 && r < nr;
  const size_t k3 = (size_t)min(c, 2) * s.npad + i0 + min(r, nr - 1);
  double x = 0.0, v = 0.0, fn = 0.0;
  if (MODE != MODE_FORCES_ONLY && mine && c < 3) {
    x = s.x[k3];
    v = s.v[k3];
    fn = s.f[k3];
  }
  __syncthreads();

  const int C = (n + 31) / 32, U = groups * C;
  if (__all_sync(0xffffffffu, mbar_wait_bounded(&bar, 0))) {
    const f32x2 k2i2 = pk2(k2inv, k2inv);
    const int hi = (w + 1) * U / kRowWarps;
    for (int u = w * U / kRowWarps; u < hi;) {
      const int g = u / C, c0 = u - g * C, c1 = min(C, c0 + hi - u);
      row_portion<MODE == MODE_TVN ? 4 : 8>(srow + 2 * g, sq, n, c0, c1, i0 + 2 * g, k2i2, part + (w + g) * 10);
      u += c1 - c0;
    }
  } else if (lane == 0) {
    sfail = 1;
  }
  __syncthreads();
  if (sfail) {
    // The copy is waited for once more before the shared memory goes.
    if (tid == 0) {
      mbar_wait_bounded(&bar, 0);
      atomicOr(s.status, LJ_DEVFLAG_TIMEOUT);
    }
    return;
  }

  // A row's value k: its slots, in FP32 TwoSum, then FP64.
  auto row_sum = [&](int k) {
    FloatAcc a{0.f, 0.f};
    const int g = r >> 1, w1 = warp_of_unit((g + 1) * C - 1, U);
    const float* p = part + g * 10 + (r & 1) * 5 + k;
    for (int ww = warp_of_unit(g * C, U); ww <= w1; ++ww) two_sum_add(a, p[ww * 10]);
    return widen(a.hi) + widen(a.lo);
  };
  double p0 = 0.0, p1 = 0.0;  // c < 3: v^2 (EVN) or tv^2; c = 3: e, w
  if (mine) {
    if (c < 3) {
      const double F = sc.fscale * row_sum(c);
      if (MODE == MODE_EVN) {
        x = drift_pos(box, x, v, fn);
        v = fma(box.hdt, F, fma(box.hdt, fn, v));
        apply_bc1(box.bc, box.L, x, v);
        s.f[k3] = F;
        s.x[k3] = x;
        s.v[k3] = v;
        predict_coord(s, sc, box, c, i0 + r, drift_pos(box, x, v, F));
        p0 = v * v;
      } else if (MODE == MODE_TVN) {
        const double tv = fma(box.qdt, fn + F, v);
        s.tf[k3] = F;
        p0 = tv * tv;
      } else {
        reinterpret_cast<float*>(s.force4 + i0 + r)[c] = (float)F;
      }
    } else if (MODE == MODE_FORCES_ONLY) {
      const double A = row_sum(3), B = row_sum(4);
      s.force4[i0 + r].w = (float)(A - B);
      p0 = fma(12.0, A, -6.0 * B);
    } else {
      const double A = row_sum(3), B = row_sum(4);
      p0 = box.eps4 * (A - B);
      p1 = box.eps4 * fma(12.0, A, -6.0 * B);
      s.e[i0 + r] = p0;
      s.w[i0 + r] = p1;
    }
  }
  if (c < 4) {  // whole warps
    const int wi = r / 32;
    if (MODE == MODE_EVN && c == 3) {
      p0 = warp_sums<2>({p0, p1});
      p1 = __shfl_sync(0xffffffffu, p0, sums_lane(1));
    } else if (MODE == MODE_EVN || (MODE == MODE_TVN) == (c < 3)) {
      p0 = warp_sum(p0);
    }
    if (lane == 0) {
      red[c][wi] = p0;
      if (c == 3) red[4][wi] = p1;
      if (rpad == 32) red[c][1] = red[c == 3 ? 4 : c][1] = 0.0;
    }
  }
  __syncthreads();
  if (MODE == MODE_FORCES_ONLY) {
    forces_only_finish(s, red[3][0] + red[3][1]);
  } else if (w == 0 && lane < 3) {
    auto both = [&](int k) { return red[k][0] + red[k][1]; };
    double* const o = s.row_part + (size_t)blockIdx.x * 8;
    if (MODE == MODE_EVN) {
      if (lane == 0) o[s.obs_slot + 0] = 0.5 * (both(0) + both(1) + both(2));
      if (lane == 1) o[s.obs_slot + 1] = 0.5 * both(3);
      if (lane == 2) o[s.obs_slot + 2] = both(4);
    } else if (lane == 0) {
      o[3] = both(0) + both(1) + both(2);
    }
  }
}

// Close of a TVN step (k_tvn_close's equations) for 32 particles: warp c holds
// component c; the fourth warp forms chi and sums the energies.
__global__ void __launch_bounds__(128) k_rows_close(StateArgs s, int n, int ctas) {
  __shared__ double chi_sh, tkin_sh, ksum[3], vw[2];
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * 32 + lane;
  const bool valid = i < n;
  const BoxArgs box = s.boxes[0];
  const size_t k3 = (size_t)min(c, 2) * s.npad + min(i, n - 1);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  DevScalars& sc = s.sc[0];
  double x = 0.0, v = 0.0, fn = 0.0, f1 = 0.0;
  if (c < 3) {
    x = s.x[k3];
    v = s.v[k3];
    fn = s.f[k3];
    f1 = s.tf[k3];
    x = drift_pos(box, x, v, fn);
  } else {
    double tv2 = 0.0;
    for (int b = lane; b < ctas; b += 32) tv2 += __ldcg(s.row_part + (size_t)b * 8 + 3);
    const double r = warp_sums<3>({tv2, valid ? s.e[i] : 0.0, valid ? s.w[i] : 0.0});
    if (lane == 0) {
      double Tkin;
      chi_sh = tvn_chi(box, r, &Tkin);
      tkin_sh = Tkin;
    }
    if (lane == sums_lane(1)) vw[0] = r;
    if (lane == sums_lane(2)) vw[1] = r;
  }
  __syncthreads();
  if (c < 3) {
    const double chi = chi_sh;
    v = fma(2. * chi - 1., v, 0.5 * (chi * box.dt) * (fn + f1));
    apply_bc1(box.bc, box.L, x, v);
    if (valid) {
      s.v[k3] = v;
      s.x[k3] = x;
      s.f[k3] = f1;
      predict_coord(s, sc, box, c, i, drift_pos(box, x, v, f1));
    }
    const double vv = warp_sum(valid ? v * v : 0.0);
    if (lane == 0) ksum[c] = vv;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double* const o = s.row_part + (size_t)blockIdx.x * 8 + s.obs_slot;
    o[0] = 0.5 * (ksum[0] + ksum[1] + ksum[2]);
    o[1] = 0.5 * vw[0];
    o[2] = vw[1];
    if (blockIdx.x == 0) {
      const int par = s.ticket - 2;
      sc.Tkin = tkin_sh;
      sc.Tkin_rec[par] = tkin_sh;
      sc.chi = chi_sh;
      sc.obs_slot[par] = s.obs_slot;
      sc.obs_nblk[par] = gridDim.x;
      sc.obs_pending[par] = MODE_TVN;
    }
  }
}

// Rows in pairs, and one SM left to the observables' CTA.
RowPlan plan_rows(int n, int sms) {
  RowPlan p{};
  if (sms < 2 || n >= kNewtonMinN) return p;
  const int unit = 2 * (sms - 1);
  p.rows = 2 * ((n + unit - 1) / unit);
  if (p.rows > kMaxRows) return RowPlan{};
  p.ctas = (n + p.rows - 1) / p.rows;
  p.smem = sizeof(int4) * (size_t)n + sizeof(float) * 10 * (size_t)(kRowWarps + p.rows / 2);
  if (p.smem < sizeof(double) * 3 * 32) p.smem = sizeof(double) * 3 * 32;  // the observables' sums
  return p;
}

cudaError_t rows_setup() {
  constexpr int kMost = sizeof(int4) * kNewtonMinN + sizeof(float) * 10 * (kRowWarps + kMaxRows / 2);
  cudaError_t e = cudaFuncSetAttribute(k_rows<MODE_EVN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rows<MODE_TVN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_rows<MODE_FORCES_ONLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
  return e;
}

cudaError_t launch_rows(const StateArgs& s, const RowPlan& p, int n, int mode, cudaStream_t st) {
  auto* k = mode == MODE_EVN ? k_rows<MODE_EVN> : mode == MODE_TVN ? k_rows<MODE_TVN> : k_rows<MODE_FORCES_ONLY>;
  return launch_dependent(k, p.ctas + (mode == MODE_FORCES_ONLY ? 0 : 1), kRowThreads, p.smem, st, s, n, p.rows,
                          p.ctas);
}

cudaError_t launch_rows_close(const StateArgs& s, int n, int parts, cudaStream_t st) {
  return launch_dependent(k_rows_close, (n + 31) / 32, 128, 0, st, s, n, parts);
}

}  // namespace ljgb
