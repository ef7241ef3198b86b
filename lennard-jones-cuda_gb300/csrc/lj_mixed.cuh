// lj_mixed.cuh -- pair arithmetic of the MIXED path: fixed-point separations,
// FP32 terms, two pairs at a time in packed FP32x2 instructions.
#pragma once

#include <cuda_runtime.h>

#include "lj_device.cuh"

namespace ljgb {

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// One pair in the MIXED path.  d = qi - qj wraps to the minimum image (qi
// in slots 1..3, see i_record_slots123).
// s = (s/r)^8 [12 (s/r)^6 - 6] (sigma units), a += (s/r)^12, b += (s/r)^6.
template <bool MASKED>
__device__ __forceinline__ void pair_mixed(const int4 qi, const int4 qj, float k2inv, bool excl,
                                           float& fx, float& fy, float& fz, float& pa,
                                           float& pb) {
  const float dx = __int2float_rn(fixed_diff(qi.y, qj.x));
  const float dy = __int2float_rn(fixed_diff(qi.z, qj.y));
  const float dz = __int2float_rn(fixed_diff(qi.w, qj.z));
  const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
  // r2 is in fixed-point units^2, between ~1e14 and ~1.4e19: far from the
  // subnormal and 2^126 ranges, so the raw approximate reciprocal applies.
  float ri = k2inv * rcp_approx(r2);
  if (MASKED) ri = excl ? 0.0f : ri;
  const float r6 = ri * ri * ri;
  const float t = __fmaf_rn(12.0f, r6, -6.0f);
  const float s = r6 * ri * t;
  fx = __fmaf_rn(s, dx, fx);
  fy = __fmaf_rn(s, dy, fy);
  fz = __fmaf_rn(s, dz, fz);
  pa = __fmaf_rn(r6, r6, pa);
  pb += r6;
}

// Packed FP32x2 arithmetic (PTX .f32x2, sm_100 and later): one instruction
// applies the operation to two independent FP32 values held in a 64-bit
// register pair.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk2(f32x2 r, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Two pairs (i, j0) and (i, j1) as the two lanes of FP32x2 operations (qi in
// slots 1..3): the
// same arithmetic as pair_mixed per lane, with half the instructions after
// the int -> float conversions.  The accumulators hold the j0 and j1 partial
// sums in their two lanes.
// On GB300 an FP32x2 instruction occupies both FMA sub-pipes (heavy and
// lite) for two cycles, so the FP32 throughput is that of two FFMAs; what it
// saves is issue slots.  The scalar loop issued ~23.7 warp-instructions per
// 32 pairs at 84% issue utilisation with the FMA pipes 64% busy; this one
// issues ~16.8 (ncu: 1.41e8 vs 1.98e8 per N=16384 launch) and ran 4.5%
// faster in the same step.  It needs ~80 registers, hence 6 (128-thread) or
// 3 (256-thread) resident CTAs per SM, and the integer differences stay on
// the ALU pipe, which has room here.
template <bool MASKED>
__device__ __forceinline__ void pair_mixed2(const int4 qi, const int4 qa, const int4 qb, f32x2 k2inv2, bool exa,
                                            bool exb, f32x2& fx, f32x2& fy, f32x2& fz, f32x2& pa, f32x2& pb) {
  const f32x2 dx = pk2(__int2float_rn(fixed_diff(qi.y, qa.x)), __int2float_rn(fixed_diff(qi.y, qb.x)));
  const f32x2 dy = pk2(__int2float_rn(fixed_diff(qi.z, qa.y)), __int2float_rn(fixed_diff(qi.z, qb.y)));
  const f32x2 dz = pk2(__int2float_rn(fixed_diff(qi.w, qa.z)), __int2float_rn(fixed_diff(qi.w, qb.z)));
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
  fx = fma2(sf, dx, fx);
  fy = fma2(sf, dy, fy);
  fz = fma2(sf, dz, fz);
  pa = fma2(r6, r6, pa);
  pb = add2(pb, r6);
}

__device__ __forceinline__ float lane_sum(f32x2 v) {
  float a, b;
  upk2(v, a, b);
  return a + b;
}

__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// two_sum_add of both lanes.
struct Float2Acc {
  f32x2 hi, lo;
};
__device__ __forceinline__ void two_sum_add2(Float2Acc& a, f32x2 t) {
  const f32x2 s = add2(a.hi, t);
  const f32x2 bp = sub2(s, a.hi);
  const f32x2 e = add2(sub2(a.hi, sub2(s, bp)), sub2(t, bp));
  a.hi = s;
  a.lo = add2(a.lo, e);
}

// Lanes with `second` keep b and give a to the lane `bit` away, the others keep a
// and give b; returns what is kept plus what the other lane gives.
__device__ __forceinline__ FloatAcc exchange1(const FloatAcc a, const FloatAcc b, bool second, int bit) {
  FloatAcc keep;
  keep.hi = second ? b.hi : a.hi;
  keep.lo = second ? b.lo : a.lo;
  const float hi = __shfl_xor_sync(0xffffffffu, second ? a.hi : b.hi, bit);
  const float lo = __shfl_xor_sync(0xffffffffu, second ? a.lo : b.lo, bit);
  two_sum_add(keep, hi);
  keep.lo = __fadd_rn(keep.lo, lo);
  return keep;
}

// pair_mixed2 with the two lanes on two i's (qa, qb in slots 1..3) against one
// j: the same arithmetic per lane.
template <bool MASKED>
__device__ __forceinline__ void pair_mixed_rows(const int4 qa, const int4 qb, const int4 qj, f32x2 k2inv2, bool exa,
                                                bool exb, f32x2& fx, f32x2& fy, f32x2& fz, f32x2& pa, f32x2& pb) {
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
  fx = fma2(sf, dx, fx);
  fy = fma2(sf, dy, fy);
  fz = fma2(sf, dz, fz);
  pa = fma2(r6, r6, pa);
  pb = add2(pb, r6);
}

}  // namespace ljgb
