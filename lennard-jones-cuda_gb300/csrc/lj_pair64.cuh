// lj_pair64.cuh -- FP64 building blocks of the pair kernels that evaluate
// every unordered pair once (lj_pairs64.cu, lj_adjoint.cu).
//
// FP64 issues at 1/64 of the FP32 rate on this part (2 lanes a clock and SM):
// one FP64 warp instruction takes the time of 16 others on every scheduler,
// so these kernels are written to the count of FP64 operations, and spend
// integer, FP32 and shuffle instructions freely to lower it.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ljgb {

// Nearest image of a separation d (every lane of a warp calls) in a period L,
// per component d - L k with k = d / L rounded, as fma(-L, round(d invL), d) gives it, bit for bit.  lo / hi are
// the bits of the smallest non-negative separations whose d invL, rounded to
// a double, reaches |k| = 1 and |k| = 2 (image_bounds): a multiplication by a
// positive constant is monotonic, so comparing |d| with them decides k
// without the product and the rounding, and one subtraction is left of about
// four FP64 operations.
struct ImageBounds {
  long long lo, hi;
};

// |x| >= the non-negative double of bits `bound`, x in words hi, lo.
__device__ __forceinline__ bool magnitude_reaches(int hi, int lo, long long bound) {
  const int m = hi & 0x7fffffff, bh = (int)(bound >> 32);
  return m > bh || (m == bh && (unsigned)lo >= (unsigned)bound);
}

template <bool TIES_AWAY>
__device__ __forceinline__ void nearest_image(double (&d)[3], double L, double invL, ImageBounds b) {
  // 32-bit words throughout: a 64-bit mask of the sign was recognised as fabs
  // and issued on the FP64 pipe
  int hi[3], lo[3];
  bool beyond = false;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    hi[c] = __double2hiint(d[c]);
    lo[c] = __double2loint(d[c]);
    beyond |= magnitude_reaches(hi[c], lo[c], b.hi);
  }
  // particles far outside the box: a vote, since a branch on the lane's own
  // flag was turned into selects and both sides' FP64 operations executed
  if (__any_sync(0xffffffffu, beyond)) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double t = d[c];
      asm volatile("" : "+d"(t));  // keeps the products below inside the branch
      d[c] = fma(-L, TIES_AWAY ? round(t * invL) : rint(t * invL), t);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const bool turn = magnitude_reaches(hi[c], lo[c], b.lo);
      const double k = __hiloint2double(turn ? __double2hiint(L) | (hi[c] & (int)0x80000000) : 0,
                                        turn ? __double2loint(L) : 0);
      d[c] -= k;
    }
  }
}

// Bounds of nearest_image for the rule round-half-away (ties_away) or
// round-half-even: half away turns to k = 1 at d invL >= 1/2, half even above
// 1/2; both turn to 2 at 3/2.
inline ImageBounds image_bounds(double L, double invL, bool ties_away);

// Seed of 1 / r2 from FP32's approximate reciprocal of the mantissa, the
// exponent set with integer operations (a conversion of r2 to FP32 would
// issue on the FP64 pipe and lose its range): relative error below 2^-21.
__device__ __forceinline__ double rcp_seed(double r2) {
  const int hi = __double2hiint(r2), lo = __double2loint(r2);
  const float m = __int_as_float(0x3f800000 | ((hi & 0xfffff) << 3) | (int)((unsigned)lo >> 29));
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(m));
  const int yb = __float_as_int(y);
  return __hiloint2double((yb >> 3) + 0x38000000 + 0x3ff00000 - (hi & 0x7ff00000), yb << 29);
}

// r2 whose reciprocal the seed's exponent cannot hold (above 2^1021, infinity
// included): no contribution, as s2 / r2 vanishes in the powers taken of it.
__device__ __forceinline__ bool beyond_seed(double r2) {
  const long long bits = __double_as_longlong(r2);  // integer tests: a comparison would issue on the FP64 pipe
  return bits >= 0x7fd0000000000000ll && bits <= 0x7ff0000000000000ll;
}

// 1 / r2 from its seed by the cubic member of Householder's iteration,
// y (1 + e + e^2) with e = 1 - r2 y: three operations, error 2^-63 before the
// last rounding.  A seed of 0 gives 0.
__device__ __forceinline__ double rcp_from_seed(double r2, double y) {
  const double e = fma(-r2, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// s2 / r2 from the seed of 1 / r2: one Newton step, the quotient, and
// Markstein's correction of it by its exact residual (P. Markstein, IBM J.
// Res. Dev. 34, 1990), which leaves the rounding of a division.
__device__ __forceinline__ double div_from_seed(double s2, double r2, double y) {
  const double y1 = fma(y, fma(-r2, y, 1.0), y);
  const double q = s2 * y1;
  return fma(fma(-r2, q, s2), y1, q);
}

__device__ __forceinline__ double shfl_next(double v, int lane) { return __shfl_sync(0xffffffffu, v, (lane + 1) & 31); }

inline ImageBounds image_bounds(double L, double invL, bool ties_away) {
  // the smallest double d >= 0 with d invL >= t (or > t), by bisection on the
  // bits: non-negative doubles order like their bits
  auto first = [&](double t, bool strict) {
    long long lo = 0, hi = 0x7ff0000000000000ll;
    while (lo < hi) {
      const long long mid = lo + (hi - lo) / 2;
      double d;
      __builtin_memcpy(&d, &mid, sizeof(d));
      const double p = d * invL;
      if (strict ? p > t : p >= t) hi = mid;
      else lo = mid + 1;
    }
    return lo;
  };
  return ImageBounds{first(0.5, !ties_away), first(1.5, false)};
}

}  // namespace ljgb
