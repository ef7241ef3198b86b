// lj_adjoint.cu -- differentiable MD: gradients of a time-averaged loss of
// the EVN velocity-Verlet trajectory with respect to eps, sigma and the
// initial positions / velocities, by a discrete adjoint.
//
// The reference has no adjoint.  The dynamics differentiated are its EVN
// step (src/library/MDSystem.cpp:443-463, periodic boundaries :406-436) with
// all-pairs minimum-image forces, generalised from the hard-coded
// eps = sigma = 1 (MDSystem.cu:44-53, MDSystem.cpp:289-298) to explicit
// 4 eps [(sigma/r)^12 - (sigma/r)^6].  Everything is FP64: the gradients are
// checked against central finite differences of this same forward pass.
//
//   loss = (1/S) sum_{m=1..S} [ wK K_m/N + wV V_m/N + wP P_m ]
//
// Forward: S steps from (x_0, v_0), keeping (x, v, F) every k steps.
// Backward: segments of k steps from the last checkpoint down; each segment
// is replayed forward (bit-identical kernels) into a (k+1)-state buffer, then
// swept in reverse.  With Xb_{S+1} = bb_{S+1} = 0, for m = S..0:
//   bb_m = dl_m/dv_m + dt Xb_{m+1} + bb_{m+1}
//   z_m  = dt^2/2 Xb_{m+1} + dt/2 bb_{m+1} (+ dt/2 bb_m for m > 0)
//   Xb_m = dl_m/dx_m + Xb_{m+1} + H(x_m) z_m,   H = dF/dx (symmetric)
//   d/d(eps, sigma) += G(x_m)^T z_m + dl_m/d(eps, sigma),  G = dF/d(eps, sigma)
// dloss/dx_0 = Xb_0, dloss/dv_0 = bb_0.  One pair pass per reverse step
// gives dl_m/dx_m + H z and the sums G^T z, V, W and dW/dsigma at x_m.
//
// Two launches a step either way: the pair pass, and one that sums its parts
// and does all of the per-particle work up to the next pass (forward: kick,
// states kept, drift; reverse: Xb_m, then z_{m-1}).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <string>
#include <vector>

#include "lj_device.cuh"
#include "lj_gb300.h"
#include "lj_init.h"
#include "lj_pair64.cuh"
#include "lj_schedule.h"

namespace ljgb {
namespace {

constexpr int kScalars = 5;  // sums over pairs of a task: e, u, then (reverse) u_sigma, z.F, z.dF/dsigma

struct AdjBox {
  int n, npad;
  double L, invL;
  double eps4, sigma2, inv_sigma;
  ImageBounds ib;  // round-half-even images
};

// The pair pass's work split (Pair64Plan of one box) and sums.
struct AdjPass {
  const Pair64Task* tasks;
  int ntasks, tiles, groups, group, parts, split, turns;  // turns = 32 / split
  double* part;  // [tile][(groups + 1) split][3][32]: F (forward), or dl/dx + H z
  double* scal;  // [task][kScalars]
};

struct AdjSums {
  double x, y, z;
};

// Pairs of tiles ta and tb, turns r0 .. r1-1, as in lj_pairs64.cu: lane = i,
// positions (and z) and sums of the j's move around the warp, so each pair is
// evaluated once for both particles.  Per pair, with s6 = (sigma^2/r^2)^3 and
// c = 4 eps s6 / r^2 (one factor of all three):
//   f = g d,  g = c (12 s6 - 6)
//   dg/dsigma = gs / sigma,  gs = c (144 s6 - 36)
//   H z: J (z_i - z_j),  J = g I + h d d^T,  h = c / r^2 (-168 s6 + 48)
// The reverse step needs F and dF/dsigma only in dl/dx = cF F + cA dF/dsigma
// and in the sums z.F and z.dF/dsigma, which over unordered pairs are those
// of g d.dz and gs d.dz: six vector sums a pair are left of eighteen.
// FP64 operations an unordered pair: 30 forward, 55 reverse (of 2 x 36 and
// 2 x 66 over ordered pairs with an IEEE division).
template <bool HVP, bool UNIT>
__device__ __forceinline__ int adj_turns(const AdjBox& b, const double* x, const double* z, double cF, double cA,
                                         int ta, int tb, int r0, int r1, const double (&xi)[3], const double (&zi)[3],
                                         AdjSums& I, AdjSums& J, double (&S)[kScalars]) {
  const int lane = threadIdx.x & 31;
  const bool vi = ta * 32 + lane < b.n, diag = ta == tb;
  int jl = (lane + r0) & 31;
  const int j = min(tb * 32 + jl, b.n - 1);
  double xj[3], zj[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    xj[c] = x[(size_t)c * b.npad + j];
    if (HVP) zj[c] = z[(size_t)c * b.npad + j];
  }
  __builtin_assume((r1 - r0) % 2 == 0);  // Pair64Plan::parts sees to it
#pragma unroll 2
  for (int r = r0; r < r1; ++r) {
    double d[3] = {xi[0] - xj[0], xi[1] - xj[1], xi[2] - xj[2]};
    nearest_image<false>(d, b.L, b.invL, b.ib);
    double r2 = fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0]));
    double y = rcp_seed(r2);
    const bool meets = vi && tb * 32 + jl < b.n && !(diag && r == 16 && lane >= 16);
    if (!meets || beyond_seed(r2)) {  // a seed of 0 makes the pair's terms 0
      r2 = 1.0;
      y = 0.0;
    }
    const double inv = rcp_from_seed(r2, y);
    const double s2 = UNIT ? inv : b.sigma2 * inv;
    const double s6 = s2 * s2 * s2;
    const double c = b.eps4 * inv * s6;
    const double t = fma(12.0, s6, -6.0);
    const double g = c * t;
    S[0] = fma(s6, s6 - 1.0, S[0]);
    S[1] = fma(s6, t, S[1]);
    double k = g;  // factor of d in i's sums
    double gz[3] = {0.0, 0.0, 0.0};
    if (HVP) {
      const double ts = fma(144.0, s6, -36.0);
      const double gs = c * ts;
      const double h = c * inv * fma(-168.0, s6, 48.0);
      double dz[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) dz[q] = zi[q] - zj[q];
      const double dot = fma(d[2], dz[2], fma(d[1], dz[1], d[0] * dz[0]));
      S[2] = fma(s6, ts, S[2]);
      S[3] = fma(g, dot, S[3]);
      S[4] = fma(gs, dot, S[4]);
      k = fma(cF, g, fma(cA, gs, h * dot));
#pragma unroll
      for (int q = 0; q < 3; ++q) gz[q] = dz[q];
    }
    if (HVP) {
      I.x = fma(g, gz[0], fma(k, d[0], I.x));
      I.y = fma(g, gz[1], fma(k, d[1], I.y));
      I.z = fma(g, gz[2], fma(k, d[2], I.z));
      J.x = shfl_next(fma(-g, gz[0], fma(-k, d[0], J.x)), lane);
      J.y = shfl_next(fma(-g, gz[1], fma(-k, d[1], J.y)), lane);
      J.z = shfl_next(fma(-g, gz[2], fma(-k, d[2], J.z)), lane);
    } else {
      I.x = fma(k, d[0], I.x);
      I.y = fma(k, d[1], I.y);
      I.z = fma(k, d[2], I.z);
      J.x = shfl_next(fma(-k, d[0], J.x), lane);
      J.y = shfl_next(fma(-k, d[1], J.y), lane);
      J.z = shfl_next(fma(-k, d[2], J.z), lane);
    }
    jl = (jl + 1) & 31;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      xj[q] = shfl_next(xj[q], lane);
      if (HVP) zj[q] = shfl_next(zj[q], lane);
    }
  }
  return jl;
}

__device__ __forceinline__ void store_adj(double* to, int at, const AdjSums& s) {
  to[at] = s.x;
  to[32 + at] = s.y;
  to[64 + at] = s.z;
}

// One task: a square of tiles by one warp, or of one tile by `parts` warps.
template <bool HVP, bool UNIT>
__device__ __forceinline__ void adj_task(const AdjBox& b, const AdjPass& a, const double* x, const double* z,
                                         double cF, double cA, const Pair64Task tk, double* sh) {
  const int lane = threadIdx.x & 31;
  const int slots = (a.groups + 1) * a.split;
  constexpr int kS = HVP ? kScalars : 2;
  double S[kScalars] = {0.0, 0.0, 0.0, 0.0, 0.0};
  auto load = [&](const double* from, int t, double (&to)[3]) {
    const int i = min(t * 32 + lane, b.n - 1);
#pragma unroll
    for (int c = 0; c < 3; ++c) to[c] = from[(size_t)c * b.npad + i];
  };
  double xi[3], zi[3] = {0.0, 0.0, 0.0};
  if (a.parts > 1) {
    const int w = threadIdx.x >> 5, ta = tk.ga, tb = tk.gb;
    const int turns = (ta == tb ? min(16, a.turns) : a.turns) / a.parts;
    const int first = (ta == tb ? 1 : 0) + a.turns * tk.slot;
    load(x, ta, xi);
    if (HVP) load(z, ta, zi);
    AdjSums I{}, J{};
    const int jl =
        adj_turns<HVP, UNIT>(b, x, z, cF, cA, ta, tb, first + w * turns, first + (w + 1) * turns, xi, zi, I, J, S);
    double* const mine = sh + w * (192 + kScalars);
    store_adj(mine, lane, I);
    store_adj(mine + 96, jl, J);
#pragma unroll
    for (int m = 0; m < kS; ++m) S[m] = warp_sum(S[m]);
    if (lane == 0)
#pragma unroll
      for (int m = 0; m < kS; ++m) mine[192 + m] = S[m];
    __syncthreads();
    for (int k = threadIdx.x; k < 192 + kS; k += blockDim.x) {
      double v = 0.0;
      for (int p = 0; p < a.parts; ++p) v += sh[p * (192 + kScalars) + k];
      if (k < 96) a.part[((size_t)ta * slots + (tb + 1) * a.split + tk.slot) * 96 + k] = v;
      else if (k < 192) a.part[((size_t)tb * slots + ta * a.split + tk.slot) * 96 + k - 96] = v;
      else a.scal[(size_t)blockIdx.x * kScalars + k - 192] = v;
    }
    return;
  }
  const int a0 = tk.ga * a.group, a1 = min(a.tiles, a0 + a.group);
  const int b0 = tk.gb * a.group, b1 = min(a.tiles, b0 + a.group);
  for (int ta = a0; ta < a1; ++ta) {
    load(x, ta, xi);
    if (HVP) load(z, ta, zi);
    AdjSums I{};
    for (int tb = max(ta, b0); tb < b1; ++tb) {
      const int r0 = (ta == tb ? 1 : 0) + a.turns * tk.slot, r1 = r0 + (ta == tb ? min(16, a.turns) : a.turns);
      double* const jslot = a.part + ((size_t)tb * slots + tk.ga * a.split + tk.slot) * 96;
      const int at = (lane + r0) & 31;
      AdjSums J{};
      if (ta > a0) J = AdjSums{jslot[at], jslot[32 + at], jslot[64 + at]};  // earlier rows' sums
      const int jl = adj_turns<HVP, UNIT>(b, x, z, cF, cA, ta, tb, r0, r1, xi, zi, I, J, S);
      store_adj(jslot, jl, J);
      __syncwarp();
    }
    store_adj(a.part + ((size_t)ta * slots + (tk.gb + 1) * a.split + tk.slot) * 96, lane, I);
  }
#pragma unroll
  for (int m = 0; m < kS; ++m) S[m] = warp_sum(S[m]);
  if (lane == 0)
#pragma unroll
    for (int m = 0; m < kS; ++m) a.scal[(size_t)blockIdx.x * kScalars + m] = S[m];
}

// FP64-pipe bound.  N = 1000: 34 us forward, 60 us reverse (79 and 142 over
// ordered pairs).
// x and z are written by the launch before, which this one may overlap until the
// wait: no __restrict__, whose promise of data that stays constant for the whole
// kernel would let them be read through the non-coherent path.
template <bool HVP>
__global__ void __launch_bounds__(256) k_adj_pairs(AdjBox b, AdjPass a, const double* x, const double* z, double cF,
                                                   double cA) {
  extern __shared__ double sh[];  // parts > 1: parts x (2 x 3 x 32 + kScalars)
  const Pair64Task tk = a.tasks[blockIdx.x];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (b.sigma2 == 1.0) adj_task<HVP, true>(b, a, x, z, cF, cA, tk, sh);
  else adj_task<HVP, false>(b, a, x, z, cF, cA, tk, sh);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// CTA of one tile for the per-particle kernels below: 12 warps sum its slots
// (component c by four warps, a quarter of the slots each), a 13th sums this
// tile's share of the tasks' scalars; then warp c holds component c of the
// tile's particles.  Fixed order throughout.  (One CTA of 128 particles and
// a thread per particle summed 12 values of 32 parts serially: 97 us at
// N = 1000.)
constexpr int kSumWarps = 4;
constexpr int kAdjTileThreads = 32 * (3 * kSumWarps + 1);

template <int NS>
__device__ __forceinline__ double adj_tile_sums(const AdjPass& a, double (&scal)[NS], bool* mine) {
  __shared__ double sum[3 * kSumWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = blockIdx.x;
  if (warp < 3 * kSumWarps) {
    const int c = warp % 3, u = warp / 3, slots = (a.groups + 1) * a.split;
    const double* p = a.part + (size_t)t * slots * 96 + c * 32 + lane;
    double q0 = 0.0, q1 = 0.0;
    for (int k = u; k < slots; k += 8 * kSumWarps) {
      double v[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) v[m] = k + m * kSumWarps < slots ? p[(size_t)(k + m * kSumWarps) * 96] : 0.0;
      q0 += (v[0] + v[2]) + (v[4] + v[6]);
      q1 += (v[1] + v[3]) + (v[5] + v[7]);
    }
    sum[warp][lane] = q0 + q1;
  } else {
    for (int k = t + lane * a.tiles; k < a.ntasks; k += 32 * a.tiles)
#pragma unroll
      for (int m = 0; m < NS; ++m) scal[m] += a.scal[(size_t)k * kScalars + m];
#pragma unroll
    for (int m = 0; m < NS; ++m) scal[m] = warp_sum(scal[m]);
  }
  __syncthreads();
  *mine = warp < 3;
  if (warp >= 3) return 0.0;
  return (sum[warp][lane] + sum[warp + 3][lane]) + (sum[warp + 6][lane] + sum[warp + 9][lane]);
}

// x + dt v + dt^2 F / 2 with a single +-L wrap, and v + dt F / 2.
__device__ __forceinline__ void adj_drift1(const AdjBox& b, double& x, double& v, double f, double dt) {
  x = fma(0.5 * dt * dt, f, fma(dt, v, x));
  if (x < 0.) x += b.L;
  if (x > b.L) x -= b.L;
  v = fma(0.5 * dt, f, v);
}

// Where a state is kept: x, v, f (any may be null).
struct AdjKeep {
  double *x, *v, *f;
};

// F of the current positions; with kick, v += dt F / 2.  The finished state
// goes to `keep` and `keep2`; with drift, x and v become those half a step on.
// Block partials (K, V, W) into blk[tile * 3 + 0..2] when blk is non-null.
__global__ void __launch_bounds__(kAdjTileThreads) k_adj_forces(AdjBox b, AdjPass a, double* x, double* v, double dt,
                                                                int kick, int drift, AdjKeep keep, AdjKeep keep2,
                                                                double* blk) {
  __shared__ double ksum[3];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  double scal[2] = {0.0, 0.0};
  bool mine;
  const double F = adj_tile_sums<2>(a, scal, &mine);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * 32 + lane;
  double vv = 0.0;
  if (mine && i < b.n) {
    const size_t k = (size_t)warp * b.npad + i;
    double xc = x[k], vc = v[k];
    if (kick) vc = fma(0.5 * dt, F, vc);
    vv = vc * vc;
    if (keep.x) keep.x[k] = xc;
    if (keep.v) keep.v[k] = vc;
    if (keep.f) keep.f[k] = F;
    if (keep2.x) keep2.x[k] = xc;
    if (keep2.v) keep2.v[k] = vc;
    if (drift) {
      adj_drift1(b, xc, vc, F, dt);
      x[k] = xc;
    }
    v[k] = vc;
  }
  if (!blk) return;
  if (mine) {
    vv = warp_sum(vv);
    if (lane == 0) ksum[warp] = vv;
  }
  __syncthreads();
  if (warp == 3 * kSumWarps && lane == 0) {
    double* const o = blk + (size_t)blockIdx.x * 3;
    o[0] = 0.5 * (ksum[0] + ksum[1] + ksum[2]);
    o[1] = b.eps4 * scal[0];        // V: each unordered pair once
    o[2] = 2.0 * (b.eps4 * scal[1]);  // W: ordered pairs
  }
}

// A replay's start from a checkpoint: the state into `keep`, x and v half a
// step on.
__global__ void k_adj_start(AdjBox b, const double* ckpt, size_t s3, double* x, double* v, double dt, AdjKeep keep) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 3 * b.npad || k % b.npad >= b.n) return;
  double xc = ckpt[k], vc = ckpt[s3 + k];
  keep.x[k] = xc;
  keep.v[k] = vc;
  adj_drift1(b, xc, vc, ckpt[2 * s3 + k], dt);
  x[k] = xc;
  v[k] = vc;
}

// Reverse step m, first half, one component: bb_m and z_m from Xb_{m+1} = X
// and bb_{m+1}.  cv = dl_m/dv_m / v_m (0 for m = 0); first = (m == 0).
__device__ __forceinline__ void adj_prep1(double X, double vm, double cv, double dt, int first, double* bb,
                                          double* z) {
  const double bn = *bb;
  const double bm = fma(dt, X, fma(cv, vm, bn));
  const double y = fma(0.5 * dt * dt, X, 0.5 * dt * bn);
  *z = first ? y : fma(0.5 * dt, bm, y);
  *bb = bm;
}

__global__ void k_adj_prep(AdjBox b, const double* vm, const double* Xb, double* bb, double* z, double cv, double dt) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 3 * b.npad || k % b.npad >= b.n) return;
  adj_prep1(Xb[k], vm[k], cv, dt, 0, bb + k, z + k);
}

// Reverse step m, second half: Xb <- dl_m/dx_m + Xb + H z (the pass's sums),
// then, for m > 0 (vm non-null), the first half of step m - 1 with its v.
// Block partials (z.F, z.dF/dsigma, V, W, dW/dsigma) into blk[tile * 5 + 0..4].
__global__ void __launch_bounds__(kAdjTileThreads) k_adj_finish(AdjBox b, AdjPass a, const double* vm, double* Xb,
                                                                double* bb, double* z, double cv, double dt,
                                                                int first, double* blk) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  double scal[kScalars] = {0.0, 0.0, 0.0, 0.0, 0.0};
  bool mine;
  const double H = adj_tile_sums<kScalars>(a, scal, &mine);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * 32 + lane;
  if (mine && i < b.n) {
    const size_t k = (size_t)warp * b.npad + i;
    const double X = Xb[k] + H;
    Xb[k] = X;
    if (vm) adj_prep1(X, vm[k], cv, dt, first, bb + k, z + k);
  }
  if (warp == 3 * kSumWarps && lane == 0) {
    double* const o = blk + (size_t)blockIdx.x * 5;
    o[0] = scal[3];
    o[1] = b.inv_sigma * scal[4];
    o[2] = b.eps4 * scal[0];
    o[3] = 2.0 * (b.eps4 * scal[1]);
    o[4] = 2.0 * (b.eps4 * b.inv_sigma * scal[2]);
  }
}

// (N x 3 interleaved) <-> component-major device layout.
__global__ void k_adj_unpack(int n, int npad, const double* in, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int c = 0; c < 3; ++c) out[(size_t)c * npad + i] = in[(size_t)i * 3 + c];
}
__global__ void k_adj_pack(int n, int npad, const double* in, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int c = 0; c < 3; ++c) out[(size_t)i * 3 + c] = in[(size_t)c * npad + i];
}

template <typename T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  cudaError_t alloc(size_t count) {
    if (count <= n && p) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
    void* q = nullptr;
    cudaError_t e = device_alloc(&q, sizeof(T) * (count ? count : 1));
    if (e == cudaSuccess) {
      p = static_cast<T*>(q);
      n = count;
    }
    return e;
  }
  void free() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
};

}  // namespace
}  // namespace ljgb

using namespace ljgb;

struct lj_adjoint {
  int device = 0;
  int n = 0, npad = 0;
  AdjBox box{};
  AdjPass pass{};
  double rho = 0, eps = 1, sigma = 1;
  double wK = 0.0, wV = 1.0, wP = 1.0;
  int every = 20;
  cudaStream_t stream = nullptr;
  DBuf<double> x, v, x0, v0, part, scal, ckpt, seg, Xb, bb, z, blk, hostio;
  DBuf<Pair64Task> tasks;
  // last forward
  bool have_forward = false;
  int seg_in_hand = -1;  // segment whose states `seg` holds (the forward pass leaves its last one there)
  double dt = 0.0;
  int S = 0;
  double loss = 0.0;
  std::vector<double> K, V, W;
  std::string err;
};

namespace {

lj_status afail(lj_adjoint* a, lj_status code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  std::vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (a) a->err = buf;
  return code;
}

#define ADJ_CUDA(a, call)                                                                           \
  do {                                                                                              \
    cudaError_t e_ = (call);                                                                        \
    if (e_ != cudaSuccess)                                                                          \
      return afail((a), e_ == cudaErrorMemoryAllocation ? LJ_ERR_OUT_OF_MEMORY : LJ_ERR_CUDA, "%s: %s", \
                   #call, cudaGetErrorString(e_));                                                  \
  } while (0)

size_t xyz(const lj_adjoint* a) { return (size_t)3 * a->npad; }

// The pair pass at positions x: forces, or (z non-null) the reverse step's.
lj_status adj_pairs(lj_adjoint* a, const double* x, const double* z, double cF, double cA) {
  const AdjPass& p = a->pass;
  const size_t smem = p.parts > 1 ? sizeof(double) * (192 + kScalars) * p.parts : 0;
  ADJ_CUDA(a, launch_dependent(z ? k_adj_pairs<true> : k_adj_pairs<false>, p.ntasks, 32 * p.parts, smem, a->stream,
                               a->box, p, x, z, cF, cA));
  return LJ_OK;
}

// F at the current positions and what follows it (k_adj_forces).
lj_status adj_forces(lj_adjoint* a, bool kick, bool drift, AdjKeep keep, AdjKeep keep2, double* blk) {
  lj_status st = adj_pairs(a, a->x.p, nullptr, 0.0, 0.0);
  if (st) return st;
  ADJ_CUDA(a, launch_dependent(k_adj_forces, a->pass.tiles, kAdjTileThreads, 0, a->stream, a->box, a->pass, a->x.p,
                               a->v.p, a->dt, kick ? 1 : 0, drift ? 1 : 0, keep, keep2, blk));
  return LJ_OK;
}

lj_status adj_copy(lj_adjoint* a, double* dst, const double* src, size_t count) {
  ADJ_CUDA(a, cudaMemcpyAsync(dst, src, sizeof(double) * count, cudaMemcpyDeviceToDevice, a->stream));
  return LJ_OK;
}

}  // namespace

extern "C" {

lj_status lj_adjoint_create(const lj_config* cfg, int32_t checkpoint_every, lj_adjoint** out) {
  if (!out) return LJ_ERR_INVALID;
  *out = nullptr;
  if (!cfg) return LJ_ERR_INVALID;
  if (cfg->n < 2 || !(cfg->density > 0) || !(cfg->epsilon > 0) || !(cfg->sigma > 0) || !(cfg->temperature >= 0))
    return LJ_ERR_INVALID;
  if (cfg->boundary != LJ_BC_PERIODIC || cfg->canonical) return LJ_ERR_UNSUPPORTED;
  if (checkpoint_every < 1) return LJ_ERR_INVALID;
  lj_adjoint* a = new lj_adjoint();
  a->device = cfg->device;
  a->n = cfg->n;
  a->npad = (cfg->n + 31) / 32 * 32;
  a->rho = cfg->density;
  a->eps = cfg->epsilon;
  a->sigma = cfg->sigma;
  a->every = checkpoint_every;
  const double L = std::cbrt((double)cfg->n / cfg->density);
  a->box = AdjBox{cfg->n, a->npad, L, 1.0 / L, 4.0 * cfg->epsilon, cfg->sigma * cfg->sigma, 1.0 / cfg->sigma,
                  image_bounds(L, 1.0 / L, false)};
  auto bail = [&](lj_status st) {
    lj_adjoint_destroy(a);
    return st;
  };
  DeviceGuard device_guard(a->device);
  if (!device_guard.ok()) return bail(LJ_ERR_NO_DEVICE);
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, a->device) != cudaSuccess)
    return bail(LJ_ERR_NO_DEVICE);
  if (cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking) != cudaSuccess) return bail(LJ_ERR_CUDA);
  const size_t s3 = xyz(a);
  Pair64Plan plan;  // of 30 and 55 operations a turn
  const cudaError_t sums = plan_pairs64_within({a->n}, sms, 41, 3, 3, &plan, [&](const Pair64Plan& p) {
    return a->part.alloc((size_t)p.slots * 96);
  });
  if (sums != cudaSuccess) return bail(sums == cudaErrorMemoryAllocation ? LJ_ERR_OUT_OF_MEMORY : LJ_ERR_CUDA);
  if (a->x.alloc(s3) || a->v.alloc(s3) || a->x0.alloc(s3) || a->v0.alloc(s3) || a->Xb.alloc(s3) ||
      a->bb.alloc(s3) || a->z.alloc(s3) || a->hostio.alloc(s3) ||
      a->scal.alloc(plan.tasks.size() * kScalars) || a->tasks.alloc(plan.tasks.size()))
    return bail(LJ_ERR_OUT_OF_MEMORY);
  if (cudaMemsetAsync(a->part.p, 0, sizeof(double) * (size_t)plan.slots * 96, a->stream) != cudaSuccess)
    return bail(LJ_ERR_CUDA);
  if (cudaMemcpyAsync(a->tasks.p, plan.tasks.data(), sizeof(Pair64Task) * plan.tasks.size(), cudaMemcpyHostToDevice,
                      a->stream) != cudaSuccess)
    return bail(LJ_ERR_CUDA);
  a->pass = AdjPass{a->tasks.p, (int)plan.tasks.size(), plan.boxes[0].tiles, plan.boxes[0].groups, plan.group,
                    plan.parts, plan.split, 32 / plan.split, a->part.p, a->scal.p};
  std::vector<double> pos((size_t)3 * a->n), vel((size_t)3 * a->n);
  if (!sample_initial_state(a->n, L, cfg->temperature, cfg->lattice, cfg->jitter, cfg->sigma, cfg->seed, pos.data(),
                            vel.data()))
    return bail(LJ_ERR_INVALID);
  lj_status st = lj_adjoint_set_state(a, pos.data(), vel.data());
  if (st) return bail(st);
  *out = a;
  return LJ_OK;
}

lj_status lj_adjoint_destroy(lj_adjoint* a) {
  if (!a) return LJ_OK;
  DeviceGuard device_guard(a->device);
  if (a->stream) cudaStreamSynchronize(a->stream);
  for (DBuf<double>* b : {&a->x, &a->v, &a->x0, &a->v0, &a->part, &a->scal, &a->ckpt, &a->seg, &a->Xb, &a->bb, &a->z,
                          &a->blk, &a->hostio})
    b->free();
  a->tasks.free();
  if (a->stream) cudaStreamDestroy(a->stream);
  delete a;
  return LJ_OK;
}

const char* lj_adjoint_last_error(const lj_adjoint* a) { return a ? a->err.c_str() : ""; }

lj_status lj_adjoint_set_state(lj_adjoint* a, const double* pos, const double* vel) {
  if (!a) return LJ_ERR_INVALID;
  if (!pos || !vel) return afail(a, LJ_ERR_INVALID, "pos and vel must be non-NULL");
  DeviceGuard device_guard(a->device);
  const size_t bytes = sizeof(double) * 3 * a->n;
  const int g = (a->n + 255) / 256;
  ADJ_CUDA(a, cudaMemcpyAsync(a->hostio.p, pos, bytes, cudaMemcpyHostToDevice, a->stream));
  k_adj_unpack<<<g, 256, 0, a->stream>>>(a->n, a->npad, a->hostio.p, a->x0.p);
  ADJ_CUDA(a, cudaStreamSynchronize(a->stream));
  ADJ_CUDA(a, cudaMemcpyAsync(a->hostio.p, vel, bytes, cudaMemcpyHostToDevice, a->stream));
  k_adj_unpack<<<g, 256, 0, a->stream>>>(a->n, a->npad, a->hostio.p, a->v0.p);
  ADJ_CUDA(a, cudaStreamSynchronize(a->stream));
  a->have_forward = false;
  return LJ_OK;
}

lj_status lj_adjoint_set_loss(lj_adjoint* a, double w_kinetic, double w_potential, double w_pressure) {
  if (!a) return LJ_ERR_INVALID;
  if (!std::isfinite(w_kinetic) || !std::isfinite(w_potential) || !std::isfinite(w_pressure))
    return afail(a, LJ_ERR_INVALID, "loss weights must be finite");
  a->wK = w_kinetic;
  a->wV = w_potential;
  a->wP = w_pressure;
  a->have_forward = false;
  return LJ_OK;
}

lj_status lj_adjoint_forward(lj_adjoint* a, double dt, int32_t nsteps, double* loss) {
  if (!a) return LJ_ERR_INVALID;
  if (!(dt > 0) || !std::isfinite(dt)) return afail(a, LJ_ERR_INVALID, "dt must be > 0");
  if (nsteps < 1) return afail(a, LJ_ERR_INVALID, "nsteps must be >= 1");
  DeviceGuard device_guard(a->device);
  a->dt = dt;
  a->S = nsteps;
  a->have_forward = false;
  a->seg_in_hand = -1;
  const size_t s3 = xyz(a);
  const int J = (nsteps + a->every - 1) / a->every;
  const int nt = a->pass.tiles;
  if (a->ckpt.alloc((size_t)J * 3 * s3) || a->seg.alloc((size_t)(a->every + 1) * 2 * s3) ||
      a->blk.alloc((size_t)(nsteps + 1) * nt * 5))
    return afail(a, LJ_ERR_OUT_OF_MEMORY, "cannot allocate %d checkpoints of %d particles", J, a->n);
  lj_status st;
  if ((st = adj_copy(a, a->x.p, a->x0.p, s3)) || (st = adj_copy(a, a->v.p, a->v0.p, s3))) return st;
  // State m: the pass at x_m, then kick, what is kept of it (a checkpoint,
  // and the last segment's states, which the reverse sweep starts with), and
  // the drift to x_{m+1}.
  const int last0 = (J - 1) * a->every;
  for (int m = 0; m <= nsteps; ++m) {
    AdjKeep ck{}, sg{};
    if (m < nsteps && m % a->every == 0) {
      double* c = a->ckpt.p + (size_t)(m / a->every) * 3 * s3;
      ck = AdjKeep{c, c + s3, c + 2 * s3};
    }
    if (m >= last0) {
      double* sl = a->seg.p + (size_t)(m - last0) * 2 * s3;
      sg = AdjKeep{sl, sl + s3, nullptr};
    }
    double* const blk = m == 0 ? nullptr : a->blk.p + (size_t)(m - 1) * nt * 3;
    if ((st = adj_forces(a, m > 0, m < nsteps, ck, sg, blk))) return st;
  }
  std::vector<double> h((size_t)nsteps * nt * 3);
  ADJ_CUDA(a, cudaMemcpyAsync(h.data(), a->blk.p, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, a->stream));
  ADJ_CUDA(a, cudaStreamSynchronize(a->stream));
  const double N = (double)a->n;
  a->K.assign(nsteps, 0.0);
  a->V.assign(nsteps, 0.0);
  a->W.assign(nsteps, 0.0);
  double l = 0.0;
  for (int m = 0; m < nsteps; ++m) {
    double s[3] = {0.0, 0.0, 0.0};
    for (int b = 0; b < nt; ++b)
      for (int c = 0; c < 3; ++c) s[c] += h[((size_t)m * nt + b) * 3 + c];
    a->K[m] = s[0];
    a->V[m] = s[1];
    a->W[m] = s[2];
    const double T = 2. * s[0] / 3. / N;                // MDSystem.cpp:325-359
    const double P = (s[2] / 6. + N * T) / (N / a->rho);
    l += (a->wK * s[0] / N + a->wV * s[1] / N + a->wP * P) / nsteps;
  }
  if (!std::isfinite(l)) return afail(a, LJ_ERR_NONFINITE, "the loss is not finite");
  a->loss = l;
  a->have_forward = true;
  a->seg_in_hand = J - 1;
  if (loss) *loss = l;
  return LJ_OK;
}

lj_status lj_adjoint_observables(lj_adjoint* a, double* K, double* V, double* W, int32_t max, int32_t* count) {
  if (!a) return LJ_ERR_INVALID;
  if (!a->have_forward) return afail(a, LJ_ERR_INVALID, "no forward pass");
  const int m = std::min<int>(max, a->S);
  for (int k = 0; k < m; ++k) {
    if (K) K[k] = a->K[k];
    if (V) V[k] = a->V[k];
    if (W) W[k] = a->W[k];
  }
  if (count) *count = a->S;
  return LJ_OK;
}

lj_status lj_adjoint_backward(lj_adjoint* a, double* d_epsilon, double* d_sigma, double* d_pos, double* d_vel) {
  if (!a) return LJ_ERR_INVALID;
  if (!a->have_forward) return afail(a, LJ_ERR_INVALID, "lj_adjoint_backward needs a forward pass first");
  DeviceGuard device_guard(a->device);
  const size_t s3 = xyz(a);
  const int S = a->S, k = a->every, J = (S + k - 1) / k;
  const double N = (double)a->n, dt = a->dt, rho = a->rho;
  const double cv = (a->wK / N + a->wP * rho * 2.0 / (3.0 * N)) / S;  // dl_m/dv_m = cv v_m
  const double cF = -a->wV / N / S;                                    // dl_m/dx_m = cF F + cA dF/dsigma
  const double cA = a->wP * rho / (6.0 * N) * (-2.0 * a->sigma) / S;
  ADJ_CUDA(a, cudaMemsetAsync(a->Xb.p, 0, sizeof(double) * s3, a->stream));
  ADJ_CUDA(a, cudaMemsetAsync(a->bb.p, 0, sizeof(double) * s3, a->stream));
  lj_status st;
  const int nt = a->pass.tiles, grid3 = (3 * a->npad + 255) / 256;
  for (int j = J - 1; j >= 0; --j) {
    const int c0 = j * k, c1 = std::min(c0 + k, S);
    auto state = [&](int m) { return a->seg.p + (size_t)(m - c0) * 2 * s3; };
    if (a->seg_in_hand != j) {
      // replay the segment from its checkpoint (same kernels as the forward)
      a->seg_in_hand = -1;
      const double* c = a->ckpt.p + (size_t)j * 3 * s3;
      ADJ_CUDA(a, launch_dependent(k_adj_start, grid3, 256, 0, a->stream, a->box, c, s3, a->x.p, a->v.p, dt,
                                   AdjKeep{state(c0), state(c0) + s3, nullptr}));
      for (int m = c0 + 1; m <= c1; ++m)
        if ((st = adj_forces(a, true, m < c1, AdjKeep{state(m), state(m) + s3, nullptr}, AdjKeep{}, nullptr)))
          return st;
      a->seg_in_hand = j;
    }
    if (j == J - 1)
      ADJ_CUDA(a, launch_dependent(k_adj_prep, grid3, 256, 0, a->stream, a->box, (const double*)(state(S) + s3),
                                   (const double*)a->Xb.p, a->bb.p, a->z.p, cv, dt));
    // reverse sweep over m = c1 .. c0+1 (.. 0 in the first segment); state
    // c0 is the previous segment's last, and this one's checkpoint
    for (int m = c1; m >= (j == 0 ? 0 : c0 + 1); --m) {
      if ((st = adj_pairs(a, state(m), a->z.p, m >= 1 ? cF : 0.0, m >= 1 ? cA * a->box.inv_sigma : 0.0))) return st;
      const double* vm = m >= 1 ? state(m - 1) + s3 : nullptr;
      ADJ_CUDA(a, launch_dependent(k_adj_finish, nt, kAdjTileThreads, 0, a->stream, a->box, a->pass, vm, a->Xb.p,
                                   a->bb.p, a->z.p, m >= 2 ? cv : 0.0, dt, m == 1 ? 1 : 0,
                                   a->blk.p + (size_t)m * nt * 5));
    }
  }
  // parameter gradients: fixed-order sums of the block partials
  std::vector<double> h((size_t)(S + 1) * nt * 5);
  ADJ_CUDA(a, cudaMemcpyAsync(h.data(), a->blk.p, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, a->stream));
  double de = 0.0, ds = 0.0;
  for (int m = 0; m <= S; ++m) {
    double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int b = 0; b < nt; ++b)
      for (int q = 0; q < 5; ++q) s[q] += h[((size_t)m * nt + b) * 5 + q];
    de += s[0] / a->eps;  // G_eps^T z = z.F / eps
    ds += s[1];           // G_sigma^T z = z.dF/dsigma
    if (m >= 1) {         // explicit: dV/deps = V/eps, dV/dsigma = W/(2 sigma), dW/deps = W/eps
      de += (a->wV * s[2] / (N * a->eps) + a->wP * rho * s[3] / (6.0 * N * a->eps)) / S;
      ds += (a->wV * s[3] / (2.0 * a->sigma * N) + a->wP * rho * s[4] / (6.0 * N)) / S;
    }
  }
  if (d_epsilon) *d_epsilon = de;
  if (d_sigma) *d_sigma = ds;
  const int g = (a->n + 255) / 256;
  const size_t bytes = sizeof(double) * 3 * a->n;
  if (d_pos) {
    k_adj_pack<<<g, 256, 0, a->stream>>>(a->n, a->npad, a->Xb.p, a->hostio.p);
    ADJ_CUDA(a, cudaMemcpyAsync(d_pos, a->hostio.p, bytes, cudaMemcpyDeviceToHost, a->stream));
    ADJ_CUDA(a, cudaStreamSynchronize(a->stream));
  }
  if (d_vel) {
    k_adj_pack<<<g, 256, 0, a->stream>>>(a->n, a->npad, a->bb.p, a->hostio.p);
    ADJ_CUDA(a, cudaMemcpyAsync(d_vel, a->hostio.p, bytes, cudaMemcpyDeviceToHost, a->stream));
  }
  ADJ_CUDA(a, cudaStreamSynchronize(a->stream));
  if (!std::isfinite(de) || !std::isfinite(ds)) return afail(a, LJ_ERR_NONFINITE, "a gradient is not finite");
  return LJ_OK;
}

}  // extern "C"
