// lj_cluster.cu -- many MIXED steps of one small box in one launch: the box
// lives in a cluster of 16 CTAs.
//
// A step of a few hundred particles is a fraction of a microsecond of pair
// arithmetic; launched by itself (lj_rows.cu) it costs 5.5 us (EVN) or 8.3
// (TVN) in launch, first loads and drain.  Here 16 CTAs on 16 SMs keep the
// state on chip for all steps of an lj_step call: every CTA holds the whole
// fixed-point shadow in shared memory and owns up to 32 rows; x, v and F of
// its rows stay in registers, a thread per particle and component; a new
// shadow coordinate is written into all 16 shared memories (distributed
// shared memory), and a cluster barrier ends the step.  Equations and
// arithmetic per pair are those of lj_rows.cu.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "lj_device.cuh"
#include "lj_kernels.h"
#include "lj_mixed.cuh"
#include "lj_stepdev.cuh"

namespace ljgb {
namespace {

namespace cg = cooperative_groups;

constexpr int kCtas = 16;           // cluster size (non-portable)
constexpr int kPairWarps = 16;      // warps of the pair phase
constexpr int kSumWarp = kPairWarps;      // sums the CTA's rows for the observables
constexpr int kObsWarp = kPairWarps + 1;  // rank 0: forms the observables
constexpr int kThreads = 32 * (kPairWarps + 2);
constexpr int kCtaRows = 32;        // rows a CTA owns at most: one warp per component in the second half
constexpr int kMaxParts = 8;        // j parts a row's sum is made of

struct ClusterShared {
  int4 q[2][kClusterMaxN];                    // the shadow, by step parity
  int4 rowq[kCtaRows];                        // own rows' records (slots 1..3)
  int4 next[kCtaRows];                        // own rows' records of the next step
  float part[kPairWarps][8][5];               // warp: 8 rows x 5 sums
  double tv2[2][kCtas][3];                    // TVN: every CTA's component sums of tv^2
  double vel[2][3][kCtaRows];                 // by step parity: the rows' velocities
  FloatAcc pot[2][2][kCtaRows];               // and sums of (s/r)^12 and (s/r)^6
  double kvw[2][kCtas][3];                    // rank 0, by step parity: every CTA's sums of v^2, e, w
  double tkin[4], chi;                        // rank 0: TVN
};

// The two halves of a cluster barrier: what the thread wrote before arriving
// is visible to every CTA's threads that have waited.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Pairs of the warp's 8 rows (four groups of 8 lanes, two rows a lane) with
// the j's of chunks c0 .. c1-1 (8 j's each, one a lane of every group).
__device__ __forceinline__ void cluster_pairs(const int4* rowq, const int4* q, int n, int i, int c0, int c1,
                                              f32x2 k2i2, float (*out)[5]) {
  const int lane = threadIdx.x & 31, sub = lane & 7, g = lane >> 3;
  int4 qa, qb;  // volatile loads into aligned register quadruples (i_record_slots123)
  asm volatile("ld.volatile.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(qa.x), "=r"(qa.y), "=r"(qa.z), "=r"(qa.w)
               : "r"(smem_addr(rowq + 2 * g)));
  asm volatile("ld.volatile.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(qb.x), "=r"(qb.y), "=r"(qb.z), "=r"(qb.w)
               : "r"(smem_addr(rowq + 2 * g + 1)));
  const int ia = i + 2 * g;
  f32x2 f[5] = {0ull, 0ull, 0ull, 0ull, 0ull};
  // The chunks with the warp's own rows (8 of them, over two chunks where the
  // CTA's first row is no multiple of 8) and the ragged last one are masked.
  const int own = i >> 3, ragged = (n & 7) ? n >> 3 : -1;
  auto masked = [&](int c) {
    const int j = c * 8 + sub;
    const bool out_of = j >= n;
    pair_mixed_rows<true>(qa, qb, q[out_of ? 0 : j], k2i2, out_of || j == ia, out_of || j == ia + 1, f[0], f[1], f[2],
                          f[3], f[4]);
  };
  for (int c = c0; c < c1;) {
    int stop = c1;
    if (ragged >= c && ragged < stop) stop = ragged;
    if (own >= c && own < stop) stop = own;
    if (own + 1 >= c && own + 1 < stop) stop = own + 1;
#pragma unroll 4
    for (; c < stop; ++c)
      pair_mixed_rows<false>(qa, qb, q[c * 8 + sub], k2i2, false, false, f[0], f[1], f[2], f[3], f[4]);
    if (c < c1) masked(c++);
  }
  // Row a to lanes 0..3 of each group, row b to lanes 4..7: that makes plain FP32
  // sums of up to 32 pairs (a lane has 16 j's at most).  The four lanes of a row
  // meet in TwoSum pairs: values 0, 1 go to the lower two and 2, 3 to the upper,
  // then one value a lane; value 4 to all.
  const bool h2 = sub & 2, h1 = sub & 1;
  float v[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    float a, b;
    upk2(f[k], a, b);
    const float give = sub < 4 ? b : a;
    v[k] = (sub < 4 ? a : b) + __shfl_xor_sync(0xffffffffu, give, 4);
  }
  const f32x2 v01 = pk2(v[0], v[1]), v23 = pk2(v[2], v[3]);
  Float2Acc p{h2 ? v23 : v01, 0ull};
  two_sum_add2(p, __shfl_xor_sync(0xffffffffu, h2 ? v01 : v23, 2));
  FloatAcc v4{v[4], 0.f};
  two_sum_add(v4, __shfl_xor_sync(0xffffffffu, v4.hi, 2));
  float x, y, xl, yl;
  upk2(p.hi, x, y);
  upk2(p.lo, xl, yl);
  const FloatAcc one = exchange1(FloatAcc{x, xl}, FloatAcc{y, yl}, h1, 1);
  v4 = exchange1(v4, v4, false, 1);
  float* const row = out[2 * g + (sub >> 2)];
  row[(h2 ? 2 : 0) + (h1 ? 1 : 0)] = one.hi + one.lo;
  if ((sub & 3) == 0) row[4] = v4.hi + v4.lo;
}

// The 16 working warps meet here; the observables' two are left out, whose
// chains are as long as a step.
__device__ __forceinline__ void sync_workers() {
  asm volatile("bar.sync 1, %0;" ::"r"(32 * kPairWarps) : "memory");
}

// CalculateParameters (write_observables) over many steps with the running
// values in registers; one thread.
struct ClusterObs {
  double t, K, V, T, P, U, W, av_U, av_T, av_p, Tkin;
  long long step, av_iters, rec_count;
  int rec_at, rec_cap;
  bool bad;
  __device__ __forceinline__ void load(const DevScalars& sc) {
    t = sc.t;
    av_U = sc.av_U;
    av_T = sc.av_T;
    av_p = sc.av_p;
    step = sc.step;
    av_iters = sc.av_iters;
    rec_count = sc.rec_count;
    rec_cap = sc.rec_cap;
    rec_at = rec_cap > 0 ? (int)(rec_count % rec_cap) : 0;
    bad = false;
  }
  __device__ __forceinline__ void add(const StateArgs& s, const BoxArgs& box, double k, double v, double w,
                                      double tkin) {
    K = k;
    V = v;
    W = w;
    T = K * box.kT;
    P = fma(W, 1. / 6., (double)box.N * T) * box.kP;
    U = K + V;
    Tkin = tkin;
    t += box.dt;
    step += 1;
    av_iters += 1;
    av_U += U;
    av_p += P;
    av_T += T;
    bad |= !isfinite(K) || !isfinite(V) || !isfinite(W);
    if (rec_cap > 0) {
      s.records[rec_at] = DevRecord{t, K, V, T, P, U, W, s.sc[0].Pshear, Tkin, av_U, av_T, av_p, av_iters, step};
      rec_at = rec_at + 1 == rec_cap ? 0 : rec_at + 1;
      rec_count += 1;
    }
  }
  __device__ __forceinline__ void store(const StateArgs& s, DevScalars& sc) const {
    sc.t = t;
    sc.K = K;
    sc.V = V;
    sc.T = T;
    sc.P_press = P;
    sc.U = U;
    sc.W = W;
    sc.Tkin = Tkin;
    sc.step = step;
    sc.av_iters = av_iters;
    sc.av_U = av_U;
    sc.av_T = av_T;
    sc.av_p = av_p;
    sc.rec_count = rec_count;
    if (bad) atomicOr(s.status, LJ_DEVFLAG_NONFINITE);
  }
};

}  // namespace

// nsteps steps of box 0.  s.q holds the first step's predicted shadow and
// receives the one after the last.
//
// What bounds a step is latency, in clocks of rank 0's first warp at N = 400 (EVN,
// 7570 in all): pair phase 4250 (13 pairs a lane and their reduction), sums and ~12
// dependent FP64 operations of 64 clocks 1870, records sent and barrier 1450; TVN
// (11 800) adds a barrier (1000), two FP64 sums over the rows and chi's rsqrt
// (3070).  N = 128: 1370 + 2010 + 1050; N = 512: 5070 + 1790 + 1400.  The sums for
// the observables run beside the next step.  us a step, lj_rows.cu -> this
// one: EVN N = 128 5.4 -> 2.3, N = 256 5.4 -> 2.8, N = 400 5.5 -> 3.8, N = 512
// 5.6 -> 4.1; TVN N = 256 8.3 -> 4.7, N = 400 9.6 -> 5.7.  16 SMs are too few
// from N ~ 700 on.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 1) k_cluster(StateArgs s, int n, int rows, int nsteps) {
  __shared__ ClusterShared sh;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int i0 = rank * rows, nr = max(0, min(rows, n - i0));
  const BoxArgs box = s.boxes[0];
  DevScalars& sc = s.sc[0];
  const double fscale = sc.fscale, qscale = sc.invP * 4294967296.0;
  const f32x2 k2i2 = pk2(sc.k2inv, sc.k2inv);
  const bool worker = w < kPairWarps;

  for (int k = tid; k < n; k += kThreads) sh.q[0][k] = s.q[k];
  if (tid < kCtaRows) sh.next[tid] = make_int4(0, 0, 0, 0);
  for (int k = tid; k < 2 * 3 * kCtaRows; k += kThreads) (&sh.vel[0][0][0])[k] = 0.0;
  for (int k = tid; k < 2 * 2 * kCtaRows; k += kThreads) (&sh.pot[0][0][0])[k] = FloatAcc{0.f, 0.f};
  // second half: warp c < 3 holds component c of the rows, warp 3 their energy sums
  const bool mine = w < 4 && lane < nr;
  const size_t k3 = (size_t)min(w, 2) * s.npad + (mine ? i0 + lane : 0);
  double x = 0.0, v = 0.0, f = 0.0, origin = 0.0;
  if (mine && w < 3) {
    x = s.x[k3];
    v = s.v[k3];
    f = s.f[k3];
    if (box.bc != 0) origin = sc.origin[w];
  }
  // pair phase: 8 rows and a part of the j's a warp
  const int quads = (rows + 7) / 8, parts = min(kMaxParts, kPairWarps / quads);
  const int quad = w / parts, prt = w - quad * parts, nch = (n + 7) / 8;
  const bool pairs = w < quads * parts && quad * 8 < nr;
  const int c0 = prt * nch / parts, c1 = (prt + 1) * nch / parts;
  // where warp w sends the CTA's new records: CTA w's shadow (parity 0)
  int4* const dest = cluster.map_shared_rank(&sh.q[0][min(i0 + lane, n - 1)], w % kCtas);

  ClusterObs obs;
  if (rank == 0 && tid == 32 * kObsWarp) obs.load(sc);
  // kSumWarp sums a finished step's rows for rank 0 while the next step's
  // pairs are evaluated; kObsWarp forms the observables one step later.
  double e = 0.0, vir = 0.0;  // kSumWarp: of row `lane`, last step
  auto send_sums = [&](int step) {
    const double(*vel)[kCtaRows] = sh.vel[step & 1];
    const double vx = vel[0][lane], vy = vel[1][lane], vz = vel[2][lane];
    const FloatAcc a = sh.pot[step & 1][0][lane], b = sh.pot[step & 1][1][lane];
    const double A = widen(a.hi) + widen(a.lo), B = widen(b.hi) + widen(b.lo);
    e = box.eps4 * (A - B);
    vir = box.eps4 * fma(12.0, A, -6.0 * B);
    const double r = warp_sums<3>({fma(vx, vx, fma(vy, vy, vz * vz)), e, vir});
    double* const to = cluster.map_shared_rank(sh.kvw[step & 1][rank], 0);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (lane == sums_lane(k)) to[k] = r;
  };
  auto observe = [&](int step) {
    double kvw[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      kvw[k] = lane < kCtas ? sh.kvw[step & 1][lane][k] : 0.0;
#pragma unroll
      for (int o = kCtas / 2; o > 0; o >>= 1) kvw[k] += __shfl_down_sync(0xffffffffu, kvw[k], o);
    }
    if (lane == 0) obs.add(s, box, 0.5 * kvw[0], 0.5 * kvw[1], kvw[2], MODE == MODE_TVN ? sh.tkin[step & 3] : 0.0);
  };
  __syncthreads();
  cluster_arrive();  // every CTA has started and read s.q
  cluster_wait();

  for (int step = 0; step < nsteps; ++step) {
    const int cur = step & 1;
    if (!worker) {
      if (w == kObsWarp && rank == 0 && step >= 2) observe(step - 2);
      if (w == kSumWarp && step >= 1) send_sums(step - 1);
      if (MODE == MODE_TVN) {
        cluster_arrive();
        cluster_wait();
      }
      cluster_arrive();
      cluster_wait();
      continue;
    }
    if (tid < kCtaRows) {
      const int4 r = sh.q[cur][min(i0 + tid, n - 1)];
      sh.rowq[tid] = make_int4(0, r.x, r.y, r.z);
    }
    sync_workers();
    if (pairs) cluster_pairs(sh.rowq + quad * 8, sh.q[cur], n, i0 + quad * 8, c0, c1, k2i2, sh.part[w]);
    sync_workers();
    // a row's value k: its parts, in FP32 TwoSum, then FP64
    auto row_sum = [&](int k) {
      FloatAcc a{0.f, 0.f};
      for (int p = 0; p < parts; ++p) two_sum_add(a, sh.part[(lane >> 3) * parts + p][lane & 7][k]);
      return a;
    };
    double F = 0.0;
    if (mine && w < 3) {
      const FloatAcc a = row_sum(w);
      F = fscale * (widen(a.hi) + widen(a.lo));
    } else if (mine) {
      sh.pot[cur][0][lane] = row_sum(3);
      sh.pot[cur][1][lane] = row_sum(4);
    }
    if (MODE == MODE_TVN) {
      if (w < 3) {
        const double tv = fma(box.qdt, f + F, v);
        const double t = warp_sum(mine ? tv * tv : 0.0);
        const double all = __shfl_sync(0xffffffffu, t, 0);
        if (lane < kCtas) *cluster.map_shared_rank(&sh.tv2[cur][rank][w], lane) = all;
      }
      cluster_arrive();
      x = drift_pos(box, x, v, f);
      cluster_wait();
      if (w < 3) {
        double t = lane < kCtas ? (sh.tv2[cur][lane][0] + sh.tv2[cur][lane][1]) + sh.tv2[cur][lane][2] : 0.0;
        t = __shfl_sync(0xffffffffu, warp_sum(t), 0);
        double Tkin;
        const double chi = tvn_chi(box, t, &Tkin);
        v = fma(2. * chi - 1., v, 0.5 * (chi * box.dt) * (f + F));
        if (rank == 0 && tid == 0) {
          sh.tkin[step & 3] = Tkin;
          sh.chi = chi;
        }
      }
    } else if (w < 3) {
      x = drift_pos(box, x, v, f);
      v = fma(box.hdt, F, fma(box.hdt, f, v));
    }
    if (w < 3) {
      f = F;
      apply_bc1(box.bc, box.L, x, v);
      const double xp = drift_pos(box, x, v, F);
      if (mine) {
        const int qn = predicted_fixed(s, box.bc, origin, qscale, xp);
        reinterpret_cast<int*>(&sh.next[lane])[w] = qn;
        sh.vel[cur][w][lane] = v;
        if (step == nsteps - 1) reinterpret_cast<int*>(s.q + i0 + lane)[w] = qn;
      }
    }
    sync_workers();
    if (lane < nr) dest[(cur ^ 1) * kClusterMaxN] = sh.next[lane];
    cluster_arrive();
    cluster_wait();
  }
  if (w == kSumWarp) send_sums(nsteps - 1);
  cluster_arrive();
  if (mine && w < 3) {
    s.x[k3] = x;
    s.v[k3] = v;
    s.f[k3] = f;
  } else if (w == kSumWarp && lane < nr) {
    s.e[i0 + lane] = e;
    s.w[i0 + lane] = vir;
  }
  cluster_wait();
  if (rank == 0 && w == kObsWarp) {
    for (int step = max(0, nsteps - 2); step < nsteps; ++step) observe(step);
    if (lane == 0) {
      obs.store(s, sc);
      if (MODE == MODE_TVN) sc.chi = sh.chi;
    }
  }
}

namespace {
cudaLaunchConfig_t cluster_config(cudaLaunchAttribute* attr, cudaStream_t st) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = kCtas;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kCtas);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}
}  // namespace

// Whether the device can hold a cluster of this kernel (it needs 16 SMs of one
// GPC).
cudaError_t cluster_setup(bool* usable) {
  *usable = false;
  for (auto* k : {k_cluster<MODE_EVN>, k_cluster<MODE_TVN>}) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cluster_config(&attr, nullptr);
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, k, &cfg);
    if (e != cudaSuccess) return e;
    if (clusters < 1) return cudaSuccess;
  }
  *usable = true;
  return cudaSuccess;
}

cudaError_t launch_cluster(const StateArgs& s, int n, int mode, int nsteps, cudaStream_t st) {
  const int rows = 2 * ((n + 2 * kCtas - 1) / (2 * kCtas));
  if (rows > kCtaRows) return cudaErrorInvalidValue;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config(&attr, st);
  return cudaLaunchKernelEx(&cfg, mode == MODE_EVN ? k_cluster<MODE_EVN> : k_cluster<MODE_TVN>, s, n, rows, nsteps);
}

}  // namespace ljgb
