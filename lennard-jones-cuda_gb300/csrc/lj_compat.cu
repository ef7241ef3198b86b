// lj_compat.cu -- the reference's extern "C" CUDA entry points
// (src/library/MDSystem.cu:155-299, declared at MDSystem.cpp:10-25) on top of
// this library's sm_103a pair kernel.  See include/lj_reference_abi.h for the
// contract and the deliberate differences.
//
// calculateNForces: float4 positions -> fixed-point shadow (frame from L or
// from the bounding box for non-periodic boxes) -> the pair kernels of a step
// without the step (the row kernel below kNewtonMinN particles, unordered pairs
// up to kNewtonMaxN, the stream-K kernel above, and where the unordered pairs'
// sums cannot be had) -> per-particle float4 forces
// and one FP64 virial sum; the 256-bin r^2 RDF, where it is asked for, is the histogram
// kernel's (lj_rdf.cu): a call of N = 8000 took 203 us with both in one kernel and
// took 155 us in two, since the force loop evaluates ordered pairs and the
// histogram each unordered pair once.  Work buffers
// are cached per particle count on a private stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "lj_device.cuh"
#include "lj_gb300.h"
#include "lj_kernels.h"
#include "lj_reference_abi.h"
#include "lj_schedule.h"

namespace ljgb {
namespace {

constexpr int kRefBins = 256;  // NdNdr2 size (MDSystem.cpp:97)
constexpr int kBlk = kFloat4Threads;

// What a call reads back, in one copy.
struct RefResult {
  unsigned long long hist[kRefBins];
  float pressure;
  int status;
};

// Force[i] = (F, sum_j r^-12 - r^-6), the segments added in FP32 TwoSum as the
// integrators do; block partial of sum_j s r^2.  The last CTA to finish adds
// the partials: pressure = (4/6) sum_i sum_j s r^2 (MDSystem.cu:105-108, 136).
__global__ void k_ref_reduce(const float* partial, const BlockInfo* blocks, int bi_threads, const DevScalars* sc,
                             float4* force, double* blk, int* ticket, RefResult* result) {
  __shared__ double sh[32];
  __shared__ bool last;
  const BlockInfo bi = blocks[blockIdx.x];
  const int tid = threadIdx.x;
  double part[1] = {0.0};
  if (tid < bi.n_i) {
    FloatAcc acc[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) acc[c] = FloatAcc{0.f, 0.f};
#pragma unroll 4
    for (int k = 0; k < bi.seg_count; ++k) {
      const size_t base = (size_t)(bi.seg_first + k) * 5 * bi_threads + tid;
#pragma unroll
      for (int c = 0; c < 5; ++c) two_sum_add(acc[c], partial[base + (size_t)c * bi_threads]);
    }
    double S[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) S[c] = (double)acc[c].hi + (double)acc[c].lo;
    const double fs = sc->fscale;
    force[bi.i0 + tid] = make_float4((float)(fs * S[0]), (float)(fs * S[1]), (float)(fs * S[2]), (float)(S[3] - S[4]));
    part[0] = 12.0 * S[3] - 6.0 * S[4];
  }
  block_sum<1>(part, sh);
  if (tid == 0) {
    blk[(size_t)blockIdx.x * 8] = part[0];
    __threadfence();
    last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double acc[1] = {0.0};
  for (int b = tid; b < (int)gridDim.x; b += blockDim.x) acc[0] += __ldcg(blk + (size_t)b * 8);
  block_sum<1>(acc, sh);
  if (tid == 0) {
    result->pressure = (float)(acc[0] * 4.0 / 6.0);
    *ticket = 0;
  }
}

struct CompatCtx {
  int device = -1;  // the device that holds the buffers below
  int n = 0;
  int shape = -1;
  int nb_bbox = 0;
  Schedule sched;
  cudaStream_t stream = nullptr;
  int4* q = nullptr;
  DevScalars* sc = nullptr;
  // the row or the unordered-pair kernel (rows.ctas > 0 or newton > 0) ...
  RowPlan rows{};
  int newton = 0;
  NewtonTask* newton_tasks = nullptr;
  int* newton_blocks = nullptr;
  float *newton_j = nullptr, *newton_i = nullptr;
  // ... or the stream-K kernel's schedule
  BlockInfo* blocks = nullptr;
  int *ctb = nullptr, *clo = nullptr, *cb = nullptr, *cj = nullptr;
  int rdf_grid = 0, num_sms = 0;
  int *rb = nullptr, *rc = nullptr, *ru = nullptr;  // ranges of the histogram pass
  RdfNear near{};                                   // large boxes: its tiles of neighbours
  float* partial = nullptr;
  double* blk = nullptr;
  RefResult* result = nullptr;       // device
  RefResult* host_result = nullptr;  // page-locked, with room for the completion word behind it
  ResultMail* mail = nullptr;        // [0] without, [1] with the histogram; null: results are copied
  int* ticket = nullptr;             // [0] reduce, [1] bounding box (0 between launches)
  void release() {
    if (stream) cudaStreamSynchronize(stream);
    cudaFree(q);
    cudaFree(sc);
    cudaFree(newton_tasks);
    cudaFree(newton_blocks);
    cudaFree(newton_j);
    cudaFree(newton_i);
    cudaFree(blocks);
    cudaFree(ctb);
    cudaFree(clo);
    cudaFree(cb);
    cudaFree(cj);
    cudaFree(rb);
    cudaFree(rc);
    cudaFree(ru);
    cudaFree(near.cells);
    cudaFree(near.rank);
    cudaFree(near.sorted);
    cudaFree(near.box);
    cudaFree(partial);
    cudaFree(blk);
    cudaFree(result);
    cudaFree(mail);
    cudaFree(ticket);
    if (host_result) cudaFreeHost(host_result);
    if (stream) cudaStreamDestroy(stream);
    *this = CompatCtx();
  }
};

std::mutex g_mu;
CompatCtx g_ctx;
int g_status = 0;
std::string g_error;

bool record(cudaError_t e, const char* what, bool loud = true) {
  if (e == cudaSuccess) return true;
  g_status = e == cudaErrorMemoryAllocation ? LJ_ERR_OUT_OF_MEMORY : LJ_ERR_CUDA;
  g_error = std::string(what) + ": " + cudaGetErrorString(e);
  if (loud) std::fprintf(stderr, "lj_gb300 reference ABI: %s\n", g_error.c_str());
  return false;
}

constexpr bool loud = true;  // (build_ctx has one of its own)
#define REF_CHECK(call) \
  if (!record((call), #call, loud)) return false

// A context for n particles on the current device, into g_ctx.  `lean`: without
// what a call can do without, the unordered pairs' sums (up to 10 KB a particle;
// the stream-K kernel takes their place) and the histogram's neighbour tiles.
bool build_ctx(int n, int shape, int dev, bool lean, bool loud) {
  int sms = 0, per_sm = 0;
  REF_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const RowPlan rows = plan_rows(n, sms);
  NewtonPlan np;
  if (!lean && n >= kNewtonMinN && n <= kNewtonMaxN) {
    int newton_per_sm = 0;
    REF_CHECK(newton_setup(&newton_per_sm));
    if (newton_per_sm > 0) np = plan_newton(n, sms * newton_per_sm * kNewtonWarps);
    if (!leaves_room(np.bytes())) np = NewtonPlan();
  }
  const bool stream_k = np.tasks.empty() && rows.ctas == 0;
  Schedule s;
  if (stream_k) {
    REF_CHECK(pair_occupancy(shape, &per_sm));
    // at most 8 CTAs per i-block (a block's epilogue sums one segment per CTA)
    const int nb_i = (n + kShapes[shape].threads - 1) / kShapes[shape].threads;
    const int ctas = std::min(sms * per_sm, 8 * nb_i);
    if (!build_schedule(&n, 1, kShapes[shape].threads, kShapes[shape].tile, ctas, 8, &s)) {
      g_status = LJ_ERR_INVALID;
      g_error = "cannot build the pair schedule";
      return false;
    }
  }
  RdfRanges rr;
  if (!build_rdf_ranges(n, sms * rdf_ctas_per_sm(), &rr)) {
    g_status = LJ_ERR_INVALID;
    g_error = "cannot build the histogram ranges";
    return false;
  }
  CompatCtx c;
  c.device = dev;
  c.n = n;
  c.shape = shape;
  c.nb_bbox = (n + kBlk - 1) / kBlk;
  c.num_sms = sms;
  // Buffers of the new context; on any failure everything allocated so far
  // is freed and the layer is left without a context (the next call retries).
  auto build = [&]() -> bool {
    // A blocking stream: the reference's ABI is synchronous and its copies
    // (copyArrayToDevice, cudaMemcpy on the legacy stream) must be ordered
    // before this stream's kernels; a pageable cudaMemcpy can return before
    // its DMA has landed.
    REF_CHECK(cudaStreamCreateWithFlags(&c.stream, cudaStreamDefault));
    const int nb = (int)s.blocks.size();
    REF_CHECK(device_alloc((void**)&c.q, sizeof(int4) * n));
    REF_CHECK(device_alloc((void**)&c.sc, sizeof(DevScalars)));
    REF_CHECK(device_alloc((void**)&c.rb, sizeof(int) * rr.G));
    REF_CHECK(device_alloc((void**)&c.rc, sizeof(int) * rr.G));
    REF_CHECK(device_alloc((void**)&c.ru, sizeof(int) * rr.G));
    if (!lean && rdf_near(n, 0.0, 1.0)) {
      REF_CHECK(device_alloc((void**)&c.near.cells, sizeof(int) * kRdfCells));
      REF_CHECK(device_alloc((void**)&c.near.rank, sizeof(int) * n));
      REF_CHECK(device_alloc((void**)&c.near.sorted, sizeof(int4) * n));
      REF_CHECK(device_alloc((void**)&c.near.box, sizeof(uint2) * 3 * (size_t)((n + 31) / 32)));
    }
    // 8 doubles per CTA, i-block, tile or bounding-box CTA, whichever are most
    REF_CHECK(device_alloc((void**)&c.blk, sizeof(double) * 8 * (size_t)std::max({nb, c.nb_bbox, (n + 31) / 32, sms})));
    if (stream_k) {
      REF_CHECK(device_alloc((void**)&c.blocks, sizeof(BlockInfo) * nb));
      REF_CHECK(device_alloc((void**)&c.ctb, sizeof(int) * (s.G + 1)));
      REF_CHECK(device_alloc((void**)&c.clo, sizeof(int) * (s.G + 1)));
      REF_CHECK(device_alloc((void**)&c.cb, sizeof(int) * s.G));
      REF_CHECK(device_alloc((void**)&c.cj, sizeof(int) * s.G));
      REF_CHECK(device_alloc((void**)&c.partial, sizeof(float) * (size_t)s.nseg * 5 * s.BI));
      REF_CHECK(cudaMemcpy(c.blocks, s.blocks.data(), sizeof(BlockInfo) * nb, cudaMemcpyHostToDevice));
      REF_CHECK(cudaMemcpy(c.ctb, s.cta_tile_begin.data(), sizeof(int) * (s.G + 1), cudaMemcpyHostToDevice));
      REF_CHECK(cudaMemcpy(c.clo, s.cta_lo.data(), sizeof(int) * (s.G + 1), cudaMemcpyHostToDevice));
      REF_CHECK(cudaMemcpy(c.cb, s.cta_block.data(), sizeof(int) * s.G, cudaMemcpyHostToDevice));
      REF_CHECK(cudaMemcpy(c.cj, s.cta_jt.data(), sizeof(int) * s.G, cudaMemcpyHostToDevice));
    } else if (rows.ctas > 0) {
      c.rows = rows;
      REF_CHECK(rows_setup());
    } else {
      REF_CHECK(device_alloc((void**)&c.newton_tasks, sizeof(NewtonTask) * np.tasks.size()));
      REF_CHECK(device_alloc((void**)&c.newton_blocks, sizeof(int) * np.block_part.size()));
      REF_CHECK(device_alloc((void**)&c.newton_j, sizeof(float) * 160 * (size_t)np.jparts));
      REF_CHECK(device_alloc((void**)&c.newton_i, sizeof(float) * 5 * kNewtonBlock * (size_t)np.iparts));
      REF_CHECK(cudaMemcpy(c.newton_tasks, np.tasks.data(), sizeof(NewtonTask) * np.tasks.size(), cudaMemcpyHostToDevice));
      REF_CHECK(cudaMemcpy(c.newton_blocks, np.block_part.data(), sizeof(int) * np.block_part.size(), cudaMemcpyHostToDevice));
      c.newton = (int)np.tasks.size();
    }
    REF_CHECK(device_alloc((void**)&c.result, sizeof(RefResult)));
    REF_CHECK(device_alloc((void**)&c.ticket, 2 * sizeof(int)));
    REF_CHECK(pinned_alloc((void**)&c.host_result, sizeof(RefResult) + sizeof(int)));
    void* mapped = nullptr;
    if (cudaHostGetDevicePointer(&mapped, c.host_result, 0) != cudaSuccess) (void)cudaGetLastError();
    else if (!stream_k) {
      REF_CHECK(device_alloc((void**)&c.mail, 2 * sizeof(ResultMail)));
      ResultMail m[2];
      for (int k = 0; k < 2; ++k) {
        const int skip = k ? 0 : (int)(offsetof(RefResult, pressure) / sizeof(int));
        const int words = (int)(sizeof(RefResult) / sizeof(int));
        m[k] = ResultMail{reinterpret_cast<const int*>(c.result) + skip, static_cast<int*>(mapped) + skip, words - skip,
                          static_cast<int*>(mapped) + words};
      }
      REF_CHECK(cudaMemcpy(c.mail, m, sizeof(m), cudaMemcpyHostToDevice));
    }
    REF_CHECK(cudaMemset(c.sc, 0, sizeof(DevScalars)));
    REF_CHECK(cudaMemset(c.result, 0, sizeof(RefResult)));
    REF_CHECK(cudaMemset(c.ticket, 0, 2 * sizeof(int)));
    REF_CHECK(cudaMemcpy(c.rb, rr.cta_block.data(), sizeof(int) * rr.G, cudaMemcpyHostToDevice));
    REF_CHECK(cudaMemcpy(c.rc, rr.cta_chunk.data(), sizeof(int) * rr.G, cudaMemcpyHostToDevice));
    REF_CHECK(cudaMemcpy(c.ru, rr.cta_units.data(), sizeof(int) * rr.G, cudaMemcpyHostToDevice));
    c.rdf_grid = rr.G;
    return true;
  };
  if (!build()) {
    c.release();
    return false;
  }
  c.sched = std::move(s);
  g_ctx = c;
  return true;
}

bool ensure_ctx(int n, int block_hint) {
  int shape = 0;
  for (int k = 0; k < kNumShapes; ++k)
    if (std::abs(kShapes[k].threads - block_hint) < std::abs(kShapes[shape].threads - block_hint)) shape = k;
  int dev = 0;
  REF_CHECK(cudaGetDevice(&dev));
  if (g_ctx.n == n && g_ctx.shape == shape && g_ctx.stream && g_ctx.device == dev) return true;
  if (g_ctx.stream && g_ctx.device != dev) {
    // The caller switched devices: free the old buffers on their own device.
    REF_CHECK(cudaSetDevice(g_ctx.device));
    g_ctx.release();
    REF_CHECK(cudaSetDevice(dev));
  } else {
    g_ctx.release();
  }
  // Without the memory for everything, with less (for as long as this context
  // is kept: until another n, shape or device, or threadExit).
  const bool can_be_lean = n >= kNewtonMinN;
  const std::string error = g_error;
  if (build_ctx(n, shape, dev, false, !can_be_lean)) return true;
  if (g_status != LJ_ERR_OUT_OF_MEMORY || !can_be_lean) {
    if (can_be_lean) std::fprintf(stderr, "lj_gb300 reference ABI: %s\n", g_error.c_str());
    return false;
  }
  g_status = 0;
  g_error = error;
  return build_ctx(n, shape, dev, true, true);
}

bool calc_forces(float* Pos, float* Force, float* host_pressure, int n, float L, int periodic, int* host_RDF,
                 float dr2, int block_size) {
  if (!Pos || !Force || !host_pressure || n < 2) {
    g_status = LJ_ERR_INVALID;
    g_error = "calculateNForces: null array or numBodies < 2";
    return false;
  }
  if (!ensure_ctx(n, block_size > 0 ? block_size : 128)) return false;
  CompatCtx& c = g_ctx;
  const float4* pos = reinterpret_cast<const float4*>(Pos);
  const bool want_rdf = host_RDF != nullptr && dr2 > 0.0f;
  const bool near = want_rdf && c.near.cells && rdf_near(n, std::sqrt((double)kRefBins * dr2), L);
  if (near) REF_CHECK(cudaMemsetAsync(c.near.cells, 0, sizeof(int) * kRdfCells, c.stream));
  if (want_rdf) REF_CHECK(cudaMemsetAsync(c.result->hist, 0, sizeof(c.result->hist), c.stream));
  REF_CHECK(launch_float4_shadow(pos, n, periodic, (double)L, c.sc, nullptr, c.blk, c.ticket + 1, c.q, c.stream));
  const RdfPass rdf{c.q, c.sc, n, c.rb, c.rc, c.ru, HistArgs{0, kRefBins, 1.0f / dr2, 0.0f, c.result->hist}, {}, nullptr};
  if (near) {
    REF_CHECK(launch_rdf_near(rdf, c.near, periodic != 0, c.num_sms * rdf_ctas_per_sm(), c.stream));
  } else if (want_rdf) {
    REF_CHECK(launch_rdf(rdf, c.rdf_grid, c.stream));
  }
  // set by the last CTA once the results are in host memory
  volatile int* const done = reinterpret_cast<volatile int*>(c.host_result + 1);
  if (c.rows.ctas > 0 || c.newton > 0) {
    StateArgs st{};
    st.q = c.q;
    st.sc = c.sc;
    st.status = &c.result->status;
    st.row_part = c.blk;
    st.blk_cnt = c.ticket;
    st.force4 = reinterpret_cast<float4*>(Force);
    st.pressure = &c.result->pressure;
    st.mail = c.mail ? c.mail + (want_rdf ? 1 : 0) : nullptr;
    *done = 0;
    if (c.newton > 0) {
      const NewtonArgs na{c.q, c.sc, c.newton_tasks, c.newton_blocks, c.newton_j, c.newton_i, n, c.newton};
      REF_CHECK(launch_newton(na, c.stream));
      REF_CHECK(launch_newton_sum(st, na, MODE_FORCES_ONLY, c.stream));
    } else {
      REF_CHECK(launch_rows(st, c.rows, n, MODE_FORCES_ONLY, c.stream));
    }
  } else {
    PairArgs a{};
    a.q = c.q;
    a.blocks = c.blocks;
    a.cta_tile_begin = c.ctb;
    a.cta_lo = c.clo;
    a.cta_block = c.cb;
    a.cta_jt = c.cj;
    a.sc = c.sc;
    a.partial = c.partial;
    a.status = &c.result->status;
    REF_CHECK(launch_pairs(c.shape, a, c.sched.G, c.stream));
    const int nb = (int)c.sched.blocks.size();
    k_ref_reduce<<<nb, c.sched.BI, 0, c.stream>>>(c.partial, c.blocks, c.sched.BI, c.sc,
                                                    reinterpret_cast<float4*>(Force), c.blk, c.ticket, c.result);
    REF_CHECK(cudaGetLastError());
  }
  // The results come by the launch's own stores and its completion word (N =
  // 8000 with RDF: 98.5 us a call with a copy behind it, 95 so; N = 1000 without
  // 39 -> 28).  If the word does not come within 20 ms, and with the stream-K
  // kernel, they come by a copy into page-locked memory.
  RefResult* const r = c.host_result;
  bool here = false;
  if (c.mail) {
    const auto t0 = std::chrono::steady_clock::now();
    for (unsigned it = 1; !here; ++it) {
      here = *done == 1;
      if ((it & 255u) == 0 && std::chrono::steady_clock::now() - t0 > std::chrono::milliseconds(20)) break;
    }
    std::atomic_thread_fence(std::memory_order_acquire);
  }
  if (!here) {
    const size_t skip = want_rdf ? 0 : offsetof(RefResult, pressure);
    REF_CHECK(cudaMemcpyAsync(reinterpret_cast<char*>(r) + skip, reinterpret_cast<const char*>(c.result) + skip,
                              sizeof(RefResult) - skip, cudaMemcpyDeviceToHost, c.stream));
    REF_CHECK(cudaStreamSynchronize(c.stream));
  }
  *host_pressure = r->pressure;
  if (r->status) {
    // A CTA whose wait timed out takes no completion ticket: the count goes back
    // to 0 as well, behind the launch's last CTA, or the next call's last CTA
    // would be taken for an earlier one.
    REF_CHECK(cudaMemsetAsync(&c.result->status, 0, sizeof(int), c.stream));
    REF_CHECK(cudaMemsetAsync(c.ticket, 0, 2 * sizeof(int), c.stream));
    REF_CHECK(cudaStreamSynchronize(c.stream));
    g_status = LJ_ERR_DEVICE_TIMEOUT;
    g_error = "calculateNForces: a device-side wait timed out";
    return false;
  }
  if (want_rdf)
    for (int b = 0; b < kRefBins; ++b) host_RDF[b] = (int)r->hist[b];
  return true;
}

}  // namespace
}  // namespace ljgb

using namespace ljgb;

extern "C" {

void allocateNBodyArrays(float* vel[2], int numBodies) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  const size_t bytes = sizeof(float) * 4 * (size_t)numBodies;
  vel[0] = vel[1] = nullptr;
  if (record(device_alloc((void**)&vel[0], bytes), "cudaMalloc") &&
      !record(device_alloc((void**)&vel[1], bytes), "cudaMalloc")) {
    cudaFree(vel[0]);
    vel[0] = nullptr;
  }
}

void allocateArray(float** dest, int number) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  record(device_alloc((void**)dest, sizeof(float) * 4 * (size_t)number), "cudaMalloc");
}

void deleteNBodyArrays(float* vel[2]) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  record(cudaFree(vel[0]), "cudaFree");
  record(cudaFree(vel[1]), "cudaFree");
}

void deleteArray(float* arr) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  record(cudaFree(arr), "cudaFree");
}

void allocateIntArray(int** dest, int number) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  record(device_alloc((void**)dest, sizeof(int) * (size_t)number), "cudaMalloc");
}

void deleteIntArray(int* arr) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  record(cudaFree(arr), "cudaFree");
}

void copyArrayFromDevice(float* host, const float* device, unsigned int pbo, int numBodies) {
  (void)pbo;
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  record(cudaMemcpy(host, device, sizeof(float) * 4 * (size_t)numBodies, cudaMemcpyDeviceToHost), "cudaMemcpy");
}

void copyArrayToDevice(float* device, const float* host, int numBodies) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  record(cudaMemcpy(device, host, sizeof(float) * 4 * (size_t)numBodies, cudaMemcpyHostToDevice), "cudaMemcpy");
}

void registerGLBufferObject(unsigned int pbo) { (void)pbo; }

void unregisterGLBufferObject(unsigned int pbo) { (void)pbo; }

void threadSync(void) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  record(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
}

void calculateNForces(float* Pos, float* Force, float* host_pressure, int numBodies, float host_L, int Lperiodic,
                      int* host_RDF, float host_dr2, int blockSize, int q) {
  (void)q;
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  calc_forces(Pos, Force, host_pressure, numBodies, host_L, Lperiodic, host_RDF, host_dr2, blockSize);
}

void threadExit(void) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_status = 0;
  g_ctx.release();
  record(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
}

int lj_debug_reference_abi_timeout(int tickets) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_ctx.stream) return LJ_ERR_INVALID;
  const int status = LJ_DEVFLAG_TIMEOUT;
  if (cudaMemcpy(g_ctx.ticket, &tickets, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(&g_ctx.result->status, &status, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
    return LJ_ERR_CUDA;
  return LJ_OK;
}

int lj_reference_abi_status(void) { return g_status; }

const char* lj_reference_abi_error(void) { return g_error.c_str(); }

}  // extern "C"

// ---------------------------------------------------------------------------
// Fixed-point shadow of caller-owned float4 positions, shared by the
// reference ABI above and the allocation-free force entry point
// (lj_noalloc.cu).
// ---------------------------------------------------------------------------
namespace ljgb {
namespace {

// Frame of the fixed-point shadow (eps = sigma = 1).  Periodic: origin 0,
// period L.  Otherwise the bounding box's low corner and a period of twice its
// largest extent, so no separation wraps.
__host__ __device__ inline void float4_frame(DevScalars* sc, double ox, double oy, double oz, double P) {
  sc->origin[0] = ox;
  sc->origin[1] = oy;
  sc->origin[2] = oz;
  sc->P = P;
  sc->invP = 1.0 / P;
  const double ks = P / 4294967296.0;
  sc->k2 = (float)(ks * ks);
  sc->k2inv = (float)(1.0 / (ks * ks));
  sc->fscale = 4.0 * ks;
}

// Bounding box of the positions: per CTA (blk[b*8 + 0..2] = min, [3..5] =
// max), then over the CTAs by the last one to finish, which writes the frame
// (and clears *status when given).
__global__ void k_float4_bbox(const float4* pos, int n, double* blk, int* ticket, DevScalars* sc, int* status) {
  __shared__ float sh[6][32];
  __shared__ bool last;
  const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float v[6] = {INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY};  // min x, y, z, min -x, -y, -z
  if (i < n) {
    const float4 p = pos[i];
    v[0] = p.x, v[1] = p.y, v[2] = p.z, v[3] = -p.x, v[4] = -p.y, v[5] = -p.z;
  }
  auto over_block = [&]() {  // of v, in every thread
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      for (int o = 16; o > 0; o >>= 1) v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
      if (lane == 0) sh[k][warp] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 6; ++k)
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v[k] = fminf(v[k], sh[k][w]);
    __syncthreads();
  };
  over_block();
  if (threadIdx.x == 0) {
    for (int k = 0; k < 6; ++k) blk[(size_t)blockIdx.x * 8 + k] = v[k];
    __threadfence();
    last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    v[k] = INFINITY;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v[k] = fminf(v[k], (float)__ldcg(blk + (size_t)b * 8 + k));
  }
  over_block();
  if (threadIdx.x != 0) return;
  double ext = 0;
  for (int k = 0; k < 3; ++k) ext = fmax(ext, -(double)v[3 + k] - (double)v[k]);
  float4_frame(sc, v[0], v[1], v[2], 2.002 * ext + 1e-3);
  *ticket = 0;
  if (status) *status = 0;
}

// With PERIODIC the frame comes by value and is written to *sc for the
// kernels that follow (and *status cleared when given).
template <bool PERIODIC>
__global__ void k_float4_quantize(const float4* pos, int n, DevScalars* sc, int4* q, DevScalars frame, int* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (PERIODIC && i == 0) {
    *sc = frame;
    if (status) *status = 0;
  }
  if (i >= n) return;
  const float4 p = pos[i];
  const DevScalars& f = PERIODIC ? frame : *sc;
  q[i] = make_int4(fixed_coord(p.x, f.origin[0], f.invP), fixed_coord(p.y, f.origin[1], f.invP),
                   fixed_coord(p.z, f.origin[2], f.invP), 0);
}

}  // namespace

cudaError_t launch_float4_shadow(const float4* pos, int n, int periodic, double L, DevScalars* sc, int* status,
                                 double* blk, int* ticket, int4* q, cudaStream_t st) {
  const int grid = (n + kFloat4Threads - 1) / kFloat4Threads;
  DevScalars frame{};
  if (periodic) {
    float4_frame(&frame, 0.0, 0.0, 0.0, L);
    k_float4_quantize<true><<<grid, kFloat4Threads, 0, st>>>(pos, n, sc, q, frame, status);
  } else {
    k_float4_bbox<<<grid, kFloat4Threads, 0, st>>>(pos, n, blk, ticket, sc, status);
    k_float4_quantize<false><<<grid, kFloat4Threads, 0, st>>>(pos, n, sc, q, frame, nullptr);
  }
  return cudaGetLastError();
}

}  // namespace ljgb
