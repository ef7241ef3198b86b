// lj_kernels.h -- launch interface of the LJ kernels (host side).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "lj_internal.h"

namespace ljgb {

constexpr int kMaxHistBins = 4096;

// Pair-histogram request.  mode 0: r^2 bins, clamp overflow to the last bin
// (MDSystem.cu:39); 1: r^2 bins, drop overflow (MDSystem.cpp:282-284);
// 2: linear r bins up to rmax (pairs with r >= rmax dropped).
struct HistArgs {
  int mode;
  int nb;
  float inv_w;   // 1/dr2 (modes 0,1) or 1/dr (mode 2)
  float rmax2;   // mode 2: rmax^2 in sigma^2
  unsigned long long* counts;  // nb counters (global, accumulated with atomics)
};

// Arguments of the persistent pair kernels (by value).
struct PairArgs {
  const int4* q;              // MIXED: fixed-point shadow (x, y, z, pad), all boxes
  const BlockInfo* blocks;    // i-blocks of the schedule
  const int* cta_tile_begin;  // G+1 tile ranges
  const int* cta_block;       // first i-block of each CTA
  const int* cta_jt;          // first j-tile (within that block) of each CTA
  const int* cta_lo;          // G+1 j offsets within the first tile (entry g+1: end in the
                              // last tile, 0 = whole tile); nullptr = whole tiles only
  const DevScalars* sc;       // per box frame / scalars
  const BoxArgs* boxes;       // per box constants
  float* partial;             // nseg x 5 x threads
  int* status;                // device status word (timeouts)
};


// Small device words copied by the pack launch: the status word (and the
// upload check's bad index, if bad is set, which is then reset to 0x7f7f7f7f)
// to words_out[0..1], and sc_nwords 32-bit words of the scalar block to sc_out.
struct Mailbox {
  const int* status;
  int* bad;
  int* words_out;
  const int* sc;
  int* sc_out;
  int sc_nwords;
  int finalize;  // != 0: compute the observables the last fused TVN step left pending first (one CTA per box)
  int* ticket;   // finalize with several boxes: the last box's CTA copies the status words (0 between launches)
  // seq != 0: the launch's last CTA writes seq into words_out[2] once every
  // store of the launch is visible to the host (grid_ticket: CTAs done, 0
  // between launches), so the host can wait on that word alone.
  int* grid_ticket;
  int seq;
};

// Pair histogram of one box of n particles (lj_rdf.cu) over the fixed-point
// shadow q: adds the counts of all ordered pairs to h.counts.  The ranges are
// those of build_rdf_ranges for at most rdf_ctas_per_sm() CTAs an SM.
struct RdfPass {
  const int4* q;
  const DevScalars* sc;    // the box's frame (k2)
  int n;
  const int* cta_block;    // first i-block of each CTA
  const int* cta_chunk;    // first j-chunk of that block
  const int* cta_units;    // chunks the CTA covers
  HistArgs hist;
  // with mail.seq != 0 the last CTA hands the counts and the status words over:
  // counts_out is host memory, mail.grid_ticket 0 between launches
  Mailbox mail;
  unsigned long long* counts_out;
};
int rdf_ctas_per_sm();
// The same by tiles of neighbours (four launches; without a.mail mode 0 alone).  Sorting
// costs about 20 us, which the pairs left out have to be worth.  us a call at
// reach / L, all pairs -> near tiles, particles in lattice order (shuffled: 5 to
// 20% more for all pairs, the same for near tiles): N = 8192 at 0.15 41 -> 47, 0.25
// 44 -> 55; N = 10000 48 -> 68, 52 -> 78; N = 12000 62 -> 62, 69 -> 75; N = 14000 79
// -> 54, 88 -> 76; N = 16384 at 0.15 95 -> 56, 0.25 108 -> 95, 0.35 120 -> 129; N =
// 32768 at 0.15 296 -> 144, 0.35 380 -> 368, 0.4 402 -> 443; N = 40000 at 0.15 435
// -> 183, 0.35 556 -> 442.  The two cross between 12000 and 14000, by how the
// sorted tiles fall; the line lies above, at 16384, where near tiles win throughout.
// (A droplet within the reach leaves nothing out.)
struct RdfNear {
  int* cells;    // kRdfCells, 0 before
  int* rank;     // n: place within the cell
  int4* sorted;  // n
  uint2* box;    // 3 per tile of 32
};
constexpr int kRdfCells = 4096;
constexpr int kRdfNearMaxN = 1 << 20;  // a CTA's 32-bit counts
inline bool rdf_near(int n, double reach, double L) {
  return n >= 16384 && n <= kRdfNearMaxN && reach <= (n >= 32768 ? 0.35 : 0.25) * L;
}
cudaError_t launch_rdf_near(const RdfPass& a, const RdfNear& s, bool periodic, int grid, cudaStream_t st);
cudaError_t launch_rdf(const RdfPass& a, int grid, cudaStream_t st);

struct PairShape {
  int threads;  // CTA size = i-block length (one i per thread)
  int tile;     // j records per staged tile
  int stages;   // depth of the bulk-copy ring
};

extern const PairShape kShapes[];
extern const int kNumShapes;

cudaError_t pair_occupancy(int shape, int* blocks_per_sm);
cudaError_t launch_pairs(int shape, const PairArgs& a, int grid, cudaStream_t st);
struct FusedPairArgs;
cudaError_t launch_pairs_fused(int shape, int mode, const FusedPairArgs& a, int grid, cudaStream_t st);

// ---------------------------------------------------------------------------
// Integrator / reduction kernels (lj_integrate.cu).  All operate on the
// i-block decomposition: grid = number of blocks, blockDim = BI.
// ---------------------------------------------------------------------------
// Where the last CTA of a MODE_FORCES_ONLY launch copies a call's results:
// `words` of src to host memory at dst, then a 1 into *done.
struct ResultMail {
  const int* src;
  int* dst;
  int words;
  int* done;
};

struct StateArgs {
  double* x;        // 3 x Npad, component-major (x | y | z)
  double* v;        // 3 x Npad
  double* f;        // 3 x Npad, forces
  double* tf;       // 3 x Npad, TVN averaged force (F_old + F_new)/2
  double* e;        // Npad per-particle pair energy sum  4eps sum [(s/r)^12-(s/r)^6]
  double* w;        // Npad per-particle virial sum  sum r.f
  int4* q;          // fixed-point shadow
  double4_32a* xd;      // FP64 position shadow
  int npad;         // stride between components
  const BlockInfo* blocks;
  const BoxArgs* boxes;
  DevScalars* sc;
  const int* sys_block_first;  // nsys + 1
  double* blk_part;            // nblocks x 8 partial sums
  const float* partial;        // pair-kernel partials
  int prec;                    // LJ_PREC_*
  int bi_threads;              // threads of the pair kernel's i-block (partial stride)
  DevRecord* records;          // per box ring (rec_cap entries each)
  int rec_stride;              // ring capacity per box
  int* status;
  int4* q_next;                // fused step: predictor shadow for the next step
  int* blk_cnt;                // fused step: segments finished per i-block
  int* glob_cnt;               // fused step: [2 + parity] pending-observables tickets
  int nblocks;                 // i-blocks of all boxes
  int nsys;                    // boxes
  int obs_slot;                // fused EVN: first block-partial slot of this step's K, V, W (0 or 4, by parity)
  double* row_part;            // row step (lj_rows.cu): 8 partial sums per CTA, in place of blk_part
  float4* force4;              // MODE_FORCES_ONLY of the row and unordered-pair kernels: (F, sum r^-12 - r^-6),
  float* pressure;             // and (4/6) sum s r^2, as calculateNForces returns them (ticket: blk_cnt[0])
  const ResultMail* mail;      // MODE_FORCES_ONLY: may be null
  int ticket;                  // fused: glob_cnt index of this step's pending-observables tickets (2 or 3)
};

enum StepMode { MODE_FORCES_ONLY = 0, MODE_EVN = 1, MODE_TVN = 2 };

// The pair kernel with the second half of the Verlet step fused into the
// last CTA of every i-block (epi = MODE_EVN or MODE_TVN).
struct FusedPairArgs {
  PairArgs pair;
  StateArgs st;
};

// Step of one box of kNewtonMinN particles or more over unordered pairs
// (lj_newton.cu; NewtonPlan).  The line lies where it overtakes the row step:
// us a step, rows / unordered pairs, N = 6000 31 / 36, N = 8000 48.9 / 48.7,
// N = 9000 64 / 59, N = 14 000 139 / 111.
constexpr int kNewtonMinN = 8192;
struct NewtonArgs {
  const int4* q;
  const DevScalars* sc;
  const NewtonTask* tasks;
  const int* block_part;  // per block of 256: first part of its i sums, count
  float* jpart;           // per tile t (block b = t / 8) b + 1 parts of 5 x 32, tile-major
  float* ipart;           // part (task + block): 5 x 256
  int n, ntasks;
};
cudaError_t newton_setup(int* ctas_per_sm);
// The j sums are 10 KB a particle at 2^18 (2.7 GB) and grow with n; larger
// boxes keep the stream-K kernel.
constexpr int kNewtonMaxN = 1 << 18;
constexpr int kNewtonWarps = 4;  // tasks of a CTA
cudaError_t launch_newton(const NewtonArgs& a, cudaStream_t st);
cudaError_t launch_newton_sum(const StateArgs& s, const NewtonArgs& a, int mode, cudaStream_t st);

// Row step of one smaller box (lj_rows.cu): ctas = 0 where it does not apply.
struct RowPlan {
  int rows, ctas;
  size_t smem;
};
RowPlan plan_rows(int n, int sms);
cudaError_t rows_setup();
// MODE_FORCES_ONLY: forces of s.q alone (force4, pressure; no box, state or observables).
cudaError_t launch_rows(const StateArgs& s, const RowPlan& p, int n, int mode, cudaStream_t st);
// parts: CTAs (row step) or tiles whose sums of tv^2 make chi
cudaError_t launch_rows_close(const StateArgs& s, int n, int parts, cudaStream_t st);

// Steps of one small box in one launch (lj_cluster.cu).
constexpr int kClusterMaxN = 512;
cudaError_t cluster_setup(bool* usable);
cudaError_t launch_cluster(const StateArgs& s, int n, int mode, int nsteps, cudaStream_t st);

// Arguments of the FP64 pair pass (lj_pairs64.cu; Pair64Plan).
struct Pair64Args {
  const double4_32a* xd;  // position shadow (x, y, z, 0)
  const Pair64Task* tasks;
  const Pair64Box* boxes64;
  const BoxArgs* boxes;
  double* part;
  int ntasks, group, parts, split, turns, nsys;  // turns = 32 / split
};
// BoxArgs::image_lo / image_hi of a period L (bits of two separations).
void fp64_image_bounds(double L, double invL, long long* lo, long long* hi);
cudaError_t launch_pairs64(const Pair64Args& a, cudaStream_t st);
// Its sums, the step's second half and the observables of every box (MODE_TVN:
// two launches).  carried: the pass ran at the drift that the previous step (or
// launch_predict) left in xd, and this one leaves the next; qhist (carried
// steps of periodic boxes, may be null): the new positions' fixed-point shadow.
cudaError_t launch_reduce64(const StateArgs& s, const Pair64Args& a, int nblocks, int mode, bool carried, int4* qhist,
                            cudaStream_t st);

cudaError_t launch_drift_mode(const StateArgs& s, int nblocks, int bi, int mode, cudaStream_t st);
cudaError_t launch_bbox(const StateArgs& s, int nblocks, int bi, cudaStream_t st);
cudaError_t launch_frame(const StateArgs& s, int nsys, bool only_nonperiodic, cudaStream_t st);
cudaError_t launch_quantize(const StateArgs& s, int nblocks, int bi, bool only_nonperiodic, cudaStream_t st);
cudaError_t launch_reduce(const StateArgs& s, int nblocks, int bi, int mode, cudaStream_t st);
cudaError_t launch_tvn_finish(const StateArgs& s, int nblocks, int bi, cudaStream_t st);
cudaError_t launch_observables(const StateArgs& s, int nsys, int mode, cudaStream_t st);
cudaError_t launch_velocity_hist(const StateArgs& s, int nblocks, int bi, double step, int nb,
                                 unsigned long long* counts, cudaStream_t st);
cudaError_t launch_predict(const StateArgs& s, int nblocks, int bi, cudaStream_t st);
cudaError_t launch_tvn_close(const StateArgs& s, int nblocks, int bi, cudaStream_t st);
cudaError_t launch_obs_finalize(const StateArgs& s, int nsys, cudaStream_t st);

// Fixed-point shadow of caller-owned float4 positions (lj_compat.cu), for the
// reference ABI and the allocation-free force entry point: writes q and the
// frame *sc, and clears *status if given.  Open boxes use blk (8 doubles per
// kFloat4Threads positions) and ticket (0 between launches).
constexpr int kFloat4Threads = 256;
cudaError_t launch_float4_shadow(const float4* pos, int n, int periodic, double L, DevScalars* sc, int* status,
                                 double* blk, int* ticket, int4* q, cudaStream_t st);

// Headless particle image (lj_render.cu): splat + shade into rgba (device).
cudaError_t launch_render(const double* x, int npad, int p0, int n, int axis, int W, int H, double L, double R,
                          unsigned long long* key, uint8_t* rgba, cudaStream_t st);

// Subsystem counters of the fluctuation runs (lj_counters_configure).
constexpr int kMaxCounterAlphas = 64;
struct CounterDev {
  int type;    // 0/1/2 slab x/y/z < alpha L; 3 cube around the centre; 4/5/6 |v_x|/|v_y|/|v_z| < alpha vmax
  int nalpha;  // alphas k = 0 .. nalpha-1
  int bin0;    // first bin of this counter in the per-step row
  int pad;
  double alpha_step;
  double vmax;
  double inv_bc;                 // 1 / (L alpha_step) (types 0-2) or 1 / (vmax alpha_step) (types 4-6)
  double tl[kMaxCounterAlphas];  // type 3: cube sides L alpha_k^(1/3)
};
// Device words of the counters (DevBuf<int> of kCtrWords): next ring row,
// steps since the last counted one, the interval, the ring's rows, and the
// per-launch ticket counter (0 between launches).
enum : int { kCtrNext = 0, kCtrPhase = 1, kCtrEvery = 2, kCtrCap = 3, kCtrTicket = 4, kCtrWords = 8 };
// One step of the counters in one launch (graph-capturable: everything that
// changes per step lives in `state`): the histogram of the counters' bin
// indices over the particles of box 0 into the step's ring row when the step
// is counted.  Row kCtrNext is zero before the launch.
cudaError_t launch_counters(const StateArgs& s, const CounterDev* cs, int nc, int nbins, int* state, int* ring, int n,
                            cudaStream_t st);
cudaError_t launch_unpack(const double* in, double* out, int n, int npad, cudaStream_t st);
cudaError_t launch_selftest_wait(int* status, cudaStream_t st);
// Up to three (N,3) interleaved <-> component-major [3][npad] transposes in one launch.
struct XyzArrays {
  const double* src[3];
  double* dst[3];
};
// `s` is read only with mb->finalize.
cudaError_t launch_pack_multi(const XyzArrays& a, int count, int n, int npad, const Mailbox* mb, const StateArgs& s,
                              cudaStream_t st);
// Upload of (N,3) positions / velocities (either may be NULL; either may be
// mapped host memory), in two launches.  Stage: every value checked (*bad
// receives the lowest index of a non-finite value, velocities after the 3n
// position values; it must hold 0x7f7f7f7f before) and written component-major
// to spos / svel ([3][npad] each).  Commit (grid = i-blocks): the staged
// arrays become x / v only if every value was finite; with `predict`, also
// the fused step's shadow of x + dt v + dt^2 F / 2 into s.q (periodic boxes).
cudaError_t launch_upload_stage(const double* pos, const double* vel, int n, int npad, double* spos, double* svel,
                                int* bad, cudaStream_t st);
cudaError_t launch_upload_commit(const StateArgs& s, int nblocks, int bi, const double* spos, const double* svel,
                                 const int* bad, bool predict, cudaStream_t st);
cudaError_t launch_scale_velocities(const StateArgs& s, int nblocks, int bi, int sysmode, double target,
                                    cudaStream_t st);

}  // namespace ljgb
