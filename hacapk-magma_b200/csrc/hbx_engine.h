// hbx_engine.h -- engine state behind the opaque hbx_hmat handle, and the
// kernel launchers shared by the hbx_* API and the HACApK drop-in symbols.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "hbx_plan.h"

namespace hbx {

// Partial-sum slots of the BiCGSTAB reductions (per CTA, compensated pairs).
enum : int {
  kSlotRhoR = 0,   // rh . r
  kSlotRR = 1,     // r . r
  kSlotRhAp = 2,   // rh . Ap
  kSlotAtT = 3,    // At . t
  kSlotAtAt = 4,   // At . At
  kSlotBB = 5,     // b . b
  kSlotAux = 6,    // scratch (true residual)
  kSlots = 8
};

// Solver scalars carried from one launch to the next.
struct BicgState {
  double alpha, zeta, rho, beta;
  double relres, bnorm;
  int iter, done, status, pad;
};

// What a solve reads back, in page-locked memory: the state after its last two
// launches, the true residual's square, the device error word.
struct SolveBack {
  BicgState state[2];
  double dot;
  int err, pad;
};

struct MatvecArgs {
  const uint8_t *stream;
  const RunRec *recs;
  const CtaInfo *ctas;
  const RunLite *lite;
  const double *x;
  const double *yin;
  double *y;
  double *zbu;
  const float *x32;  // FP32 engines: x rounded to float (gathered instead of x)
  float *zbu32;      // FP32 engines: zbu rounded to float (gathered by the U runs)
  uint64_t zbu_len;
  double alpha, beta;
  unsigned *gbar;
  int *err;
  unsigned long long timeout_ns;
  unsigned long long *prof;  // optional: per-CTA %globaltimer stamps [num_ctas][16], slots 0-5
  uint32_t keep_frac;        // fraction (of 2^16) of each CTA's stream kept in L2 between passes; 0: no hints
  uint32_t stall;            // test hook: the launch's grid barrier waits for one instance more than can
                             // complete, so its bounded waits expire (hbx_debug_stall_next_barrier)
  const int *skip;           // optional: the launch does nothing while *skip is set (a solver's done flag)
  // optional (block-diagonal engines): chunk g of CTA c covers instances
  // [lo, hi] = chunk_inst[chunk_base[c] + g] (lo | hi << 16); a chunk none of
  // whose instances is active (inst_pre: prefix counts of active instances,
  // count + 1 entries) is not copied, and the rows of inactive instances
  // come out undefined
  const uint32_t *chunk_inst, *chunk_base;
  const int *inst_pre;
};

struct BicgArgs {
  const uint8_t *stream;
  const RunRec *recs;
  const CtaInfo *ctas;
  const RunLite *lite;
  const Atom *atoms;
  double *zbu;      // [2][zbu_len]: one copy per H-matvec of a step
  uint64_t zbu_len;
  unsigned *gbar;
  int *err;
  unsigned long long timeout_ns;
  const double *b;
  double *u, *r, *rh, *p, *ap, *t, *at;
  float *p32, *t32, *zbu32;  // FP32 engines: float copies of the matvec inputs (zbu32: [2][zbu_len])
  double *part;   // [kSlots][num_ctas][2]
  BicgState *state;
  double *hist;   // relres per iteration (max_iter + 1 entries)
  unsigned long long *prof;  // optional: per-CTA %globaltimer stamps [num_ctas][16], slots 8-15
  double tol;
  int max_iter;
  int steps;           // steps of one launch, at most
  uint32_t keep_frac;  // as MatvecArgs::keep_frac
};

// Multi-RHS product on the tensor cores (hbx_mrhs.cu): Y = alpha*H*X +
// beta*Yin for kNrhs right-hand sides, rows of kNrhs values (RHS-contiguous).
constexpr int kNrhs = 64;
struct MatmatArgs {
  const uint8_t *stream;  // packed with pair_panels (FP32)
  const CtaInfo *ctas;
  const RunLite *lite;
  const uint32_t *cols;  // vector row of every panel column (x, or zbu for U runs), kNoCol: a zero column
  const float *x;     // [nd][kNrhs]
  const double *yin;  // [nd][kNrhs], read when beta != 0
  double *y;          // [nd][kNrhs]
  float *zbu;         // [zbu_len][kNrhs]
  double alpha, beta;
  unsigned *gbar;
  int *err;
  unsigned long long timeout_ns;
  const int *go;  // optional: the launch does nothing while *go is 0 (a solver's flag)
};
size_t matmat_smem_bytes();
cudaError_t configure_matmat();
cudaError_t launch_matmat(const MatmatArgs &a, int num_ctas, cudaStream_t s);
constexpr uint32_t kNoCol = 0xffffffffu;
// Forms MatmatArgs::cols from the run records (once per engine).
cudaError_t launch_matmat_cols(const RunRec *recs, const CtaInfo *ctas, int num_ctas, uint32_t *cols, cudaStream_t s);

// FP64 product with kNrhs right-hand sides of a single-vector FP64 engine
// (hbx_mm64.cu).  A unit: runs [r0, r0 + n0) and [r1, r1 + n1) of CTA `cta`.
struct Mm64Unit {
  uint32_t cta, r0, n0, r1, n1;
};
struct Mm64Args {
  const uint8_t *stream;
  const RunRec *recs;
  const CtaInfo *ctas;
  const Mm64Unit *units;
  uint32_t nunits;
  unsigned *next;  // unit counters of the two launches
  const double *x, *yin;
  double *y, *zbu;  // zbu: [zbu_len][kNrhs]
  double alpha, beta;
};
cudaError_t configure_mm64();
// The P units and the row-atom units of a plan, each in descending cost.
void mm64_units(const std::vector<CtaInfo> &ctas, const std::vector<RunLite> &lite, std::vector<Mm64Unit> &p,
                std::vector<Mm64Unit> &rest);
cudaError_t launch_mm64(const Mm64Args &a, const Mm64Unit *p, uint32_t np, const Mm64Unit *rest, uint32_t nrest,
                        cudaStream_t s);

// Multi-RHS BiCGSTAB (hbx_mrhs_solve.cu): scalars of one right-hand side.
struct MrScal {
  double alpha, zeta, rho, beta, rr, rtol;
  int active, iters, status, pad;
};
// One step for every right-hand side still running (7 launches, two of them
// the product through `matmat`); nothing is done once *any_active is 0.
struct MrStep {
  int nd, max_iter;
  MrScal *sc;
  int *any_active;
  unsigned *ticket;  // last-block counter of the reductions, zero between launches
  double *r, *rh, *p, *ap, *at, *x, *part;  // t lies in r between the step's two products
  float *f32;  // the product's input (p, then t, rounded to float)
  cudaError_t (*matmat)(void *ctx, const float *x, double *y, cudaStream_t s);
  void *ctx;
};
int mr_row_blocks(int nd);
cudaError_t mr_launch_norms(int nd, const double *v, double *part, unsigned *ticket, double *out, cudaStream_t s);
cudaError_t mr_launch_setup(const MrStep &a, const double *R, const double *thresh, const int *mask, cudaStream_t s);
cudaError_t mr_launch_step(const MrStep &a, cudaStream_t s);
cudaError_t mr_launch_transpose(int rows, int cols, const double *in, double *out, cudaStream_t s);
cudaError_t mr_launch_resid(int nd, const double *B, const double *HU, double *R, cudaStream_t s);
cudaError_t mr_launch_add(int nd, const int *mask, const double *D, double *U, cudaStream_t s);

// Batched BiCGSTAB over the instances of a block-diagonal engine
// (hbx_batch.cu); one MrScal per instance, rtol = the relative tolerance.
struct BtFlags {
  int any, done;    // some instance runs; none does (MatvecArgs::skip)
  unsigned ticket;  // last-block counter, zero between launches
};
struct BtCta {  // a CTA of the vector kernels
  int k;                           // its instance (-1: none)
  uint8_t size, rank, base, pad;   // CTAs of the instance, this one's place, the first one's rank in the cluster
};
struct BtGrid {
  const BtCta *map;  // on the device
  int ctas, cluster;
};
struct BtStep {
  int count, max_iter;
  BtGrid grid;
  const int *off;                // instance row offsets [count + 1]
  MrScal *sc;
  BtFlags *flags;
  int *pre;    // optional: prefix counts of active instances, refreshed by every step
  float *x32;  // FP32 / BF16 engines: the products' input as float (p, then t)
  double *r, *rh, *p, *ap, *t, *at, *u, *bnorm;
  cudaError_t (*matvec)(void *ctx, const double *x, double *y, cudaStream_t s);
  void *ctx;
};
// The CTAs of the instances at rows off[k]..off[k + 1]; returns the cluster size.
int bt_map(const std::vector<int> &off, std::vector<BtCta> &map);
cudaError_t bt_launch_norms(const BtGrid &g, const int *off, const double *x, double *out, cudaStream_t s);
cudaError_t bt_launch_init(const BtStep &a, const double *b, double tol, const double *rtol, cudaStream_t s);
cudaError_t bt_launch_mask(size_t n, const int *rinst, const int *flag, double *r, cudaStream_t s);
cudaError_t bt_launch_step(const BtStep &a, cudaStream_t s);

// Dot products of up to kMaxDots vector pairs per launch (hbx_gcr.cu;
// compensated per-block partials part[blocks][kMaxDots][2], summed in block
// order into out[k]); the GCR restart length is at most kMaxDots.
constexpr int kMaxDots = 64;
int gcr_dot_blocks(size_t n);
cudaError_t gcr_launch_dots(int k, const double *const *x, const double *const *y, size_t n, double *part,
                            double *out, cudaStream_t s);

// GCR(m) (hbx_gcr.cu; m_HACApK_solve.f90:506-571), state on the device.
struct GcrState {
  double bnorm, relres, tol, alpha;
  double capap[kMaxDots], beta[kMaxDots];
  int step, max_iter, done, status;
  unsigned ticket;  // last-block counter of the fused reductions
  int pad;
};
struct GcrVecs {
  const double *b;
  double *u, *r, *ar;  // ar: A r of the current step
  double *p, *ap;      // m slots of nd each
};
cudaError_t gcr_launch_init(const GcrVecs &v, size_t n, GcrState *st, double *part, double tol, int max_iter,
                            cudaStream_t s);
cudaError_t gcr_launch_alpha0(const GcrVecs &v, size_t n, GcrState *st, double *part, cudaStream_t s);
cudaError_t gcr_launch_update(const GcrVecs &v, size_t n, int ik, GcrState *st, double *part, cudaStream_t s);
cudaError_t gcr_launch_orth(const GcrVecs &v, size_t n, int ik, int ikn, GcrState *st, double *part,
                            cudaStream_t s);

// Pipelined BiCGSTAB (hbx_pipe.cu; HACApK_SOLVER_PIPE.c:144-600).  The state
// lives on the device so that a batch of steps runs as one captured graph.
struct PipeState {
  double alpha, beta, zeta, znorm, bnorm, relres, tol;
  int step, max_iter, done, status;
  unsigned ticket;  // last-block counter of the fused reductions
  int expired;      // a launch of k_pipe_steps found the error word set and did nothing
};
struct PipeVecs {
  const double *b;
  double *u, *r, *r0, *w, *t, *v, *p, *s, *z, *q, *y;
};
constexpr int kPipeVecs = 10;  // r, r0, w, t, v, p, s, z, q, y
cudaError_t pipe_launch_init(const PipeVecs &v, size_t n, PipeState *st, double *part, double *hist, double tol,
                             int max_iter, cudaStream_t s);
cudaError_t pipe_launch_a(const PipeVecs &v, size_t n, PipeState *st, double *part, cudaStream_t s);
cudaError_t pipe_launch_b(const PipeVecs &v, size_t n, PipeState *st, double *part, double *hist, cudaStream_t s);

// FP64 engines: up to `steps` steps in one launch (k_pipe_steps, hbx_kernels.cu).
struct PipeStepArgs {
  const uint8_t *stream;
  const RunRec *recs;
  const CtaInfo *ctas;
  const RunLite *lite;
  double *zbu;  // [2][zbu_len]: one copy per product of a step
  uint64_t zbu_len;
  unsigned *gbar;
  int *err;
  unsigned long long timeout_ns;
  uint32_t keep_frac;
  PipeVecs v;
  size_t n;
  PipeState *st;
  double *part, *hist;
  int nvb;  // blocks of the dots' grid (set by the launcher)
  int steps;
};
cudaError_t launch_pipe_steps(PipeStepArgs a, int num_ctas, cudaStream_t s);
// Up to this many rows a thread of k_pipe_steps has one element (two blocks of
// the dots' grid per CTA: 75,776 rows on 148 CTAs).  Beyond, the products are
// most of a step and the stand-alone vector kernels, with four times the warps,
// stream better (with several elements per thread a solve of 81,920 rows took
// 19.6 ms either way, of 327,680 114.1 ms in k_pipe_steps and 112.2 as launches).
inline size_t pipe_steps_max_rows(int num_ctas) { return (size_t)num_ctas * 512; }

// Static scratch of hbx_matvec_noalloc (hbx_kernels.cu): 256 bytes of
// barrier words, then room for kNoallocZbuMax zbu doubles.
constexpr size_t kNoallocScratchBytes = size_t(1) << 20;
constexpr size_t kNoallocCtlBytes = 256;
constexpr uint64_t kNoallocZbuMax = (kNoallocScratchBytes - kNoallocCtlBytes) / sizeof(double);
cudaError_t noalloc_scratch_address(void **ptr);

// The packed stream of `plan` formed on the device from the host leaves
// (hbx_pack.cu); a temporary of the leaves' size comes from `alloc`, whose
// cudaErrorMemoryAllocation is returned with nothing written.
cudaError_t pack_on_device(const stc_HACApK_leafmtxp *st, const Plan &plan, const RunRec *d_recs, const CtaInfo *d_ctas,
                           uint8_t *d_stream, cudaError_t (*alloc)(void *, size_t));

// Kernel launchers (hbx_kernels.cu).
size_t kernel_smem_bytes();
cudaError_t configure_kernels();
cudaError_t configure_step_kernels();     // the step kernels' translation unit
cudaError_t configure_step_kernels_lp();  // the FP32 / BF16 step kernels' unit
cudaError_t launch_bicg_steps_lp(const BicgArgs &a, int num_ctas, cudaStream_t s, int precision);
cudaError_t launch_matvec(const MatvecArgs &a, int num_ctas, cudaStream_t s, int precision);
cudaError_t launch_bicg_setup(const BicgArgs &a, int num_ctas, cudaStream_t s);
cudaError_t launch_bicg_steps(const BicgArgs &a, int num_ctas, cudaStream_t s, int precision);
cudaError_t launch_axpy(double alpha, const double *x, double *y, size_t n, cudaStream_t s);
cudaError_t launch_to_float(const double *x, float *y, size_t n, cudaStream_t s);
// n doubles of a0 to b0 and (when a1 is set) of a1 to b1, and (when w is set) the
// word *w to *wout; either side may be page-locked host memory.
cudaError_t launch_copy(const double *a0, double *b0, const double *a1, double *b1, const int *w, int *wout, size_t n,
                        cudaStream_t s);
// Host vectors up to this size go through page-locked memory and the copy
// kernel, longer ones by the runtime's copies of pageable memory.  y += H x with
// host vectors, the runtime's copies -> this: 81 KB 134 -> 99 us, 640 KB 442 ->
// 358, 4 MB 1,440 -> 1,300; 16 MB 5,700 -> 6,220 (one core copies the vectors).
constexpr size_t kIoBytes = 4 << 20;
// The slot's partials of x.y over own rows; then out[0] = the total (one block).
cudaError_t launch_dot(const BicgArgs &a, const double *x, const double *y, int slot, double *out,
                       int num_ctas, cudaStream_t s);

}  // namespace hbx

struct hbx_hmat {
  int device = 0;
  int num_ctas = 0;
  int transposed = 0;  // the packed stream holds H^T
  int nrhs = 1;        // right-hand sides per product (kNrhs: multi-RHS engine, hbx_matmat only)
  uint32_t *d_mcols = nullptr;  // multi-RHS engine: MatmatArgs::cols
  float *d_zbum = nullptr;  // multi-RHS engine: zbu for all right-hand sides [zbu_len][kNrhs]
  // multi-RHS solver workspace (hbx_bicgstab_multi)
  double *d_mrv = nullptr;      // r, rh, p, ap, at, x, R, and two kNrhs x nd scratch arrays
  float *d_mr32 = nullptr;      // nd x kNrhs
  double *d_mrpart = nullptr;   // [row blocks][2][kNrhs]
  hbx::MrScal *d_mrsc = nullptr;
  int *d_mrint = nullptr;       // any_active, mask[kNrhs], the reductions' ticket
  double *d_mrdbl = nullptr;    // thresholds[kNrhs], norms[kNrhs]
  void *h_mrpin = nullptr;      // pinned: MrScal[kNrhs], norms, thresholds, ints
  // FP64 product with kNrhs right-hand sides (hbx_mm64.cu), made by the first
  // multi-RHS solve that uses this engine: units, their counters, zbu
  hbx::Mm64Unit *d_mm64 = nullptr;
  uint32_t mm64_p = 0, mm64_rest = 0;
  unsigned *d_mm64_next = nullptr;
  double *d_mm64_zbu = nullptr;
  // block-diagonal batch of independent instances (hbx_create_batch)
  std::vector<int> inst_off;    // row offsets, count + 1 entries (empty: one instance)
  int *d_inst_off = nullptr;    // the same on the device
  int *d_rinst = nullptr;       // instance of every row
  // per-instance stream skipping (hbx_create_batch; MatvecArgs::chunk_inst):
  // the chunk table, each CTA's first entry, prefix counts of active
  // instances, and whether products skip inactive instances right now
  uint32_t *d_chunk_inst = nullptr, *d_chunk_base = nullptr;
  int *d_inst_pre = nullptr;
  int skip_inactive = 0;
  int merge_keep = -1;  // the planner's merged D+U setting in use
  int l2_keep_mb = 0;   // the L2 budget of the stream in use (MB; 0: no hints)
  void *d_rflag = nullptr;  // refined batch: per-instance flags and inner tolerances
  double *d_btv = nullptr;      // r, rh, p, ap, t, at (6 nd)
  hbx::MrScal *d_btsc = nullptr;
  double *d_btdbl = nullptr;    // bnorm [count], true norms [count], norms of the outer loop [count]
  hbx::BtFlags *d_btflags = nullptr;
  hbx::BtGrid btgrid{};         // the vector kernels' CTAs
  int *h_btany = nullptr;       // page-locked: any_active after the last two batches of steps
  hbx::Plan plan;
  uint8_t *d_stream = nullptr;
  hbx::RunRec *d_recs = nullptr;
  long long num_runs = 0;
  hbx::CtaInfo *d_ctas = nullptr;
  hbx::RunLite *d_lite = nullptr;
  hbx::Atom *d_atoms = nullptr;
  double *d_zbu = nullptr;
  unsigned *d_gbar = nullptr;
  int *d_err = nullptr;
  unsigned long long timeout_ns = 2000000000ull;
  uint32_t keep_frac = 0;  // fraction (of 2^16) of every CTA's stream kept in L2 between passes
  uint32_t stall_next = 0; // test hook: the next k_matvec launch's grid barrier cannot complete
  unsigned long long *d_prof = nullptr;  // phase stamps of the last matvec (HBX_PROFILE=1)
  double setup_seconds = 0.0;
  cudaStream_t stream = nullptr;  // used by the host-vector calls
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr, ev3 = nullptr, ev4 = nullptr, ev5 = nullptr;
  // host-vector staging
  double *d_x = nullptr, *d_y = nullptr;
  double *h_pin = nullptr;        // page-locked staging of short host vectors: 2*nd doubles and the error word
  // solver workspace
  double *d_work = nullptr;       // r, rh, p, ap, t, at, b, u  (8*nd)
  double *d_part = nullptr;
  double *d_dot = nullptr;
  hbx::BicgState *d_state = nullptr;
  hbx::SolveBack *h_back = nullptr;  // page-locked: what a solve reads back
  double *d_hist = nullptr;
  double *d_refine = nullptr;     // mixed-precision solve: outer residual and correction (2*nd)
  float *d_f32 = nullptr;         // FP32 engines: x, p, t (3*nd) and zbu (zbu_len) rounded to float
  int hist_cap = 0;
  // GCR(m): r, A r, p[m], Ap[m] (nd each); device state and its pinned copy;
  // per-block partials; the captured restart cycle(s)
  double *d_gcr = nullptr;
  int gcr_m = 0;
  hbx::GcrState *d_gcrs = nullptr, *h_gcrs = nullptr;
  double *d_gcrpart = nullptr;
  cudaGraphExec_t ggraph = nullptr;
  int ggraph_m = 0, ggraph_cycles = 0;
  const void *ggraph_key = nullptr;
  // pipelined BiCGSTAB: vectors (kPipeVecs*nd), device state, pinned copy,
  // per-block partials, relres history, captured step batch
  double *d_pipe = nullptr;
  hbx::PipeState *d_pstate = nullptr, *h_pstate = nullptr;
  double *d_ppart = nullptr, *d_phist = nullptr;
  int phist_cap = 0;
  cudaGraphExec_t pgraph = nullptr;
  int pgraph_batch = 0;
  const void *pgraph_key = nullptr;
};
