// hbx_kernels.cu -- persistent sm_100a kernels of the H-matvec / BiCGSTAB path.
//
// k_matvec      one H-matvec: y = alpha*H*x + beta*yin (HACApK_BATCH.c:47-255
//               replaced: one launch instead of ceil(n/5000) vbatched GEMVs per
//               phase, no atomics, no zeroing of zbu/zau).
// k_bicg_setup  r = b - H u has been formed by k_matvec; sets rh = r, p = Ap = 0
//               and the first reduction partials (HACApK_SOLVER.c:533-594).
// k_pipe_steps  pipelined BiCGSTAB steps (hbx_pipe.cu), several in one launch.
// k_bicg_steps  BiCGSTAB steps of HACApK_SOLVER.c:602-732, several in one
//               launch: both H-matvecs, the vector updates and all dot
//               products, with compensated (Dot2) partial sums reduced in a
//               fixed order.
//
// The file is compiled three times: as itself (k_matvec and the small vector
// kernels, 16 consumer warps), with HBX_STEP_TU and HBX_CONSUMER_WARPS=13
// (k_bicg_setup, the FP64 k_bicg_steps and the dot kernels): with fewer
// threads per CTA the step kernel gets the registers it needs without
// spilling, and its scalar phases synchronise fewer warps (C1 step 121.4 ->
// 115 us, while the standalone product is fastest with 16); and with
// HBX_STEP_TU, HBX_STEP_LP and HBX_CONSUMER_WARPS=kStepWarpsLp (the FP32 and
// BF16 k_bicg_steps, whose consumer warps form two groups like the FP32 and
// BF16 products').
//
// All kernels run one CTA per SM: consumer warps, a bulk-copy producer
// warp, kGatherWarps gather warps, a grid-barrier warp and a block-sum warp.
// The producer streams the CTA's packed runs through a shared-memory ring
// with cp.async.bulk; the consumers take every 16th panel of every run
// (rotated so the work stays balanced), multiply it by the run's staged
// vector and accumulate in registers; at a block end they park their partial
// sums and go on, and the block-sum warp adds them in a fixed order and
// writes the rows.  Grid-wide dependencies (zbu complete, dot products
// complete) use a bounded grid barrier; the launch is cooperative so every
// CTA is resident.
#include "hbx_device.cuh"
#include "hbx_dots.cuh"
#include "hbx_engine.h"

#include <algorithm>

namespace hbx {
namespace {

constexpr int NW = kConsumerWarps;
constexpr int kConsumerThreads = NW * 32;
// Consumer groups: the FP32 and BF16 product kernels split their warps into
// kProductGroups groups taking alternate runs; the FP64 product (whose
// summation order the drop-in's iteration counts follow, and which a CPU
// replay reproduces bit for bit) and the step kernels keep one group.
template <int kPrec>
constexpr int groups_of() {
  return ((NW == kProductWarps || NW == kStepWarpsLp) && kPrec != kFP64) ? kProductGroups : 1;
}
static_assert(kStages % kProductGroups == 0, "a stage slot always serves the same consumer group");
#ifdef HBX_STEP_LP
static_assert(NW == kStepWarpsLp, "the FP32 / BF16 step unit is built with kStepWarpsLp consumer warps");
#elif defined(HBX_STEP_TU)
static_assert(NW == kStepWarps, "the FP64 step unit is built with kStepWarps consumer warps");
#else
static_assert(NW == kProductWarps, "the product unit is built with kProductWarps consumer warps");
#endif

struct Smem {
  uint8_t *ring;
  uint64_t *full, *empty;
  double *red;     // [kRedSlots][NW][64] partial sums of a block end
  uint8_t *stage;  // [kStages][kStageBytes]
  RunLite *lite;   // the CTA's run summaries
  uint8_t *rec;    // [kGatherWarps][kRecSlots] run records
  double *scal;    // 64 doubles
  uint64_t *sfull, *sempty, *rfull;
  uint64_t *xready, *pdone, *gdone, *redfull, *rdone;
  unsigned *rsum;
};

__device__ __forceinline__ Smem smem_layout(uint8_t *base) {
  Smem s;
  s.ring = base + SharedLayout::ring;
  s.full = reinterpret_cast<uint64_t *>(base + SharedLayout::full);
  s.empty = reinterpret_cast<uint64_t *>(base + SharedLayout::empty);
  s.red = reinterpret_cast<double *>(base + SharedLayout::red);
  s.stage = base + SharedLayout::stage;
  s.lite = reinterpret_cast<RunLite *>(base + SharedLayout::lite);
  s.rec = base + SharedLayout::rec;
  s.scal = reinterpret_cast<double *>(base + SharedLayout::scal);
  s.sfull = reinterpret_cast<uint64_t *>(base + SharedLayout::sfull);
  s.sempty = reinterpret_cast<uint64_t *>(base + SharedLayout::sempty);
  s.rfull = reinterpret_cast<uint64_t *>(base + SharedLayout::rfull);
  s.xready = reinterpret_cast<uint64_t *>(base + SharedLayout::xready);
  s.pdone = reinterpret_cast<uint64_t *>(base + SharedLayout::pdone);
  s.gdone = reinterpret_cast<uint64_t *>(base + SharedLayout::gdone);
  s.redfull = reinterpret_cast<uint64_t *>(base + SharedLayout::redfull);
  s.rdone = reinterpret_cast<uint64_t *>(base + SharedLayout::rdone);
  s.rsum = reinterpret_cast<unsigned *>(base + SharedLayout::rsum);
  return s;
}

// Barriers (but the ring's: producer_start), the block-sum counter, the
// launch's first grid-barrier generation and the CTA's run summaries (`lite`,
// nr of them) in shared memory.  Thread t0 sets up the barriers; threads t0
// and up copy the summaries.  The caller synchronises the CTA afterwards.
__device__ __forceinline__ void init_cta_part(const Smem &s, const RunLite *lite, uint32_t nr, const unsigned *gbar,
                                              uint32_t t0, uint32_t group_warps) {
  if (threadIdx.x == t0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&s.sfull[i], 33);  // 32 cp.async arrivals of a gather warp + its lane 0
      mbar_init(&s.sempty[i], group_warps);  // the slot's runs belong to one consumer group
    }
    for (int i = 0; i < kGatherWarps * (int)kRecSlots; ++i) mbar_init(&s.rfull[i], 32);
    mbar_init(s.xready, 1);
    mbar_init(s.pdone, 1);
    mbar_init(s.gdone, 1);
    for (uint32_t i = 0; i < kRedSlots; ++i) mbar_init(&s.redfull[i], NW);
    mbar_init(s.rdone, 1);
    s.rsum[0] = 0;
    s.rsum[1] = grid_gen0(gbar);
    s.rsum[2] = 0;
    s.rsum[3] = 0;
    s.rsum[4] = 0;
    mbar_fence_init();
  }
  if (threadIdx.x < t0 || s.lite == lite) return;  // summaries read where they lie (see cta_smem)
  const uint4 *src = reinterpret_cast<const uint4 *>(lite);
  uint4 *dst = reinterpret_cast<uint4 *>(s.lite);
  for (uint32_t k = threadIdx.x - t0; k < nr; k += blockDim.x - t0) dst[k] = __ldg(src + k);
}

// The CTA's shared-memory layout; a CTA with more runs than the summary
// array holds reads its run summaries from global memory instead.
__device__ __forceinline__ Smem cta_smem(uint8_t *base, const RunLite *lite, uint32_t nr) {
  Smem s = smem_layout(base);
  if (nr > (uint32_t)kMaxCtaRuns) s.lite = const_cast<RunLite *>(lite);
  return s;
}

#ifndef HBX_STEP_TU
__device__ __forceinline__ void init_cta(const Smem &s, const RunLite *lite, uint32_t nr, const unsigned *gbar,
                                         uint32_t group_warps) {
  init_cta_part(s, lite, nr, gbar, 0, group_warps);
  __syncthreads();
}
#endif

// ---- grid-barrier warp: once per pass, after the CTA's P blocks are summed
// (pdone), arrive on the grid barrier, wait for it and release the U runs
// (gdone).  The barrier latency stays off the consumer and gather warps.
// Pass p uses grid-barrier instance (p / 2) * kstep + (p odd ? k1 : k0) of the
// launch.  It returns early once the solve has stopped (rsum[4]).
// `beyond` > 0 (a test hook) waits for an instance that no launch of this
// grid completes, so the bounded waits of the whole CTA expire.
__device__ __forceinline__ void sync_warp(unsigned *gbar, uint32_t npass, uint32_t k0, uint32_t k1, uint32_t kstep,
                                          const Smem &sm, int *err, uint64_t tmo, uint32_t beyond = 0) {
  for (uint32_t p = 0; p < npass; ++p) {
    if (!mbar_wait(sm.pdone, p & 1, tmo)) {
      atomicOr(err, kErrPipeline);
      return;  // the waits on gdone are bounded too
    }
    if (ld_acquire_s(&sm.rsum[4])) return;
    const unsigned target = grid_target(sm.rsum[1], (p / 2) * kstep + ((p & 1) ? k1 : k0) + beyond, gridDim.x);
    grid_arrive(gbar, target);  // a release: the CTA's zbu stores (before pdone) are visible grid-wide
    if (!grid_wait(gbar, target, tmo)) {
      atomicOr(err, kErrGridBarrier);
      return;
    }
    st_release_s(&sm.rsum[3], p + 1);  // the gather warps' U runs of pass p may start
    mbar_arrive(sm.gdone);
  }
}

// x of the launch's pass `pass` is ready: the gather warps' count, then the
// block-sum warp's barrier.  One thread.
__device__ __forceinline__ void signal_xready(const Smem &sm, unsigned pass) {
  st_release_s(&sm.rsum[2], pass + 1);
  mbar_arrive(sm.xready);
}

// Where the block sums of one H-matvec pass go.
struct PassOut {
  double alpha, beta;
  const double *yin;
  double *y, *zbu;
  float *zbu32;     // FP32 engines: zbu rounded to float (what the U runs gather)
};

// End of a block for a consumer warp: park its row sums (rows lane and
// lane + 32) in red slot nb mod kRedSlots, once the block-sum warp has
// emptied it, and arrive on the slot's barrier, `arrivals` times.  Returns
// false after a timed-out wait.
__device__ __forceinline__ bool block_end(double t0, double t1, uint32_t nb, uint32_t arrivals, const Smem &sm,
                                          int *err, uint64_t tmo) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t slot = nb % kRedSlots;
  auto free_slot = [&]() { return ld_acquire_s(sm.rsum) + kRedSlots > nb; };
  if (nb >= kRedSlots && !__all_sync(0xffffffffu, free_slot())) {
    const uint64_t ts = gtimer();
    while (!__all_sync(0xffffffffu, free_slot())) {
      if (__any_sync(0xffffffffu, gtimer() - ts > tmo)) {
        if (lane == 0) atomicOr(err, kErrPipeline);
        return false;
      }
    }
  }
  double *rb = sm.red + slot * (NW * 64) + w * 64;
  rb[lane] = t0;
  rb[32 + lane] = t1;
  __syncwarp();
  if (lane == 0) mbar_arrive(&sm.redfull[slot], arrivals);
  return true;
}

// p[0], p[64], ... of N warps, added in warp order.
template <int N>
__device__ __forceinline__ double warp_order_sum(const double *p) {
  double s = p[0];
#pragma unroll
  for (int k = 1; k < N; ++k) s += p[k * 64];
  return s;
}

// A row's sum s of a D, DU or U block.
__device__ __forceinline__ void put_row(const PassOut &o, uint32_t kind, uint32_t row, double s) {
  if (kind == kRunU) {
    o.y[row] = fma(o.alpha, s, o.y[row]);
  } else {  // an atom's first (a merged one: only) block
    double v = o.alpha * s;
    if (o.beta != 0.0) v = fma(o.beta, o.yin[row], v);
    o.y[row] = v;
  }
}

// ---- block-sum warp: for every block end of every pass, in order, wait
// until all consumer warps parked their partial sums, add them in warp order
// and write the rows -- P: zbu = s;  D: y = alpha*s + beta*yin;  U: y +=
// alpha*s (the atom's D block was summed before, in this same order) --
// then free the slot.  After the pass's last P block it signals pdone (the
// CTA's zbu rows are complete), after the pass's last block rdone.
template <int kPrec, class Outs>  // outs(pass): where that pass's sums go
__device__ __forceinline__ void sum_warp(uint32_t nr, uint32_t npass, uint32_t nblk_p, Outs outs, const Smem &sm,
                                         int *err, uint64_t tmo) {
  constexpr int kGroups = groups_of<kPrec>(), kGroupWarps = NW / kGroups;
  const uint32_t lane = threadIdx.x & 31;
  uint32_t nb = 0;
  for (uint32_t pass = 0; pass < npass; ++pass) {
    const PassOut o = outs(pass);
    // Not before the pass has started: rdone must not run a phase ahead of
    // the consumers' wait on it (a CTA without blocks would otherwise
    // complete both passes' phases at once).
    if (!warp_wait(sm.xready, pass & 1, tmo)) {
      if (lane == 0) atomicOr(err, kErrPipeline);
      return;
    }
    if (ld_acquire_s(&sm.rsum[4])) {  // no such pass: wake the grid-barrier warp too
      if (lane == 0) mbar_arrive(sm.pdone);
      return;
    }
    uint32_t np_done = 0;
    for (uint32_t r = 0; r < nr; ++r) {
      const RunLite L = sm.lite[r];
      if (!(L.flags & kLast)) continue;
      const uint32_t slot = nb % kRedSlots;
      if (!warp_wait(&sm.redfull[slot], (nb / kRedSlots) & 1, tmo)) {
        if (lane == 0) atomicOr(err, kErrPipeline);
        return;  // the consumers' bounded waits end the launch
      }
      const uint32_t kind = L.flags & 0xffu;
      const double *rb = sm.red + slot * (NW * 64);
      if constexpr (kPrec == kFP64) {
        for (uint32_t i = lane; i < L.nrow; i += 32) {
          const double s = warp_order_sum<NW>(rb + i);
          if (kind == kRunP) o.zbu[L.out + i] = s;
          else put_row(o, kind, L.out + i, s);
        }
      } else {
        // a block of one run has sums of that run's group alone
        const bool single = L.flags & kFirst;
        if (single) rb += (pass * nr + r) % kGroups * (kGroupWarps * 64);
        auto total = [&](uint32_t i) {
          double s = warp_order_sum<kGroupWarps>(rb + i);
          if (!single)
            for (int k = kGroupWarps; k < NW; ++k) s += rb[k * 64 + i];
          return s;
        };
        if (kind == kRunP) {
          float *z = o.zbu32 + L.out;  // U runs gather the float copy alone
          const double s0 = total(lane);
          if (L.nrow > 32) {
            const double s1 = total(lane + 32);
            z[lane] = (float)s0;
            if (lane + 32 < L.nrow) z[lane + 32] = (float)s1;
          } else if (lane < L.nrow) {
            z[lane] = (float)s0;
          }
        } else {
          const double s = total(lane);
          if (lane < L.nrow) put_row(o, kind, L.out + lane, s);
        }
      }
      ++nb;
      __syncwarp();
      if (lane == 0) {
        __threadfence_block();
        st_release_s(sm.rsum, nb);  // the slot may be refilled
        if (kind == kRunP && ++np_done == nblk_p) mbar_arrive(sm.pdone);  // the CTA's zbu rows are complete
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(sm.rdone);
  }
}

// One H-matvec pass of a consumer warp over the CTA's runs (the pass starts
// at absolute ring chunk R.base and is K chunks long).  For every run the
// warp waits for its staged vector, multiplies its panels (every 16th,
// rotated), gives the stage slot back and, at a block end, parks its row
// sums for the block-sum warp.  Before it can block, a warp gives back every
// ring chunk below the run it is about to process, so no wait holds a chunk
// another warp needs.  nb counts the block ends over the launch.
//
// A run costs every warp that takes part in it some 300 instructions beside
// its panels (the waits, the ring's bookkeeping, the parking), which bounds the
// FP32 and BF16 kernels; there a warp has nothing to do with the other group's
// runs, unless a block has runs of both.  (With every warp parking at every
// block end a BiCGSTAB step took 78.2 us instead of 75.1 at 9,999 rows of leaf
// size 15 in FP32, 71.5 instead of 69.0 in BF16, 265 instead of 258 at 81,920.)
template <int kPrec>
__device__ __forceinline__ void consume_pass(Ring &R, uint32_t K, uint32_t nr, uint32_t &nb, uint32_t pass,
                                             const Smem &sm, int *err, uint64_t tmo) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool bad = R.bad;
  double t0 = 0.0, t1 = 0.0;  // this lane's block sums: rows lane and lane + 32
  constexpr int kGroups = groups_of<kPrec>(), kGroupWarps = NW / kGroups;
  const uint32_t grp = kGroups == 1 ? 0u : (uint32_t)w / kGroupWarps;
  const uint32_t wl = kGroups == 1 ? (uint32_t)w : (uint32_t)w % kGroupWarps;
  for (uint32_t r = 0; r < nr; ++r) {
    const RunLite L = sm.lite[r];
    const uint32_t g = pass * nr + r, slot = g % kStages;
    const bool own = kGroups == 1 || g % kGroups == grp;  // a run of this warp's group
    if (own) {
      R.release_below(R.base + (L.pos >> kChunkLog));
      // Every warp of the group observes every phase of the slot's barrier,
      // panels or not: a warp that skipped phases could take an older
      // completed phase for the one it waits on.
      if (!bad && !warp_wait(&sm.sfull[slot], (g / kStages) & 1, tmo)) {
        bad = true;
        if (lane == 0) atomicOr(err, kErrPipeline);
      }
      if (!bad) run_panels<kPrec, kGroupWarps>(L, smem_u32(sm.stage + slot * kStageBytes), R, wl, t0, t1);
      bad = bad || R.bad;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.sempty[slot]);
    }
    if (L.flags & kLast) {
      // A block of one run concerns its group alone, which arrives for the others.
      const bool single = kGroups > 1 && (L.flags & kFirst);
      if (!single || own) {
        R.release_below(R.base + ((L.pos + 16u * L.nrow * L.npanel) >> kChunkLog));
        if (!bad && !block_end(t0, t1, nb, single ? kGroups : 1, sm, err, tmo)) bad = true;
      }
      ++nb;
      t0 = 0.0;
      t1 = 0.0;
    }
  }
  R.release_below(R.base + K);
}

// The consumer warps' part of one H-matvec pass: the P-done signal of a CTA
// without P blocks, the pass, then the wait for the block-sum warp (every
// row of the pass is written) and, in warp 0, for the pass's grid barrier
// (the caller's next grid barrier must not start before it completes).
template <int kPrec>
__device__ __forceinline__ void matvec_pass(Ring &R, uint32_t K, uint32_t nr, uint32_t &nb, uint32_t pass,
                                            uint32_t nblk_p, const Smem &sm, int *err, uint64_t tmo) {
  if (nblk_p == 0 && threadIdx.x == 0) mbar_arrive(sm.pdone);
  consume_pass<kPrec>(R, K, nr, nb, pass, sm, err, tmo);
  if (!warp_wait(sm.rdone, pass & 1, tmo) && (threadIdx.x & 31) == 0) atomicOr(err, kErrPipeline);
  if (threadIdx.x < 32 && !warp_wait(sm.gdone, pass & 1, tmo) && threadIdx.x == 0) atomicOr(err, kErrGridBarrier);
}

// Bytes at the head of a CTA's stream read with the evict_last policy: a
// fraction keep_frac / 2^16 of the stream, whole chunks (0: no cache hints).
__device__ __forceinline__ uint32_t keep_bytes(uint32_t stream_bytes, uint32_t keep_frac) {
  if (keep_frac == 0) return 0;
  const uint64_t b = ((uint64_t)stream_bytes * keep_frac) >> 16;
  const uint64_t r = (b + kChunkBytes - 1) & ~(uint64_t)(kChunkBytes - 1);
  return r > 0xffffffffull ? 0xffffffffu : (uint32_t)r;
}

// Grid-barrier instance k of the launch for this CTA, by one whole warp.
__device__ __forceinline__ void arrive_and_wait(unsigned *gbar, unsigned k, int *err, uint64_t timeout_ns,
                                                const Smem &sm) {
  const unsigned target = grid_target(sm.rsum[1], k, gridDim.x);
  if ((threadIdx.x & 31) == 0) grid_arrive(gbar, target);
  __syncwarp();
  if (!grid_wait_warp(gbar, target, timeout_ns) && (threadIdx.x & 31) == 0) atomicOr(err, kErrGridBarrier);
}

// Full grid barrier (instance k of the launch) among the consumer warps of
// every CTA: what their threads wrote before it is read after it (bar.sync,
// then the arriving thread's release; no fence of their own).
__device__ __forceinline__ void grid_sync(unsigned *gbar, unsigned k, int *err, uint64_t timeout_ns, const Smem &sm) {
  named_bar(1, kConsumerThreads);
  if (threadIdx.x < 32) arrive_and_wait(gbar, k, err, timeout_ns, sm);
  named_bar(1, kConsumerThreads);
}


// kPrec: storage precision of the factors; FP32 and BF16 engines gather the
// float copies of the vectors.
#ifndef HBX_STEP_TU
template <int kPrec>
__global__ void __launch_bounds__(kThreads, 1) k_matvec(MatvecArgs a) {
  constexpr bool kF32 = kPrec != kFP64;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (a.skip && *(volatile const int *)a.skip) return;  // set by an earlier launch: the same on every CTA
  const CtaInfo ci = a.ctas[blockIdx.x];
  const uint32_t nr = ci.nr_p + ci.nr_d + ci.nr_u;
  const Smem sm = cta_smem(smem_raw, a.lite + ci.rec_begin, nr);
  const uint64_t t_start = a.prof ? gtimer() : 0;
  uint32_t issued0 = 0;
  const StreamSrc ss{a.stream + ci.stream_off, ci.stream_bytes, keep_bytes(ci.stream_bytes, a.keep_frac),
                     a.chunk_inst ? a.chunk_inst + a.chunk_base[blockIdx.x] : nullptr, a.inst_pre};
  if (threadIdx.x == kProducerWarp * 32) issued0 = producer_start(ss, 1, sm.ring, sm.full, sm.empty);
  init_cta(sm, a.lite + ci.rec_begin, nr, a.gbar, NW / groups_of<kPrec>());
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t K = (ci.stream_bytes + kChunkBytes - 1) >> kChunkLog;
  if (w == kProducerWarp) {
    if (lane == 0 && K > 0)
      producer_run(ss, 1, issued0, sm.ring, sm.full, sm.empty, a.err, a.timeout_ns);
    return;
  }
  if (w >= kGatherWarp0 && w < kSyncWarp) {
    const void *xs = kF32 ? static_cast<const void *>(a.x32) : static_cast<const void *>(a.x);
    const void *zs = kF32 ? static_cast<const void *>(a.zbu32) : static_cast<const void *>(a.zbu);
    const GatherCtx c{a.recs + ci.rec_begin, nr, ci.nr_p + ci.nr_d, 1, xs, xs, zs, zs, a.err, a.timeout_ns};
    gather_warp<kPrec>(c, sm, (uint32_t)(w - kGatherWarp0));
    return;
  }
  if (w == kSyncWarp) {
    if (lane == 0) sync_warp(a.gbar, 1, 0, 0, 0, sm, a.err, a.timeout_ns, a.stall ? 1u : 0u);
    return;
  }
  if (w == kSumWarp) {
    sum_warp<kPrec>(nr, 1, ci.nblk_p,
             [&](uint32_t) { return PassOut{a.alpha, a.beta, a.yin, a.y, a.zbu, kF32 ? a.zbu32 : nullptr}; }, sm, a.err,
             a.timeout_ns);
    return;
  }
  if (threadIdx.x == 0) signal_xready(sm, 0);  // x is an input: ready from the start
  uint32_t nb = 0;
  Ring R{sm.ring, sm.full, sm.empty, 0, 0, 0, a.timeout_ns, a.err, false};
  matvec_pass<kPrec>(R, K, nr, nb, 0, ci.nblk_p, sm, a.err, a.timeout_ns);
  if (a.prof && threadIdx.x == 0) {
    a.prof[blockIdx.x * 16 + 0] = t_start;
    a.prof[blockIdx.x * 16 + 5] = gtimer();
  }
}

// ---------------------------------------------------------- pipelined BiCGSTAB
// Grid-barrier instances of one pipelined step, in order: z and the y.q, y.y
// partials complete, zbu of v = H z, v, then w and its five partials, zbu of
// t = H w, t.
enum : unsigned {
  kGridZ = 0, kGridPassV = 1, kGridV = 2, kGridW = 3, kGridPassT = 4, kGridT2 = 5, kGridPipeStep = 6
};
// Partials of dot j: slots [kPipeSlot + j][dot_blocks] of 16-byte pairs.
constexpr int kPipeSlotA = 0, kPipeSlotB = 2;

// The block partials of K dots in hbx_dots.cuh's order (blocks of kDotThreads
// threads, an element per thread): eight consumer warps stand for block `vb`,
// so the totals are those of the stand-alone kernels bit for bit.
template <int K>
__device__ __forceinline__ void pipe_partials(const PipeStepArgs &a, int slot0, uint32_t vb, Acc2 (&acc)[K], const Smem &sm) {
  static_assert(NW == 2 * kDotThreads / 32, "two blocks of the dots' grid per CTA");
  constexpr int kBlockWarps = kDotThreads / 32;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, wb = w % kBlockWarps;
  double *sc = sm.red + w / kBlockWarps * (kBlockWarps * K * 2);  // free: every warp has waited for the block-sum warp
#pragma unroll
  for (int k = 0; k < K; ++k) {
    acc[k] = warp_merge(acc[k]);
    if (lane == 0) {
      sc[(wb * K + k) * 2 + 0] = acc[k].s;
      sc[(wb * K + k) * 2 + 1] = acc[k].c;
    }
  }
  named_bar(1, kConsumerThreads);
  if (wb == 0 && lane < K && vb < (uint32_t)a.nvb) {
    Acc2 t{sc[lane * 2], sc[lane * 2 + 1]};
    for (int q = 1; q < kBlockWarps; ++q) t = acc2_merge(t, Acc2{sc[(q * K + lane) * 2], sc[(q * K + lane) * 2 + 1]});
    reinterpret_cast<double2 *>(a.part)[(size_t)(slot0 + lane) * a.nvb + vb] = make_double2(t.s, t.c);
  }
}

// pair_total of hbx_dots.cuh over a slot's partials (a whole warp), the loads
// of five chunks of 32 under way together.
__device__ __forceinline__ double pipe_total(const PipeStepArgs &a, int slot) {
  constexpr int kBatch = 5;
  const int lane = threadIdx.x & 31;
  const double2 *part = reinterpret_cast<const double2 *>(a.part) + (size_t)slot * a.nvb;
  Acc2 t{0.0, 0.0};
  for (int b0 = 0; b0 < a.nvb; b0 += 32 * kBatch) {
    Acc2 v[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int b = b0 + 32 * k + lane;
      v[k] = Acc2{0.0, 0.0};
      if (b < a.nvb) {
        const double2 x = __ldcg(part + b);
        v[k] = Acc2{x.x, x.y};
      }
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k)
      if (b0 + 32 * k < a.nvb) t = acc2_merge(t, warp_merge(v[k]));
  }
  return t.s + t.c;
}

// Up to a.steps pipelined BiCGSTAB steps (the arithmetic and the summation
// order of k_pipe_a, k_matvec, k_pipe_b, k_matvec: hbx_pipe.cu).  As four
// launches a step paid four launch boundaries, two products with a cold ring
// and two tickets on which the last block started its totals; here six grid
// barriers take their place, the ring runs on through the vector work, and no
// graph is captured for a new u.  An element is always the same thread's, so of
// the vectors only v and t (written by rows), z and w (gathered) cross CTAs.
// The early end of a launch is k_bicg_steps'.  Solves to 1e-8, launches -> this:
// N = 320 430 -> 306 us, 1,280 715 -> 571, 5,120 1,250 -> 1,050, 6,001 (leaf size
// 32, ragged) 1,814 -> 1,527, 20,480 3,660 -> 3,410 (60 products of 265 MB at 6.55
// TB/s: 2,430; the six barriers of a step and the vector work: some 20 us).
__global__ void __launch_bounds__(kThreads, 1) k_pipe_steps(const __grid_constant__ PipeStepArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // An earlier launch ended the solve.  (A CTA's threads decide together, as in
  // k_bicg_steps: where waits run out the first CTA may end it in this launch.)
  if (__syncthreads_or(*(volatile const int *)&a.st->done)) return;
  const CtaInfo ci = a.ctas[blockIdx.x];
  const uint32_t nr = ci.nr_p + ci.nr_d + ci.nr_u;
  const Smem sm = cta_smem(smem_raw, a.lite + ci.rec_begin, nr);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t npass = 2u * (uint32_t)a.steps;
  const StreamSrc ss{a.stream + ci.stream_off, ci.stream_bytes, keep_bytes(ci.stream_bytes, a.keep_frac)};
  uint32_t issued0 = 0;
  if (threadIdx.x == kProducerWarp * 32) issued0 = producer_start(ss, npass, sm.ring, sm.full, sm.empty);
  init_cta(sm, a.lite + ci.rec_begin, nr, a.gbar, NW);
  const uint32_t K = (ci.stream_bytes + kChunkBytes - 1) >> kChunkLog;
  if (w == kProducerWarp) {
    if (lane == 0 && K > 0)
      producer_run(ss, npass, issued0, sm.ring, sm.full, sm.empty, a.err, a.timeout_ns, &sm.rsum[4]);
    return;
  }
  const PipeVecs &v = a.v;
  if (w >= kGatherWarp0 && w < kSyncWarp) {
    const GatherCtx c{a.recs + ci.rec_begin, nr, ci.nr_p + ci.nr_d, npass, v.z, v.w, a.zbu, a.zbu + a.zbu_len, a.err,
                      a.timeout_ns};
    gather_warp<kFP64>(c, sm, (uint32_t)(w - kGatherWarp0));
    return;
  }
  if (w == kSyncWarp) {
    if (lane == 0) sync_warp(a.gbar, npass, kGridPassV, kGridPassT, kGridPipeStep, sm, a.err, a.timeout_ns);
    return;
  }
  if (w == kSumWarp) {
    sum_warp<kFP64>(nr, npass, ci.nblk_p,
                    [&](uint32_t pass) {
                      return PassOut{1.0, 0.0, nullptr, (pass & 1) ? v.t : v.v, a.zbu + ((pass & 1) ? a.zbu_len : 0),
                                     nullptr};
                    },
                    sm, a.err, a.timeout_ns);
    return;
  }
  // scal: alpha, beta, zeta, r.r0, done, steps taken; [8..12] the five totals
  enum { kAlpha = 0, kBeta, kZeta, kZnorm, kDone, kStep, kTot = 8 };
  Ring R{sm.ring, sm.full, sm.empty, 0, 0, 0, a.timeout_ns, a.err, false};
  uint32_t nb = 0;
  if (threadIdx.x == 0) {
    sm.scal[kAlpha] = __ldcg(&a.st->alpha);
    sm.scal[kBeta] = __ldcg(&a.st->beta);
    sm.scal[kZeta] = __ldcg(&a.st->zeta);
    sm.scal[kZnorm] = __ldcg(&a.st->znorm);
    sm.scal[kStep] = (double)__ldcg(&a.st->step);  // (state is written after the first grid barrier)
    sm.scal[kDone] = *(volatile const int *)a.err ? 1.0 : 0.0;  // an earlier wait ran out
  }
  named_bar(1, kConsumerThreads);
  // The launch's later passes do not follow: wake the warps that wait for one.
  auto stop = [&]() {
    if (threadIdx.x == 0) {
      st_release_s(&sm.rsum[4], 1u);
      signal_xready(sm, 0x7ffffffeu);
    }
    named_bar(1, kConsumerThreads);
    if (lane == 0) mbar_arrive(&sm.empty[R.released % kRingChunks]);
  };
  auto finish = [&](int status) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.st->status = status;
      a.st->done = 1;
    }
  };
  if (sm.scal[kDone] != 0.0) {
    // done stays unset: a CTA that has yet to start must come this way too
    if (blockIdx.x == 0 && threadIdx.x == 0) a.st->expired = 1;
    stop();
    return;
  }
  auto mul = [](double x, double y) { return __dmul_rn(x, y); };
  auto add = [](double x, double y) { return __dadd_rn(x, y); };

  // One product per turn, its call in one place: the loop over the panels keeps
  // the registers that it has in k_matvec when little else is live.  (Called in
  // two places, or as a function, it spilled inside the runs: 81,920 rows 21.7 and
  // 22.6 ms instead of 19.6.)
  for (uint32_t pass = 0; pass < npass; ++pass) {
    const unsigned k0 = (pass >> 1) * kGridPipeStep;
    // (volatile: kept live through the product, the element's index and
    // addresses spill inside the loop over the panels)
    uint32_t tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    const uint32_t vb = blockIdx.x + (tid >= kConsumerThreads / 2 ? gridDim.x : 0u);
    const uint32_t i = vb * kDotThreads + tid % kDotThreads;
    const bool own = i < (uint32_t)a.n;
    if ((pass & 1u) == 0) {
      if (pass > 0) grid_sync(a.gbar, k0 - kGridPipeStep + kGridT2, a.err, a.timeout_ns, sm);
      // p, s, z (copies on the first step), q, y; y.q, y.y.  (Reading ahead of
      // the barrier gained nothing: the values spilled.)
      Acc2 acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
      if (own) {
        const double alpha = sm.scal[kAlpha], beta = sm.scal[kBeta], nzeta = -sm.scal[kZeta], t = __ldcg(&v.t[i]);
        const double r = __ldcg(&v.r[i]), wv = __ldcg(&v.w[i]), vv = __ldcg(&v.v[i]);
        double p = __ldcg(&v.p[i]), s = __ldcg(&v.s[i]), z = __ldcg(&v.z[i]);
        if (sm.scal[kStep] == 0.0) {
          p = r, s = wv, z = t;
        } else {
          p = add(mul(beta, add(p, mul(nzeta, s))), r);
          s = add(mul(beta, add(s, mul(nzeta, z))), wv);
          z = add(mul(beta, add(z, mul(nzeta, vv))), t);
        }
        const double q = add(r, mul(-alpha, s)), y = add(wv, mul(-alpha, z));
        v.z[i] = z;
        v.p[i] = p;
        v.s[i] = s;
        v.q[i] = q;
        v.y[i] = y;
        dot2_add(acc[0], y, q);
        dot2_add(acc[1], y, y);
      }
      pipe_partials<2>(a, kPipeSlotA, vb, acc, sm);
      grid_sync(a.gbar, k0 + kGridZ, a.err, a.timeout_ns, sm);
      if (threadIdx.x == 0) signal_xready(sm, pass);
      // zeta while the gathers start; a zeta that is not finite ends the solve
      // after this product, before u changes
      if (w < 2) {
        const double d = pipe_total(a, kPipeSlotA + w);
        if (lane == 0) sm.scal[kTot + w] = d;
      }
    } else {
      grid_sync(a.gbar, k0 + kGridV, a.err, a.timeout_ns, sm);
      const double alpha = sm.scal[kAlpha], zeta = __ddiv_rn(sm.scal[kTot], sm.scal[kTot + 1]);
      if (blockIdx.x == 0 && threadIdx.x == 0) a.st->zeta = zeta;
      if (!isfinite(zeta)) {  // y = 0 (HACApK_SOLVER_PIPE.c:433 divides unchecked)
        finish(HBX_ERR_BREAKDOWN);
        stop();
        return;
      }
      // u, r, w; r.r0, w.r0, s.r0, z.r0, r.r
      Acc2 acc[5] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
      if (own) {
        const double q = __ldcg(&v.q[i]), y = __ldcg(&v.y[i]), r0 = __ldcg(&v.r0[i]), t = __ldcg(&v.t[i]);
        const double p = __ldcg(&v.p[i]), s = __ldcg(&v.s[i]), z = __ldcg(&v.z[i]), u = __ldcg(&v.u[i]);
        const double wv = add(mul(-zeta, add(t, mul(-alpha, __ldcg(&v.v[i])))), y);
        const double r = add(q, mul(-zeta, y));
        v.w[i] = wv;
        v.r[i] = r;
        v.u[i] = add(add(u, mul(alpha, p)), mul(zeta, q));
        dot2_add(acc[0], r, r0);
        dot2_add(acc[1], wv, r0);
        dot2_add(acc[2], s, r0);
        dot2_add(acc[3], z, r0);
        dot2_add(acc[4], r, r);
      }
      pipe_partials<5>(a, kPipeSlotB, vb, acc, sm);
      grid_sync(a.gbar, k0 + kGridW, a.err, a.timeout_ns, sm);
      if (w < 5) {
        const double d = pipe_total(a, kPipeSlotB + w);
        if (lane == 0) sm.scal[kTot + w] = d;
      }
      named_bar(1, kConsumerThreads);
      if (threadIdx.x == 0) {
        const int step = (int)sm.scal[kStep] + 1;
        const double znorm = sm.scal[kTot];
        const double beta = mul(__ddiv_rn(alpha, zeta), __ddiv_rn(znorm, sm.scal[kZnorm]));
        const double den =
            __dsub_rn(add(sm.scal[kTot + 1], mul(beta, sm.scal[kTot + 2])), mul(mul(beta, zeta), sm.scal[kTot + 3]));
        const double alpha_new = __ddiv_rn(znorm, den);
        const double bnorm = __ldcg(&a.st->bnorm);
        const double rel = bnorm > 0.0 ? __ddiv_rn(__dsqrt_rn(sm.scal[kTot + 4]), bnorm) : 0.0;
        int done = 1, status = HBX_OK;
        if (*(volatile const int *)a.err) status = HBX_ERR_TIMEOUT;  // a wait ran out: no more of them
        else if (rel < __ldcg(&a.st->tol)) status = HBX_OK;
        else if (!isfinite(rel) || !isfinite(alpha_new) || !isfinite(beta)) status = HBX_ERR_BREAKDOWN;
        else if (step >= __ldcg(&a.st->max_iter)) status = HBX_ERR_NOT_CONVERGED;
        else done = 0;
        sm.scal[kAlpha] = alpha_new;
        sm.scal[kBeta] = beta;
        sm.scal[kZeta] = zeta;
        sm.scal[kZnorm] = znorm;
        sm.scal[kDone] = done;
        sm.scal[kStep] = (double)step;
        if (blockIdx.x == 0) {
          a.st->znorm = znorm;
          a.st->beta = beta;
          a.st->alpha = alpha_new;
          a.st->relres = rel;
          a.st->step = step;
          a.hist[step] = rel;
          if (done) finish(status);
        }
      }
      named_bar(1, kConsumerThreads);
      if (sm.scal[kDone] != 0.0) {
        stop();
        return;
      }
      if (threadIdx.x == 0) signal_xready(sm, pass);
    }
    R.base = pass * K;
    matvec_pass<kFP64>(R, K, nr, nb, pass, ci.nblk_p, sm, a.err, a.timeout_ns);  // v = H z, then t = H w
  }
}

#endif  // !HBX_STEP_TU

#ifdef HBX_STEP_TU
// ---------------------------------------------------------------- BiCGSTAB
template <class F>
__device__ __forceinline__ void for_own_rows(const Atom *atoms, const CtaInfo &ci, F f) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t q = w; q < ci.n_atoms; q += NW) {
    const Atom A = atoms[ci.atom_begin + q];
    if ((uint32_t)lane < A.h) f(A.r0 + lane);
  }
}

// The same over the warp's atoms after its first one (index w + NW, ...).
template <class F>
__device__ __forceinline__ void for_more_rows(const Atom *atoms, const CtaInfo &ci, F f) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t q = w + NW; q < ci.n_atoms; q += NW) {
    const Atom A = atoms[ci.atom_begin + q];
    if ((uint32_t)lane < A.h) f(A.r0 + lane);
  }
}

// The partials of a slot lie back to back over the CTAs, 16 bytes each: every
// CTA reads all of them after a grid barrier, 148 warps at once, and with one
// 128-byte line per CTA (all its slots together) that took 3.5 us, of which the
// 19 lines of a slot take under one.
__device__ __forceinline__ double2 *part_of(double *part, int ncta, int slot, int cta) {
  return reinterpret_cast<double2 *>(part) + (size_t)slot * ncta + cta;
}

// Per-CTA compensated partial sums of NS dot products over the owned rows.
// acc[] holds the calling thread's partials; the result goes to slots slot0+k.
template <int NSL>
__device__ __forceinline__ void cta_partials(Acc2 (&acc)[NSL], double *part, int slot0, const Smem &sm) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NSL; ++k) acc[k] = warp_merge(acc[k]);
  double *sc = sm.red;  // reuse: [NW][NSL][2]
  named_bar(1, kConsumerThreads);  // red may still be read by an atom reduction
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NSL; ++k) {
      sc[(w * NSL + k) * 2 + 0] = acc[k].s;
      sc[(w * NSL + k) * 2 + 1] = acc[k].c;
    }
  }
  named_bar(1, kConsumerThreads);
  if (w == 0 && lane < NSL) {
    Acc2 t{sc[lane * 2], sc[lane * 2 + 1]};
    for (int q = 1; q < NW; ++q) t = acc2_merge(t, Acc2{sc[(q * NSL + lane) * 2], sc[(q * NSL + lane) * 2 + 1]});
    *part_of(part, gridDim.x, slot0 + lane, blockIdx.x) = make_double2(t.s, t.c);
    __threadfence();
  }
  named_bar(1, kConsumerThreads);
}

// Total of one slot over all CTAs, same operation order in every CTA (full warp).
// (The loads of a lane are issued together, then merged in CTA order; a
// merge with a zero pair leaves the sum unchanged.)
__device__ __forceinline__ double reduce_slot(const double *part, int ncta, int slot) {
  constexpr int kBatch = 5;
  const int lane = threadIdx.x & 31;
  Acc2 a{0.0, 0.0};
  for (int c0 = 0; c0 < ncta; c0 += 32 * kBatch) {
    Acc2 v[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int c = c0 + lane + 32 * k;
      v[k] = Acc2{0.0, 0.0};
      if (c < ncta) {
        const double2 x = __ldcg(part_of(const_cast<double *>(part), ncta, slot, c));
        v[k] = Acc2{x.x, x.y};
      }
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) a = acc2_merge(a, v[k]);
  }
  a = warp_merge(a);
  return a.s + a.c;
}

// Totals of N slots at once (full warp), each as reduce_slot sums it: the
// loads of all slots are under way together.
template <int N>
__device__ __forceinline__ void reduce_slots(const double *part, int ncta, const int (&slot)[N], double (&tot)[N]) {
  constexpr int kBatch = 5;
  const int lane = threadIdx.x & 31;
  Acc2 a[N];
#pragma unroll
  for (int q = 0; q < N; ++q) a[q] = Acc2{0.0, 0.0};
  for (int c0 = 0; c0 < ncta; c0 += 32 * kBatch) {
    Acc2 v[N][kBatch];
#pragma unroll
    for (int q = 0; q < N; ++q)
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const int c = c0 + lane + 32 * k;
        v[q][k] = Acc2{0.0, 0.0};
        if (c < ncta) {
          const double2 x = __ldcg(part_of(const_cast<double *>(part), ncta, slot[q], c));
          v[q][k] = Acc2{x.x, x.y};
        }
      }
#pragma unroll
    for (int q = 0; q < N; ++q)
#pragma unroll
      for (int k = 0; k < kBatch; ++k) a[q] = acc2_merge(a[q], v[q][k]);
  }
#pragma unroll
  for (int q = 0; q < N; ++q) {
    a[q] = warp_merge(a[q]);
    tot[q] = a[q].s + a[q].c;
  }
}

// Grid-barrier instances of one BiCGSTAB step, in order: p complete, zbu of
// the first H-matvec complete, the r^.Ap partials, t complete, zbu of the
// second H-matvec, the At.t / At.At partials, the r^.r / r.r partials.
enum : unsigned {
  kGridP = 0, kGridPass0 = 1, kGridAlpha = 2, kGridT = 3, kGridPass1 = 4, kGridZeta = 5, kGridEnd = 6, kGridStep = 7
};

// The CTA's compensated partials of NSL dots to slots slot0 + k, then
// grid-barrier instance `inst`, all in warp 0 after one barrier of the CTA: the
// partials are all that the others wait for, and warp 0 goes straight on to
// their totals (the other warps wait for those at the caller's next barrier).
// The caller's warps have waited for the block-sum warp (rdone), so sm.red is
// free.
template <int NSL>
__device__ __forceinline__ void share_partials(Acc2 (&acc)[NSL], double *part, int slot0, unsigned *gbar, unsigned inst,
                                               int *err, uint64_t timeout_ns, const Smem &sm) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NSL; ++k) acc[k] = warp_merge(acc[k]);
  double *sc = sm.red;  // reuse: [NW][NSL][2]
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NSL; ++k) {
      sc[(w * NSL + k) * 2 + 0] = acc[k].s;
      sc[(w * NSL + k) * 2 + 1] = acc[k].c;
    }
  }
  named_bar(1, kConsumerThreads);
  if (w != 0) return;
  if (lane < NSL) {
    Acc2 t{sc[lane * 2], sc[lane * 2 + 1]};
    for (int q = 1; q < NW; ++q) t = acc2_merge(t, Acc2{sc[(q * NSL + lane) * 2], sc[(q * NSL + lane) * 2 + 1]});
    *part_of(part, gridDim.x, slot0 + lane, blockIdx.x) = make_double2(t.s, t.c);
  }
  __syncwarp();
  arrive_and_wait(gbar, inst, err, timeout_ns, sm);
}

#ifndef HBX_STEP_LP
__global__ void __launch_bounds__(kThreads, 1) k_bicg_setup(BicgArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const Smem sm = smem_layout(smem_raw);
  if ((threadIdx.x >> 5) >= NW) return;
  const CtaInfo ci = a.ctas[blockIdx.x];
  Acc2 acc[3] = {{0, 0}, {0, 0}, {0, 0}};
  for_own_rows(a.atoms, ci, [&](uint32_t r) {
    const double rv = a.r[r];
    a.rh[r] = rv;
    a.p[r] = 0.0;
    a.ap[r] = 0.0;
    dot2_add(acc[0], rv, rv);
    dot2_add(acc[1], rv, rv);
    const double bv = a.b[r];
    dot2_add(acc[2], bv, bv);
  });
  // slots 0,1 then 5
  Acc2 a01[2] = {acc[0], acc[1]};
  cta_partials<2>(a01, a.part, kSlotRhoR, sm);
  Acc2 a5[1] = {acc[2]};
  cta_partials<1>(a5, a.part, kSlotBB, sm);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    BicgState st{};
    *a.state = st;
  }
}
#endif

// Up to a.steps BiCGSTAB steps.  One launch per step paid a launch boundary
// and a cold start -- barriers, run summaries, the first chunks of the stream
// -- every step; within a launch the ring stays full from step to step and a
// grid barrier takes their place.  When the stop test ends the solve before
// a.steps, the warps that run ahead are told (rsum[4]) and woken: the producer
// by one more emptied slot, the gather and block-sum warps by the signal of a
// pass that does not follow, the grid-barrier warp by the block-sum warp.
// HBM bounds the passes; the seven barriers of a step bound small matrices.
// Time of a step, one launch per step -> this: N = 320 27.3 -> 20.5 us, 1,280
// 38.6 -> 31.1, 5,120 48.8 -> 41.8, 20,480 119 -> 109.5 (two passes of 265 MB
// at 6.55 TB/s: 81).
template <int kPrec>
__global__ void __launch_bounds__(kThreads, 1) k_bicg_steps(BicgArgs a) {
  constexpr bool kF32 = kPrec != kFP64;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // An earlier launch ended the solve (or its waits ran out).  The first CTA may
  // end it in this launch before another has started, so a CTA's threads decide
  // together.
  if (__syncthreads_or(*(volatile const int *)&a.state->done)) return;
  const CtaInfo ci = a.ctas[blockIdx.x];
  const uint32_t nr = ci.nr_p + ci.nr_d + ci.nr_u;
  const Smem sm = cta_smem(smem_raw, a.lite + ci.rec_begin, nr);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ncta = gridDim.x;
  const uint32_t npass = 2u * (uint32_t)a.steps;
  auto stamp = [&](int k) {
    if (a.prof && threadIdx.x == 0) a.prof[blockIdx.x * 16 + 8 + k] = gtimer();
  };
  // A consumer warp's first owned atom and this lane's row of it: r, p and t
  // stay in registers through the launch, the other vectors' entries are read
  // ahead of the barrier before their use (the rows of further atoms are read
  // where needed).
  const Atom a0 = (w < NW && (uint32_t)w < ci.n_atoms) ? a.atoms[ci.atom_begin + w] : Atom{0, 0};
  const bool own0 = (uint32_t)lane < a0.h;
  const uint32_t row0 = a0.r0 + lane;
  double c_r = 0.0, c_p = 0.0, c_t = 0.0;
  if (own0) {
    c_r = a.r[row0];
    c_p = __ldcg(&a.p[row0]);  // see S1
  }
  // the producer starts the stream of the first H-matvec while the other
  // threads set up the CTA
  const StreamSrc ss{a.stream + ci.stream_off, ci.stream_bytes, keep_bytes(ci.stream_bytes, a.keep_frac)};
  uint32_t issued0 = 0;
  if (threadIdx.x == kProducerWarp * 32) issued0 = producer_start(ss, npass, sm.ring, sm.full, sm.empty);
  init_cta_part(sm, a.lite + ci.rec_begin, nr, a.gbar, 128, NW / groups_of<kPrec>());
  __syncthreads();

  const uint32_t K = (ci.stream_bytes + kChunkBytes - 1) >> kChunkLog;
  if (w == kProducerWarp) {
    if (lane == 0 && K > 0)
      producer_run(ss, npass, issued0, sm.ring, sm.full, sm.empty, a.err, a.timeout_ns, &sm.rsum[4]);
    return;
  }
  if (w >= kGatherWarp0 && w < kSyncWarp) {
    const void *x0 = kF32 ? static_cast<const void *>(a.p32) : static_cast<const void *>(a.p);
    const void *x1 = kF32 ? static_cast<const void *>(a.t32) : static_cast<const void *>(a.t);
    const void *z0 = kF32 ? static_cast<const void *>(a.zbu32) : static_cast<const void *>(a.zbu);
    const void *z1 =
        kF32 ? static_cast<const void *>(a.zbu32 + a.zbu_len) : static_cast<const void *>(a.zbu + a.zbu_len);
    const GatherCtx c{a.recs + ci.rec_begin, nr, ci.nr_p + ci.nr_d, npass, x0, x1, z0, z1, a.err, a.timeout_ns};
    gather_warp<kPrec>(c, sm, (uint32_t)(w - kGatherWarp0));
    return;
  }
  if (w == kSyncWarp) {
    if (lane == 0) sync_warp(a.gbar, npass, kGridPass0, kGridPass1, kGridStep, sm, a.err, a.timeout_ns);
    return;
  }
  // The two H-matvecs of a step write separate zbu copies: a CTA may still
  // gather the first's when another writes the second's.
  if (w == kSumWarp) {
    sum_warp<kPrec>(nr, npass, ci.nblk_p,
             [&](uint32_t pass) {
               const size_t z = (pass & 1) ? a.zbu_len : 0;
               return PassOut{1.0, 0.0, nullptr, (pass & 1) ? a.at : a.ap, a.zbu + z, kF32 ? a.zbu32 + z : nullptr};
             },
             sm, a.err, a.timeout_ns);
    return;
  }
  Ring R{sm.ring, sm.full, sm.empty, 0, 0, 0, a.timeout_ns, a.err, false};
  uint32_t nb = 0;
  bool broke = false;  // the last step broke down and formed no new partials
  // the previous step's alpha, zeta, rho and count: scal[24..27] (identical in every CTA)

  for (int it = 0; it <= a.steps; ++it) {
    const unsigned k0 = (unsigned)it * kGridStep;
    const double l_ap = own0 ? a.ap[row0] : 0.0;
    // ---- S0: scalars of the previous step; stop test at the top of the loop
    // (HACApK_SOLVER.c:602-603).  Every CTA computes identical values.  (The
    // step before has passed the grid barrier of its partials; one that broke
    // down formed none, and those of the step before it stand.)
    if (it == 0 && threadIdx.x == 0) {
      sm.scal[24] = __ldcg(&a.state->alpha);
      sm.scal[25] = __ldcg(&a.state->zeta);
      sm.scal[26] = __ldcg(&a.state->rho);
      sm.scal[27] = (double)__ldcg(&a.state->iter);
    }
    if (w == 0) {
      const int expired = lane == 0 ? *(volatile const int *)a.err : 0;
      double tot[3];
      reduce_slots<3>(a.part, ncta, {kSlotRhoR, kSlotRR, kSlotBB}, tot);
      const double rho_new = tot[0], rr = tot[1], bb = tot[2];
      if (lane == 0) {
        const double alpha = sm.scal[24], zeta = sm.scal[25], rho = sm.scal[26];
        const int iter = (int)sm.scal[27];
        const double bnorm = sqrt(bb);
        const double relres = (bnorm > 0.0) ? sqrt(rr) / bnorm : 0.0;
        int done = 0, status = HBX_OK;
        double beta = 0.0;
        if (expired) { done = 1; status = HBX_ERR_TIMEOUT; }  // a wait ran out: no more of them
        else if (broke) { done = 1; status = HBX_ERR_BREAKDOWN; }
        // NaN or Inf in b or x0 shows in b.b or r.r before the first step
        else if (!isfinite(bb) || !isfinite(rr)) { done = 1; status = iter == 0 ? HBX_ERR_NONFINITE : HBX_ERR_BREAKDOWN; }
        else if (relres < a.tol) { done = 1; status = HBX_OK; }
        else if (!isfinite(relres)) { done = 1; status = HBX_ERR_BREAKDOWN; }
        else if (iter >= a.max_iter) { done = 1; status = HBX_ERR_NOT_CONVERGED; }
        else if (iter > 0) {
          // beta = -alpha/zeta * (rh.r_new)/znormold with the reference's sign
          // flips (HACApK_SOLVER.c:650-655, :699, :724) = (alpha/zeta) rho_new/rho_old
          beta = (alpha / zeta) * (rho_new / rho);
          if (!isfinite(beta)) { done = 1; status = HBX_ERR_BREAKDOWN; }
        }
        sm.scal[0] = done;
        sm.scal[2] = beta;
        sm.scal[3] = zeta;
        sm.scal[4] = rho_new;
        sm.scal[5] = relres;
        sm.scal[7] = bnorm;
        if (done && blockIdx.x == 0) {
          a.state->status = status;
          a.state->relres = relres;
          a.state->bnorm = bnorm;
          a.state->done = 1;
        }
      }
    }
    named_bar(1, kConsumerThreads);
    if (sm.scal[0] != 0.0 || it == a.steps) {
      if (it < a.steps) {  // the launch's later passes do not follow
        if (threadIdx.x == 0) {
          st_release_s(&sm.rsum[4], 1u);
          signal_xready(sm, 0x7ffffffeu);
        }
        named_bar(1, kConsumerThreads);
        if (lane == 0) mbar_arrive(&sm.empty[R.released % kRingChunks]);
      }
      return;
    }
    const double beta = sm.scal[2], zeta_prev = sm.scal[3];
    stamp(0);

    // ---- S1: p = r + beta*(p - zeta*Ap)  (p = r on the first step)
    if (own0) {
      c_p = (beta == 0.0) ? c_r : fma(-zeta_prev, l_ap, c_p) * beta + c_r;
      a.p[row0] = c_p;
      if (kF32) a.p32[row0] = (float)c_p;
    }
    if (beta == 0.0) {
      for_more_rows(a.atoms, ci, [&](uint32_t r) {
        const double v = a.r[r];
        a.p[r] = v;
        if (kF32) a.p32[r] = (float)v;
      });
    } else {
      for_more_rows(a.atoms, ci, [&](uint32_t r) {
        // p through L2 only: a line of p cached in L1 here could hold rows of
        // another CTA that the gather warps read after it rewrote them
        const double v = fma(-zeta_prev, a.ap[r], __ldcg(&a.p[r])) * beta;
        const double pv = v + a.r[r];
        a.p[r] = pv;
        if (kF32) a.p32[r] = (float)pv;
      });
    }
    grid_sync(a.gbar, k0 + kGridP, a.err, a.timeout_ns, sm);
    if (threadIdx.x == 0) signal_xready(sm, 2u * it);  // p complete grid-wide: the step's first pass may be gathered
    stamp(1);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      const int iter = (int)sm.scal[27];
      a.state->iter = iter + 1;
      a.state->beta = beta;
      a.state->rho = sm.scal[4];
      a.state->relres = sm.scal[5];
      a.state->bnorm = sm.scal[7];
      a.hist[iter] = sm.scal[5];
    }

    // ---- S2: Ap = H p;  rh . Ap
    R.base = 2u * it * K;
    matvec_pass<kPrec>(R, K, nr, nb, 2u * it, ci.nblk_p, sm, a.err, a.timeout_ns);
    stamp(2);
    double c_ap = 0.0;
    {
      Acc2 acc[1] = {{0, 0}};
      if (own0) {
        c_ap = a.ap[row0];
        dot2_add(acc[0], a.rh[row0], c_ap);
      }
      for_more_rows(a.atoms, ci, [&](uint32_t r) { dot2_add(acc[0], a.rh[r], a.ap[r]); });
      share_partials<1>(acc, a.part, kSlotRhAp, a.gbar, k0 + kGridAlpha, a.err, a.timeout_ns, sm);
    }
    if (w == 0) {
      const double zden = reduce_slot(a.part, ncta, kSlotRhAp);
      if (lane == 0) sm.scal[8] = sm.scal[4] / zden;
    }
    named_bar(1, kConsumerThreads);
    const double alpha = sm.scal[8];
    stamp(3);

    // ---- S3: t = r - alpha*Ap
    if (own0) {
      c_t = fma(-alpha, c_ap, c_r);
      a.t[row0] = c_t;
      if (kF32) a.t32[row0] = (float)c_t;
    }
    for_more_rows(a.atoms, ci, [&](uint32_t r) {
      const double v = fma(-alpha, a.ap[r], a.r[r]);
      a.t[r] = v;
      if (kF32) a.t32[r] = (float)v;
    });
    grid_sync(a.gbar, k0 + kGridT, a.err, a.timeout_ns, sm);
    if (threadIdx.x == 0) signal_xready(sm, 2u * it + 1u);  // t complete grid-wide: the second pass may be gathered
    stamp(4);

    // ---- S4: At = H t;  At . t,  At . At
    R.base += K;
    matvec_pass<kPrec>(R, K, nr, nb, 2u * it + 1u, ci.nblk_p, sm, a.err, a.timeout_ns);
    stamp(5);
    double c_at = 0.0, c_u = 0.0, c_rh = 0.0;
    {
      Acc2 acc[2] = {{0, 0}, {0, 0}};
      if (own0) {
        c_at = a.at[row0];
        c_u = a.u[row0];
        c_rh = a.rh[row0];
        dot2_add(acc[0], c_at, c_t);
        dot2_add(acc[1], c_at, c_at);
      }
      for_more_rows(a.atoms, ci, [&](uint32_t r) {
        const double atv = a.at[r];
        dot2_add(acc[0], atv, a.t[r]);
        dot2_add(acc[1], atv, atv);
      });
      share_partials<2>(acc, a.part, kSlotAtT, a.gbar, k0 + kGridZeta, a.err, a.timeout_ns, sm);
    }
    double sums[2] = {0.0, 0.0};
    if (w == 0) reduce_slots<2>(a.part, ncta, {kSlotAtT, kSlotAtAt}, sums);
    if (threadIdx.x == 0) {
      const double zeta = (sums[1] != 0.0) ? sums[0] / sums[1] : 0.0;
      sm.scal[9] = zeta;
      sm.scal[24] = alpha;
      sm.scal[25] = zeta;
      sm.scal[26] = sm.scal[4];
      sm.scal[27] += 1.0;
      if (blockIdx.x == 0) {
        a.state->alpha = alpha;
        a.state->zeta = zeta;
      }
    }
    named_bar(1, kConsumerThreads);
    const double zeta = sm.scal[9];
    stamp(6);

    // ---- S5: u += alpha*p + zeta*t;  r = t - zeta*At;  rh . r,  r . r
    // A breakdown (alpha or zeta not finite: r^.Ap or At.At zero or
    // overflowing, which HACApK_SOLVER.c:650, :694 divide by unchecked) keeps
    // u and r of the previous step; the stop test then ends the solve with
    // HBX_ERR_BREAKDOWN.
    broke = !isfinite(alpha) || !isfinite(zeta);
    if (!broke) {
      Acc2 acc[2] = {{0, 0}, {0, 0}};
      if (own0) {
        c_u = fma(zeta, c_t, fma(alpha, c_p, c_u));
        a.u[row0] = c_u;
        c_r = fma(-zeta, c_at, c_t);
        a.r[row0] = c_r;
        dot2_add(acc[0], c_rh, c_r);
        dot2_add(acc[1], c_r, c_r);
      }
      for_more_rows(a.atoms, ci, [&](uint32_t r) {
        const double uv = fma(alpha, a.p[r], a.u[r]);
        a.u[r] = fma(zeta, a.t[r], uv);
        const double rv = fma(-zeta, a.at[r], a.t[r]);
        a.r[r] = rv;
        dot2_add(acc[0], a.rh[r], rv);
        dot2_add(acc[1], rv, rv);
      });
      share_partials<2>(acc, a.part, kSlotRhoR, a.gbar, k0 + kGridEnd, a.err, a.timeout_ns, sm);
    }
    stamp(7);
  }
}

// A slot's partials over own rows, then (block 0 of a second launch) the total.
#ifndef HBX_STEP_LP
__global__ void __launch_bounds__(kThreads, 1) k_dot_partial(BicgArgs a, const double *x, const double *y, int slot) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const Smem sm = smem_layout(smem_raw);
  if ((threadIdx.x >> 5) >= NW) return;
  const CtaInfo ci = a.ctas[blockIdx.x];
  Acc2 acc[1] = {{0, 0}};
  for_own_rows(a.atoms, ci, [&](uint32_t r) { dot2_add(acc[0], x[r], y[r]); });
  cta_partials<1>(acc, a.part, slot, sm);
}
#endif

// y = (float)x: the input of an FP32 engine's matvec.
#endif  // HBX_STEP_TU

#ifndef HBX_STEP_TU
__global__ void k_to_float(const double *x, float *y, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = (float)x[i];
}

// Short host vectors to the device and back: PCIe latency bounds it.  A copy of
// pageable memory by the runtime takes 15 us and more (81 KB); through page-locked
// memory, read and written across PCIe by this kernel, both vectors of a call and
// the error word take one launch each way.
__global__ void k_copy(const double *a0, double *b0, const double *a1, double *b1, const int *w, int *wout, size_t n) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  for (size_t k = i; k < n; k += stride) {
    const double v = a0[k];
    if (a1) b1[k] = a1[k];
    b0[k] = v;
  }
  if (w && i == 0) *wout = *w;
}

// y += a * x (the refinement update of the mixed-precision solve).
__global__ void k_axpy(double a, const double *x, double *y, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = fma(a, x[i], y[i]);
}

#endif  // !HBX_STEP_TU

#ifdef HBX_STEP_TU
#ifndef HBX_STEP_LP
__global__ void k_dot_total(const double *part, int ncta, int slot, double *out) {
  const double v = reduce_slot(part, ncta, slot);
  if (threadIdx.x == 0) *out = v;
}
#endif

#endif  // HBX_STEP_TU

}  // namespace

#ifndef HBX_STEP_TU
// ---- fixed scratch for hbx_matvec_noalloc -------------------------------
// One 1 MiB array per device, held by every GPU that loads this library until
// the process exits: [0, 256) barrier words, [256, end) the zbu segments.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];

// Host side: the device address of g_noalloc_scratch on the current device.
cudaError_t noalloc_scratch_address(void **ptr) { return cudaGetSymbolAddress(ptr, g_noalloc_scratch); }

size_t kernel_smem_bytes() { return SharedLayout::bytes; }

cudaError_t configure_kernels() {
  const int smem = (int)SharedLayout::bytes;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(k_matvec<kFP64>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_pipe_steps, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_matvec<kFP32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_matvec<kBF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  return configure_step_kernels();
}

#endif  // !HBX_STEP_TU

template <class Args>
static cudaError_t launch_coop(void (*kern)(Args), const Args &a, int num_ctas, cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(num_ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = SharedLayout::bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, a);
}

#ifndef HBX_STEP_TU
cudaError_t launch_matvec(const MatvecArgs &a, int num_ctas, cudaStream_t s, int precision) {
  if (precision == kBF16) return launch_coop(k_matvec<kBF16>, a, num_ctas, s);
  return precision == kFP32 ? launch_coop(k_matvec<kFP32>, a, num_ctas, s) : launch_coop(k_matvec<kFP64>, a, num_ctas, s);
}

cudaError_t launch_pipe_steps(PipeStepArgs a, int num_ctas, cudaStream_t s) {
  a.nvb = dot_blocks(a.n);
  return launch_coop(k_pipe_steps, a, num_ctas, s);
}

cudaError_t launch_to_float(const double *x, float *y, size_t n, cudaStream_t s) {
  k_to_float<<<296, 256, 0, s>>>(x, y, n);
  return cudaGetLastError();
}

cudaError_t launch_copy(const double *a0, double *b0, const double *a1, double *b1, const int *w, int *wout, size_t n,
                        cudaStream_t s) {
  const unsigned blocks = (unsigned)std::min<size_t>(148, (n + 255) / 256);
  k_copy<<<std::max(1u, blocks), 256, 0, s>>>(a0, b0, a1, b1, w, wout, n);
  return cudaGetLastError();
}

cudaError_t launch_axpy(double alpha, const double *x, double *y, size_t n, cudaStream_t s) {
  k_axpy<<<296, 256, 0, s>>>(alpha, x, y, n);
  return cudaGetLastError();
}
#elif !defined(HBX_STEP_LP)
cudaError_t configure_step_kernels() {
  const int smem = (int)SharedLayout::bytes;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(k_bicg_setup, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_bicg_steps<kFP64>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_dot_partial, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  return configure_step_kernels_lp();
}

cudaError_t launch_bicg_setup(const BicgArgs &a, int num_ctas, cudaStream_t s) {
  k_bicg_setup<<<num_ctas, kThreads, SharedLayout::bytes, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_bicg_steps(const BicgArgs &a, int num_ctas, cudaStream_t s, int precision) {
  if (precision != kFP64) return launch_bicg_steps_lp(a, num_ctas, s, precision);
  return launch_coop(k_bicg_steps<kFP64>, a, num_ctas, s);
}

cudaError_t launch_dot(const BicgArgs &a, const double *x, const double *y, int slot, double *out, int num_ctas,
                       cudaStream_t s) {
  k_dot_partial<<<num_ctas, kThreads, SharedLayout::bytes, s>>>(a, x, y, slot);
  k_dot_total<<<1, 32, 0, s>>>(a.part, num_ctas, slot, out);
  return cudaGetLastError();
}
#else
// The FP32 and BF16 step kernels: kStepWarpsLp consumer warps in two groups.
cudaError_t configure_step_kernels_lp() {
  const int smem = (int)SharedLayout::bytes;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(k_bicg_steps<kFP32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_bicg_steps<kBF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
  return cudaSuccess;
}

cudaError_t launch_bicg_steps_lp(const BicgArgs &a, int num_ctas, cudaStream_t s, int precision) {
  return precision == kBF16 ? launch_coop(k_bicg_steps<kBF16>, a, num_ctas, s)
                            : launch_coop(k_bicg_steps<kFP32>, a, num_ctas, s);
}
#endif  // HBX_STEP_TU

}  // namespace hbx
