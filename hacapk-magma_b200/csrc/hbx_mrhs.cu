// hbx_mrhs.cu -- H-matrix product with many right-hand sides on the sm_100a
// tensor cores: Y = alpha * H X + beta * Yin for kNrhs = 64 right-hand sides.
//
// The packed stream is the FP32 engine's (panels of 4 columns x h rows, 16
// bytes a row) with every run an even number of panels, so two panels make
// the K = 8 of one TF32 step.  Per CTA (one per SM), 23 warps:
//
//   warps 0-3   epilogue: TMEM accumulator -> zbu (P blocks) or Y (D, U)
//   warp 4      tcgen05: allocates TMEM; one thread issues the MMAs
//   warp 5      bulk-copy producer of the stream ring (16 KB chunks)
//   warps 6-21  gather: X (or zbu) columns of a run, 128 at a time, into a
//               K-major operand stage [4-column chunk][rhs][4] (32 KB), four
//               warps per stage
//   warp 22     grid barrier between the P blocks and the U runs
//
// The MMA thread is the one that elect.sync names: the compiler then knows that
// one thread is active.  Under threadIdx.x % 32 == 0 it does not, and guards
// every MMA with a loop over the active lanes: 107 cycles an MMA of M = 64,
// N = 24, K = 8 with this kernel's descriptors, against 35 here, four at a time
// (the tensor core takes 23).  Two threads of the first kind on alternate
// blocks, which this replaces, kept the product on 81,920 unknowns at 513 us.
//
// One MMA: D[rhs][row] += Xs[rhs][k..k+8] * Panel[row][k..k+8]^T with
// M = 64 right-hand sides, N = the block's rows rounded up to 8, A (the
// staged X) and B (two panels straight from the ring) both K-major in the
// canonical no-swizzle layout: 8-row core matrices of 16-byte rows, the next
// 8 rows 128 bytes on (SBO), the next 4 columns LBO on (1 KB for A, 16h for
// B).  D lives in TMEM (M = 64: rhs m in lane (m mod 16) + 32 (m / 16)); four
// 64-column accumulators let the epilogue of a block overlap the MMAs of
// the next ones.  The ring is smaller than k_matvec's (the product is bound by
// the X stages, not by the stream) and MMAs read it in place: a panel pair
// that runs past the
// ring's end reads a mirror of the first bytes of slot 0 that the producer
// keeps behind the ring.  Rows of D past h come from bytes after the pair
// and are never stored.
//
// No counterpart in the reference (its batched GEMV takes one vector).
#include "hbx_device.cuh"
#include "hbx_engine.h"

namespace hbx {
namespace {

constexpr int kSliceCols = 128;                        // stage columns per slice
constexpr int kSliceChunks = kSliceCols / 4;           // 4-column K chunks per slice
constexpr int kChunkXBytes = kNrhs * 16;               // one chunk, all right-hand sides: 1 KB
constexpr int kSliceBytes = kSliceChunks * kChunkXBytes;  // 32 KB
constexpr int kMChunkLog = 14;  // ring chunk: 16 KB
constexpr int kMChunkBytes = 1 << kMChunkLog;
constexpr int kMRingChunks = 5;
constexpr uint32_t kMRingBytes = (uint32_t)kMRingChunks * kMChunkBytes;
constexpr int kXStages = 4;
constexpr int kMirrorBytes = 2304;  // >= 2 panels of 64 rows + 7 rows past them
constexpr int kAccCols = 64;        // TMEM columns per accumulator (rows of a block <= 64)
constexpr int kAccs = 4;            // accumulators: blocks in flight between the MMAs and the epilogue
constexpr int kTmemCols = kAccs * kAccCols;
constexpr int kEpiWarps = 4, kMmaWarp = 4, kProdWarpM = 5, kGathWarp0 = 6, kGathWarps = 16,
              kSyncWarpM = kGathWarp0 + kGathWarps;
constexpr int kSliceWarps = kGathWarps / kXStages;      // gather warps per stage, side by side
constexpr int kWarpCols = kSliceCols / kSliceWarps;     // stage columns of one gather warp
static_assert(kWarpCols == 32, "one column source a lane");
constexpr int kThreadsM = (kSyncWarpM + 1) * 32;

struct MLayout {
  static constexpr uint32_t ring = 0;
  static constexpr uint32_t xst = (kMRingBytes + kMirrorBytes + 1023) / 1024 * 1024;  // [kXStages] slices
  static constexpr uint32_t lite = xst + kXStages * kSliceBytes;                      // [kMaxPairRuns] summaries
  static constexpr uint32_t full = lite + kMaxPairRuns * 16;
  static constexpr uint32_t empty = full + 8 * kMRingChunks;
  static constexpr uint32_t xfull = empty + 8 * kMRingChunks;
  static constexpr uint32_t xempty = xfull + 8 * kXStages;
  static constexpr uint32_t accfull = xempty + 8 * kXStages;
  static constexpr uint32_t accempty = accfull + 8 * kAccs;
  static constexpr uint32_t pdone = accempty + 8 * kAccs;
  static constexpr uint32_t gdone = pdone + 8;
  static constexpr uint32_t mdone = gdone + 8;
  static constexpr uint32_t tmem = mdone + 8;  // TMEM base address (tcgen05.alloc writes it)
  static constexpr uint32_t gen0 = tmem + 4;   // first grid-barrier generation of the launch
  static constexpr uint32_t bytes = gen0 + 4;
};
static_assert(MLayout::bytes <= 227 * 1024, "shared memory per CTA");
static_assert(MLayout::xst % 1024 == 0 && MLayout::lite % 16 == 0 && MLayout::full % 8 == 0, "layout alignment");

// ---- tcgen05 ----------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, no swizzle, K-major canonical layout.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3fffu);
  d |= (uint64_t)((lbo >> 4) & 0x3fffu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3fffu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of sm_100
  return d;                // base offset 0, absolute LBO, layout SWIZZLE_NONE
}

// Instruction descriptor: kind::tf32, D f32, A and B K-major, M x N.
__device__ __forceinline__ uint32_t idesc_tf32(uint32_t m, uint32_t n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// The barrier receives one arrival once every MMA this thread issued so far
// has completed.
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// ---- producer with the ring-end mirror ------------------------------------
// The factors pass through L2 with evict_first, and Y past it: X and zbu are
// what is read again (86 MB on 81,920 unknowns; without the hints the gather
// went to HBM, 473 us instead of 343).
__device__ __forceinline__ void mr_issue(const uint8_t *src, uint32_t bytes, uint32_t g, uint8_t *ring,
                                         uint64_t *full, uint64_t policy) {
  const uint32_t s = g % kMRingChunks;
  const uint32_t off = g << kMChunkLog;
  const uint32_t nb = min((uint32_t)kMChunkBytes, bytes - off);
  const uint32_t nm = s == 0 ? min(nb, (uint32_t)kMirrorBytes) : 0u;
  mbar_arrive_expect_tx(&full[s], nb + nm);
  bulk_g2s_hint(ring + ((size_t)s << kMChunkLog), src + off, nb, &full[s], policy);
  if (nm) bulk_g2s_hint(ring + kMRingBytes, src + off, nm, &full[s], policy);
}

__device__ __forceinline__ void mr_producer(const uint8_t *src, uint32_t bytes, uint8_t *ring, uint64_t *full,
                                            uint64_t *empty, int *err, uint64_t tmo) {
  const uint32_t K = (bytes + kMChunkBytes - 1) >> kMChunkLog;
  const uint64_t policy = l2_policy_stream();
  uint32_t issued = 0;
  for (uint32_t g = 0; g < K; ++g) {
    if (g >= (uint32_t)kMRingChunks && !mbar_wait(&empty[g % kMRingChunks], ((g / kMRingChunks) - 1) & 1, tmo)) {
      atomicOr(err, kErrProducer);
      break;
    }
    mr_issue(src, bytes, g, ring, full, policy);
    issued = g + 1;
  }
  // copies still in flight land before the CTA exits
  const uint32_t g0 = issued > (uint32_t)kMRingChunks ? issued - kMRingChunks : 0;
  for (uint32_t g = g0; g < issued; ++g) mbar_wait(&full[g % kMRingChunks], (g / kMRingChunks) & 1, tmo);
}

struct MSmem {
  uint8_t *ring, *xst;
  RunLite *lite;
  uint64_t *full, *empty, *xfull, *xempty, *accfull, *accempty, *pdone, *gdone, *mdone;
  uint32_t *tmem, *gen0;
};

__device__ __forceinline__ MSmem mlayout(uint8_t *b) {
  MSmem s;
  s.ring = b + MLayout::ring;
  s.xst = b + MLayout::xst;
  s.lite = reinterpret_cast<RunLite *>(b + MLayout::lite);
  s.full = reinterpret_cast<uint64_t *>(b + MLayout::full);
  s.empty = reinterpret_cast<uint64_t *>(b + MLayout::empty);
  s.xfull = reinterpret_cast<uint64_t *>(b + MLayout::xfull);
  s.xempty = reinterpret_cast<uint64_t *>(b + MLayout::xempty);
  s.accfull = reinterpret_cast<uint64_t *>(b + MLayout::accfull);
  s.accempty = reinterpret_cast<uint64_t *>(b + MLayout::accempty);
  s.pdone = reinterpret_cast<uint64_t *>(b + MLayout::pdone);
  s.gdone = reinterpret_cast<uint64_t *>(b + MLayout::gdone);
  s.mdone = reinterpret_cast<uint64_t *>(b + MLayout::mdone);
  s.tmem = reinterpret_cast<uint32_t *>(b + MLayout::tmem);
  s.gen0 = reinterpret_cast<uint32_t *>(b + MLayout::gen0);
  return s;
}

// A block without columns (a D block of an atom that no dense leaf touches)
// is one run of no panels: nothing is multiplied for it.
__device__ __forceinline__ bool empty_block(const RunLite &L) {
  return L.npanel == 0 && (L.flags & kFirst) && (L.flags & kLast);
}

__device__ __forceinline__ uint32_t run_slices(const RunLite &L) {
  return (4u * L.npanel + kSliceCols - 1) / kSliceCols;
}

// ---- gather warp gi: its columns of slices q = gs, gs + kXStages, ... ----
// A slice is a transpose: its columns are rows of X (or zbu), 64 consecutive
// floats each, and the stage holds 16-byte groups of 4 columns per right-hand
// side.  A lane loads its two right-hand sides (lane, lane + 32) of 4 columns
// and stores two groups, so loads and stores are whole lines and no lane
// exchanges anything; the loads of half its columns are in flight while it
// waits for the stage.  What bounds the kernel is this gather (263 of its 287
// us on 81,920 unknowns): 1.3 GB through L2 with 64 KB in flight per SM.
// Measured there: 4-byte asynchronous copies into the stage, one per element,
// 583 us in all (with the old issue loop); 16-byte loads transposed 4 x 4 in
// registers on 8 warps 411; this with the stage waited for before the loads
// 318; 3 stages, 64-, 96-, 160- or 192-column slices 302-375.  Which row a
// column is comes from `cols`, one word a column, fetched a slice ahead.
constexpr int kGathUnroll = 4;  // chunks of 4 columns whose loads are in flight together
static_assert(kWarpCols % (4 * kGathUnroll) == 0, "whole batches of chunks");

__device__ __forceinline__ void mr_gather(const MatmatArgs &a, const CtaInfo &ci, uint32_t nr, const MSmem &sm,
                                          uint32_t gi) {
  const int lane = threadIdx.x & 31;
  const uint32_t gs = gi / kSliceWarps, col0 = (gi % kSliceWarps) * kWarpCols;  // this warp's stage and columns of it
  // a place in the CTA's slices: slice s of run r, whose first slice is q and
  // first panel column c
  struct Place {
    uint32_t r, q, s;
    uint64_t c;
  };
  // on to the next slice of this warp's stage, from (r, s)
  auto settle = [&](Place &p) {
    for (; p.r < nr; ++p.r, p.s = 0) {
      const uint32_t np = sm.lite[p.r].npanel, nsl = (4u * np + kSliceCols - 1) / kSliceCols;
      p.s += (gs + kXStages - (p.q + p.s) % kXStages) % kXStages;
      if (p.s < nsl) return;
      p.q += nsl;
      p.c += 4u * np;
    }
  };
  // the vector row of its slice's column `lane` of this warp's
  auto fetch = [&](const Place &p) {
    const uint32_t ncol = p.r < nr ? 4u * sm.lite[p.r].npanel : 0u, sc = p.s * kSliceCols + col0 + lane;
    return sc < ncol ? __ldg(a.cols + p.c + sc) : kNoCol;
  };
  float4 *const st = reinterpret_cast<float4 *>(sm.xst + gs * kSliceBytes + (col0 / 4) * kChunkXBytes);
  bool ok = true, zbu_ready = false;
  Place at{0, 0, 0, ci.col_begin};
  settle(at);
  uint32_t next_row = fetch(at);
  while (at.r < nr) {
    const RunLite L = sm.lite[at.r];
    const uint32_t qs = at.q + at.s, cols = min((uint32_t)kSliceCols, 4u * L.npanel - at.s * kSliceCols);
    const bool zbu = (L.flags & 0xffu) == kRunU;
    if (zbu && !zbu_ready) {
      ok = warp_wait(sm.gdone, 0, a.timeout_ns);  // every CTA's zbu rows are written
      __threadfence();
      zbu_ready = true;
      if (!ok) break;
    }
    const float *vec = (zbu ? a.zbu : a.x) + lane;
    const uint32_t row = next_row;
    ++at.s;
    settle(at);
    next_row = fetch(at);
    const uint32_t nchunk = (min(max(cols, col0), col0 + kWarpCols) - col0) / 4;  // of this warp
    // the MMAs have left the stage's previous slice (a warp without columns in
    // this slice waits too: its arrival below belongs to this slice's phase)
    auto stage_free = [&]() {
      return qs < (uint32_t)kXStages || warp_wait(&sm.xempty[gs], ((qs / kXStages) - 1) & 1, a.timeout_ns);
    };
    if (nchunk == 0) ok = stage_free();
    for (uint32_t k0 = 0; k0 < nchunk; k0 += kGathUnroll) {
      float v[kGathUnroll][4][2];
#pragma unroll
      for (uint32_t u = 0; u < kGathUnroll; ++u)
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) {
          const uint32_t src = __shfl_sync(0xffffffffu, row, 4 * (k0 + u) + c);  // kNoCol past the slice's columns
          v[u][c][0] = v[u][c][1] = 0.0f;
          if (src != kNoCol) {  // through L2: zbu is written by this launch
            const float *p = vec + (size_t)src * kNrhs;
            v[u][c][0] = __ldcg(p);
            v[u][c][1] = __ldcg(p + 32);
          }
        }
      if (k0 == 0 && !(ok = stage_free())) break;  // the loads need no stage, the stores do
#pragma unroll
      for (uint32_t u = 0; u < kGathUnroll; ++u) {
        if (k0 + u >= nchunk) break;
        float4 *dst = st + (k0 + u) * kNrhs + lane;
        dst[0] = make_float4(v[u][0][0], v[u][1][0], v[u][2][0], v[u][3][0]);
        dst[32] = make_float4(v[u][0][1], v[u][1][1], v[u][2][1], v[u][3][1]);
      }
    }
    if (!ok) break;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // visible to the tensor cores
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.xfull[gs]);
  }
  if (!ok && lane == 0) atomicOr(a.err, kErrPipeline);
}

__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

constexpr uint32_t kMmaUnroll = 4;  // 1: 356 us, 2: 321, 4: 318, 8: 318 (81,920 unknowns)
// ---- MMA thread (the elected one of warp kMmaWarp) ------------------------------
// Per slice: wait for its X stage and for every ring chunk its panel pairs
// touch (at most 32 KB of pairs, three chunks), then issue its MMAs back to
// back with the descriptors advanced in place, and commit the stage back.
__device__ __forceinline__ void mr_mma(const MatmatArgs &a, uint32_t nr, uint32_t K, const MSmem &sm) {
  const RunLite *lite = sm.lite;
  const uint64_t tmo = a.timeout_ns;
  const uint32_t tbase = *sm.tmem;
  const uint32_t ring_s = smem_u32(sm.ring), xst_s = smem_u32(sm.xst);
  uint32_t waited = 0, released = 0, q = 0, nb = 0;  // nb: blocks so far
  bool ok = true;
  // Releases ring chunks below c once the MMAs issued so far are done with
  // them; a chunk is waited for (full) before its release, so the empty
  // phases stay in order.
  auto release_below = [&](uint32_t c) {
    while (ok && released < c) {
      if (waited <= released) {
        ok = mbar_wait(&sm.full[released % kMRingChunks], (released / kMRingChunks) & 1, tmo);
        if (!ok) return;
        waited = released + 1;
      }
      tc_commit(&sm.empty[released % kMRingChunks]);
      ++released;
    }
  };
  for (uint32_t r = 0; r < nr && ok; ++r) {
    const RunLite L = lite[r];
    if (empty_block(L)) continue;
    const uint32_t h = L.nrow, n8 = (h + 7u) & ~7u, pb = 16u * h;
    const uint32_t idesc = idesc_tf32(kNrhs, n8);
    const uint32_t buf = nb % kAccs;
    const uint32_t dtm = tbase + buf * kAccCols;
    uint32_t acc = (L.flags & kFirst) ? 0u : 1u;
    if (!acc) {
      // the epilogue has read this accumulator's previous block
      if (nb >= (uint32_t)kAccs && !(ok = mbar_wait(&sm.accempty[buf], ((nb / kAccs) - 1) & 1, tmo))) break;
      tc_fence_after();  // the epilogue's TMEM reads come before these MMAs' writes
    }
    const uint32_t nsl = run_slices(L), npair = L.npanel / 2u;
    const uint64_t bhi = smem_desc(0, pb, 128);  // the descriptor without its address
    for (uint32_t s = 0; s < nsl; ++s, ++q) {
      const uint32_t slot = q % kXStages;
      const uint32_t p0 = s * (kSliceCols / 8), p1 = min(npair, p0 + kSliceCols / 8);
      const uint32_t pos0 = L.pos + 2u * p0 * pb, pos1 = L.pos + 2u * p1 * pb;
      release_below(pos0 >> kMChunkLog);
      const uint32_t clast = (pos1 - 1u) >> kMChunkLog;
      while (ok && waited <= clast) {
        ok = mbar_wait(&sm.full[waited % kMRingChunks], (waited / kMRingChunks) & 1, tmo);
        waited += ok ? 1u : 0u;
      }
      if (ok) ok = mbar_wait(&sm.xfull[slot], (q / kXStages) & 1, tmo);
      if (!ok) break;
      uint64_t adesc = smem_desc(xst_s + slot * kSliceBytes, kChunkXBytes, 128);
      uint32_t baddr = ring_s + ((pos0 >> kMChunkLog) % kMRingChunks) * kMChunkBytes + (pos0 & (kMChunkBytes - 1));
      const uint32_t step = 2u * pb;
      uint32_t p = p0;
      for (; p + kMmaUnroll <= p1; p += kMmaUnroll) {
        uint32_t ad[kMmaUnroll], bd[kMmaUnroll];
#pragma unroll
        for (uint32_t u = 0; u < kMmaUnroll; ++u) {
          ad[u] = (uint32_t)adesc + u * ((2u * kChunkXBytes) >> 4);
          uint32_t ba = baddr + u * step;
          if (ba >= ring_s + kMRingBytes) ba -= kMRingBytes;  // a pair that starts past the ring's end
          bd[u] = (uint32_t)bhi | (ba >> 4);
        }
#pragma unroll
        for (uint32_t u = 0; u < kMmaUnroll; ++u) {
          mma_tf32(dtm, (adesc & 0xffffffff00000000ull) | ad[u], (bhi & 0xffffffff00000000ull) | bd[u], idesc, acc);
          acc = 1;
        }
        adesc += kMmaUnroll * ((2u * kChunkXBytes) >> 4);
        baddr += kMmaUnroll * step;
        if (baddr >= ring_s + kMRingBytes) baddr -= kMRingBytes;
      }
      for (; p < p1; ++p) {
        mma_tf32(dtm, adesc, bhi | (uint64_t)(baddr >> 4), idesc, acc);
        acc = 1;
        adesc += (2u * kChunkXBytes) >> 4;  // the next two K chunks of the stage
        baddr += step;
        if (baddr >= ring_s + kMRingBytes) baddr -= kMRingBytes;
      }
      tc_commit(&sm.xempty[slot]);  // the stage slot is free once these MMAs are done
    }
    if (ok && (L.flags & kLast)) {
      tc_commit(&sm.accfull[buf]);
      ++nb;
    }
  }
  if (ok) release_below(K);
  if (!ok) atomicOr(a.err, kErrPipeline);
  // every MMA has completed before TMEM is handed back
  tc_commit(sm.mdone);
  mbar_wait(sm.mdone, 0, tmo);
}

// ---- epilogue warps -----------------------------------------------------------
// Warp w reads TMEM lanes 32w..32w+31 (rhs 16w + lane for lane < 16): all of
// a block's columns (its rows) first, then, for D and U blocks, all the Y
// values it updates, so each block costs one round trip of each kind.
__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ void mr_epilogue(const MatmatArgs &a, uint32_t nr, uint32_t nblk_p, const MSmem &sm) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t m = 16u * w + lane;  // right-hand side of this thread's TMEM lane (lane < 16)
  const uint32_t tlane = (32u * (uint32_t)w) << 16;  // this warp's TMEM lane quarter
  uint32_t nb = 0, np_done = 0;
  if (nblk_p == 0 && lane == 0) mbar_arrive(sm.pdone);
  bool ok = true;
  for (uint32_t r = 0; r < nr && ok; ++r) {
    const RunLite L = sm.lite[r];
    if (!(L.flags & kLast)) continue;
    const uint32_t h = L.nrow, kind = L.flags & 0xffu;
    if (empty_block(L)) {
      // no columns: D rows are beta * yin, P rows zero, U rows unchanged
      if (lane < 16)
        for (uint32_t i = 0; i < h; ++i) {
          const size_t o = (size_t)(L.out + i) * kNrhs + m;
          if (kind == kRunD) a.y[o] = a.beta != 0.0 ? a.beta * a.yin[o] : 0.0;
          else if (kind == kRunP) a.zbu[o] = 0.0f;
        }
      __syncwarp();
      if (kind == kRunP && ++np_done == nblk_p && lane == 0) mbar_arrive(sm.pdone);
      continue;
    }
    const uint32_t buf = nb % kAccs;
    ok = warp_wait(&sm.accfull[buf], (nb / kAccs) & 1, a.timeout_ns);
    if (!ok) break;
    tc_fence_after();
    const uint32_t taddr = *sm.tmem + tlane + buf * kAccCols;
    // 16 rows at a time: their columns from TMEM, then (D with beta, U) the
    // Y values they update, then the stores
    const bool add = kind == kRunU || (kind == kRunD && a.beta != 0.0);
    const double *src = kind == kRunU ? a.y : a.yin;
    const double c = kind == kRunU ? 1.0 : a.beta;
    for (uint32_t r0 = 0; r0 < h; r0 += 16) {
      uint32_t v[16];
      tmem_ld8_async(taddr + r0, v);
      if (r0 + 8 < h) tmem_ld8_async(taddr + r0 + 8, v + 8);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (lane < 16) {
        const size_t o0 = (size_t)(L.out + r0) * kNrhs + m;
        const uint32_t n = min(16u, h - r0);
        if (kind == kRunP) {
#pragma unroll
          for (uint32_t i = 0; i < 16; ++i)
            if (i < n) a.zbu[o0 + (size_t)i * kNrhs] = __uint_as_float(v[i]);
        } else {
          double old[16];
#pragma unroll
          for (uint32_t i = 0; i < 16; ++i) old[i] = (add && i < n) ? __ldcs(src + o0 + (size_t)i * kNrhs) : 0.0;
#pragma unroll
          for (uint32_t i = 0; i < 16; ++i)
            if (i < n) __stcs(a.y + o0 + (size_t)i * kNrhs, fma(a.alpha, (double)__uint_as_float(v[i]), c * old[i]));
        }
      }
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.accempty[buf]);
    if (kind == kRunP && ++np_done == nblk_p && lane == 0) mbar_arrive(sm.pdone);  // this warp's zbu rows are out
    ++nb;
  }
  if (!ok && lane == 0) atomicOr(a.err, kErrPipeline);
}

__global__ void __launch_bounds__(kThreadsM, 1) k_matmat(MatmatArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (a.go && !*(volatile const int *)a.go) return;  // set by an earlier launch: the same on every CTA
  const MSmem sm = mlayout(smem_raw);
  const CtaInfo ci = a.ctas[blockIdx.x];
  const uint32_t nr = ci.nr_p + ci.nr_d + ci.nr_u;
  const uint32_t K = (ci.stream_bytes + kMChunkBytes - 1) >> kMChunkLog;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kMRingChunks; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], 1);
    }
    for (int i = 0; i < kXStages; ++i) {
      mbar_init(&sm.xfull[i], kSliceWarps);
      mbar_init(&sm.xempty[i], 1);
    }
    for (int i = 0; i < kAccs; ++i) {
      mbar_init(&sm.accfull[i], 1);
      mbar_init(&sm.accempty[i], kEpiWarps);
    }
    mbar_init(sm.pdone, kEpiWarps);
    mbar_init(sm.gdone, 1);
    mbar_init(sm.mdone, 1);
    *sm.gen0 = grid_gen0(a.gbar);
    mbar_fence_init();
  }
  {  // the CTA's run summaries
    const uint4 *src = reinterpret_cast<const uint4 *>(a.lite + ci.rec_begin);
    uint4 *dst = reinterpret_cast<uint4 *>(sm.lite);
    for (uint32_t k = threadIdx.x; k < nr; k += blockDim.x) dst[k] = __ldg(src + k);
  }
  if (w == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(sm.tmem)),
                 "r"((uint32_t)kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (w == kProdWarpM) {
    if (lane == 0 && K > 0) mr_producer(a.stream + ci.stream_off, ci.stream_bytes, sm.ring, sm.full, sm.empty, a.err, a.timeout_ns);
    return;
  }
  if (w >= kGathWarp0 && w < kGathWarp0 + kGathWarps) {
    mr_gather(a, ci, nr, sm, (uint32_t)(w - kGathWarp0));
    return;
  }
  if (w == kSyncWarpM) {
    if (lane == 0) {
      if (!mbar_wait(sm.pdone, 0, a.timeout_ns)) {
        atomicOr(a.err, kErrPipeline);
        return;
      }
      const unsigned target = grid_target(*sm.gen0, 0, gridDim.x);
      grid_arrive(a.gbar, target);
      if (!grid_wait(a.gbar, target, a.timeout_ns)) {
        atomicOr(a.err, kErrGridBarrier);
        return;
      }
      mbar_arrive(sm.gdone);
    }
    return;
  }
  if (w == kMmaWarp) {
    if (elect_one()) mr_mma(a, nr, K, sm);
    __syncwarp();
  } else {
    mr_epilogue(a, nr, ci.nblk_p, sm);
  }
  // TMEM goes back once the MMAs are complete and the epilogue has read it
  tc_fence_before();
  named_bar(2, (kEpiWarps + 1) * 32);
  tc_fence_after();
  if (w == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*sm.tmem), "r"((uint32_t)kTmemCols)
                 : "memory");
}

// cols[CTA's col_begin + column] = the vector row of the run's column (kNoCol past its real ones).
__global__ void k_matmat_cols(const RunRec *recs, const CtaInfo *ctas, uint32_t *cols) {
  const CtaInfo ci = ctas[blockIdx.x];
  const uint32_t nr = ci.nr_p + ci.nr_d + ci.nr_u;
  uint64_t c = ci.col_begin;
  for (uint32_t r = 0; r < nr; ++r) {
    const RunRec &rec = recs[ci.rec_begin + r];
    const uint32_t ncol = 4u * rec.hdr.npanel, vlen = rec.hdr.vlen;
    for (uint32_t k = threadIdx.x; k < ncol; k += blockDim.x) {
      uint32_t row = kNoCol;
      if (k < vlen) {
        uint32_t lo = 0, hi = rec.hdr.nseg;  // the last segment that starts at or before k (in stage order)
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) >> 1;
          if (rec.seg[mid].dst <= k) lo = mid;
          else hi = mid;
        }
        row = rec.seg[lo].src + (k - rec.seg[lo].dst);
      }
      cols[c + k] = row;
    }
    c += ncol;
  }
}

}  // namespace

cudaError_t launch_matmat_cols(const RunRec *recs, const CtaInfo *ctas, int num_ctas, uint32_t *cols, cudaStream_t s) {
  k_matmat_cols<<<num_ctas, 256, 0, s>>>(recs, ctas, cols);
  return cudaGetLastError();
}

size_t matmat_smem_bytes() { return MLayout::bytes; }

cudaError_t configure_matmat() {
  return cudaFuncSetAttribute(k_matmat, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MLayout::bytes);
}

cudaError_t launch_matmat(const MatmatArgs &a, int num_ctas, cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(num_ctas);
  cfg.blockDim = dim3(kThreadsM);
  cfg.dynamicSmemBytes = MLayout::bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_matmat, a);
}

}  // namespace hbx
