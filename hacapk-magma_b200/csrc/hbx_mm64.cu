// hbx_mm64.cu -- the FP64 product with kNrhs right-hand sides of an FP64
// single-vector engine: Y = alpha * H X + beta * Yin, X, Y and Yin nd x kNrhs
// doubles, row-major.  The refinement residuals of the multi-RHS solver.
//
// 64 single-vector products read the factors 64 times (47 us each at 264 MB:
// 3.0 ms); this reads them once (0.30 ms), and the arithmetic, 64 fused
// multiply-adds a word, becomes the bound: 18.4e12 a second measured (0.11 ms
// there), the same on the FP64 tensor cores (mma.sync m8n8k4; tcgen05 has no FP64 kind) and on the FP64
// pipes.  The tensor instruction is taken because a warp's operands for 256 of
// them are two shared loads.
//
// Work is dealt out by unit: a P slab, or a row atom (its D block and, where
// the atom is split, its U block, in this order, so each row of Y is written by
// one CTA).  The units lie in descending cost and CTAs take them from a
// counter.  P units first, in a launch of their own; the second launch reads
// the zbu rows they wrote.
//
// Per unit a CTA streams 32 columns at a time: the columns' rows of X (or zbu)
// and the columns' panels come into a ring of shared stages with 16-byte
// asynchronous copies, and each of the 8 warps multiplies all rows of the
// block (8 at a time) with its 8 right-hand sides.  The pitches of both stages
// keep the fragments of a half warp on different banks.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <vector>

#include "hbx_device.cuh"
#include "hbx_engine.h"

namespace hbx {
namespace {

constexpr int kMmThreads = 256;
constexpr int kMmCols = 32;                           // columns of a stage
constexpr int kMmStages = 3;
constexpr uint32_t kXPitch = kNrhs * 8 + 32;          // a column's row of X: 512 bytes, 32 on
constexpr uint32_t kAPitch = (kSlabMax + 4) * 16;     // a panel: up to 64 rows of 16 bytes, 64 bytes on
constexpr uint32_t kABytes = kMmCols / 2 * kAPitch;
constexpr uint32_t kMmStageBytes = kABytes + kMmCols * kXPitch;
constexpr uint32_t kMaxCols = kStageBytes / 8;        // columns of a run
constexpr uint32_t kMmSmem = kMmStages * kMmStageBytes + kMaxCols * 4 + kRecBytes + 16;
constexpr uint32_t kNoRow = 0xffffffffu;              // a zero column
static_assert(kAPitch % 128 == 64 && kXPitch % 128 == 32, "fragments of a half warp on different banks");

__device__ __forceinline__ void cp_async16z(void *dst, const void *src, bool take) {  // 16 bytes, or zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(take ? 16 : 0)
               : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// kTiles: row tiles of 8 that a block may have (P slabs 8, row atoms 4).
template <int kTiles>
__global__ void __launch_bounds__(kMmThreads, 2) k_mm64(Mm64Args a) {
  extern __shared__ __align__(128) uint8_t sm[];
  uint32_t *rows = reinterpret_cast<uint32_t *>(sm + kMmStages * kMmStageBytes);
  uint8_t *rec = sm + kMmStages * kMmStageBytes + kMaxCols * 4;
  uint32_t *next = reinterpret_cast<uint32_t *>(rec + kRecBytes);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  for (;;) {
    if (threadIdx.x == 0) *next = atomicAdd(a.next, 1u);
    __syncthreads();
    const uint32_t ui = *next;
    if (ui >= a.nunits) return;
    const Mm64Unit U = a.units[ui];
    const CtaInfo ci = a.ctas[U.cta];
    const uint8_t *stream = a.stream + ci.stream_off;
    double c[kTiles][2];
    for (uint32_t k = 0; k < (uint32_t)U.n0 + U.n1; ++k) {
      const uint32_t run = ci.rec_begin + (k < U.n0 ? U.r0 + k : U.r1 + (k - U.n0));
      __syncthreads();  // the previous run's rows and record are read, *next too
      if (threadIdx.x < kRecBytes / 16)
        cp_async16cg(rec + threadIdx.x * 16, reinterpret_cast<const uint8_t *>(a.recs + run) + threadIdx.x * 16);
      cp_async_wait_all();
      __syncthreads();
      const Run hd = *reinterpret_cast<const Run *>(rec);
      const Seg *seg = reinterpret_cast<const Seg *>(rec + sizeof(Run));
      const uint32_t kind = hd.flags & 0xffu, h = hd.nrow, np = hd.npanel, nch = (2u * np + kMmCols - 1) / kMmCols;
      // the vector row of every column; kSegZbu marks a row of zbu
      for (uint32_t i = hd.vlen + threadIdx.x; i < nch * kMmCols; i += kMmThreads) rows[i] = kNoRow;
      for (uint32_t s = w; s < hd.nseg; s += kMmThreads / 32) {
        const Seg sg = seg[s];
        const uint32_t src = kind == kRunU ? (sg.src | kSegZbu) : sg.src;
        for (uint32_t e = lane; e < sg.len; e += 32) rows[sg.dst + e] = src + e;
      }
      if (hd.flags & kFirst) {
#pragma unroll
        for (int t = 0; t < kTiles; ++t) c[t][0] = c[t][1] = 0.0;
      }
      __syncthreads();
      const uint8_t *pan = stream + hd.pos;
      auto load = [&](uint32_t ch) {
        uint8_t *st = sm + (ch % kMmStages) * kMmStageBytes;
        const uint32_t p0 = ch * (kMmCols / 2), n = min((uint32_t)kMmCols / 2, np - p0);
        for (uint32_t e = threadIdx.x; e < (kMmCols / 2) * h; e += kMmThreads) {
          const uint32_t p = e / h, i = e - p * h;
          const bool take = p < n;  // past the run's panels: zeros
          cp_async16z(st + p * kAPitch + i * 16, pan + (size_t)(take ? (p0 + p) * h + i : 0u) * 16, take);
        }
#pragma unroll
        for (uint32_t k2 = 0; k2 < kMmCols * kNrhs / 2 / kMmThreads; ++k2) {
          const uint32_t col = k2 * (kMmThreads / 32) + w;
          const uint32_t src = rows[ch * kMmCols + col];
          const bool take = src != kNoRow;
          const double *v = (take && (src & kSegZbu)) ? a.zbu + (size_t)(src & ~kSegZbu) * kNrhs
                                                      : a.x + (take ? (size_t)src * kNrhs : 0);
          cp_async16z(st + kABytes + col * kXPitch + lane * 16, v + lane * 2, take);
        }
        cp_async_commit();
      };
      for (uint32_t ch = 0; ch < (uint32_t)kMmStages - 1; ++ch) {
        if (ch < nch) load(ch);
        else cp_async_commit();
      }
      for (uint32_t ch = 0; ch < nch; ++ch) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kMmStages - 2) : "memory");
        __syncthreads();  // chunk ch has landed; chunk ch - 1 is read
        if (ch + kMmStages - 1 < nch) load(ch + kMmStages - 1);
        else cp_async_commit();
        const uint32_t st = smem_u32(sm + (ch % kMmStages) * kMmStageBytes);
        const uint32_t as = st + (uint32_t)(q >> 1) * kAPitch + (uint32_t)g * 16 + (uint32_t)(q & 1) * 8;
        const uint32_t xs = st + kABytes + (uint32_t)q * kXPitch + (uint32_t)(w * 8 + g) * 8;
#pragma unroll
        for (uint32_t k4 = 0; k4 < kMmCols / 4; ++k4) {
          const double b = lds_f64(xs + k4 * 4 * kXPitch);
#pragma unroll
          for (int t = 0; t < kTiles; ++t)
            if (8u * t < h) dmma(c[t], lds_f64(as + k4 * 2 * kAPitch + t * 128), b);
        }
      }
      if (!(hd.flags & kLast)) continue;
      // rows of the block: tile t row g, right-hand sides 8 w + 2 q and the next
#pragma unroll
      for (int t = 0; t < kTiles; ++t) {
        const uint32_t i = 8u * t + g;
        if (i >= h) continue;
        const size_t o = (size_t)(hd.out + i) * kNrhs + w * 8 + 2 * q;
        double v0 = c[t][0], v1 = c[t][1];
        if (kind == kRunP) {
          a.zbu[o] = v0;
          a.zbu[o + 1] = v1;
          continue;
        }
        if (kind == kRunU) {  // after the atom's D block, by this same thread
          v0 = fma(a.alpha, v0, a.y[o]);
          v1 = fma(a.alpha, v1, a.y[o + 1]);
        } else {
          v0 *= a.alpha;
          v1 *= a.alpha;
          if (a.beta != 0.0) {
            v0 = fma(a.beta, a.yin[o], v0);
            v1 = fma(a.beta, a.yin[o + 1], v1);
          }
        }
        a.y[o] = v0;
        a.y[o + 1] = v1;
      }
    }
  }
}

}  // namespace

cudaError_t configure_mm64() {
  cudaError_t e = cudaFuncSetAttribute(k_mm64<kSlabMax / 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_mm64<kAtomMax / 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmSmem);
  return e;
}

void mm64_units(const std::vector<CtaInfo> &ctas, const std::vector<RunLite> &lite, std::vector<Mm64Unit> &p,
                std::vector<Mm64Unit> &rest) {
  struct Costed {
    uint64_t cost;
    Mm64Unit u;
  };
  std::vector<Costed> cp, cr;
  for (size_t c = 0; c < ctas.size(); ++c) {
    const CtaInfo &ci = ctas[c];
    const uint32_t nr = ci.nr_p + ci.nr_d + ci.nr_u;
    std::map<uint32_t, size_t> of_row;  // this CTA's D units by first row
    for (uint32_t r = 0; r < nr;) {
      uint32_t n = 0;
      uint64_t cost = 0;
      const RunLite &F = lite[ci.rec_begin + r];
      for (bool last = false; !last && r + n < nr; ++n) {
        const RunLite &L = lite[ci.rec_begin + r + n];
        cost += 64 + (uint64_t)((L.nrow + 7) / 8) * L.npanel;
        last = (L.flags & kLast) != 0;
      }
      const uint32_t kind = F.flags & 0xffu;
      if (kind == kRunP) {
        cp.push_back({cost, Mm64Unit{(uint32_t)c, r, n, 0, 0}});
      } else if (kind == kRunU) {
        Costed &d = cr[of_row.at(F.out)];
        d.cost += cost;
        d.u.r1 = r;
        d.u.n1 = n;
      } else {
        if (kind == kRunD) of_row[F.out] = cr.size();
        cr.push_back({cost, Mm64Unit{(uint32_t)c, r, n, 0, 0}});
      }
      r += n;
    }
  }
  auto sorted = [](std::vector<Costed> &v, std::vector<Mm64Unit> &out) {
    std::stable_sort(v.begin(), v.end(), [](const Costed &x, const Costed &y) { return x.cost > y.cost; });
    out.clear();
    for (const Costed &x : v) out.push_back(x.u);
  };
  sorted(cp, p);
  sorted(cr, rest);
}

cudaError_t launch_mm64(const Mm64Args &base, const Mm64Unit *p, uint32_t np, const Mm64Unit *rest, uint32_t nrest,
                        cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(base.next, 0, 2 * sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  constexpr uint32_t kGrid = 148 * 2;  // two CTAs per SM (105 KB of stages each)
  Mm64Args a = base;
  if (np > 0) {
    a.units = p;
    a.nunits = np;
    k_mm64<kSlabMax / 8><<<std::min(np, kGrid), kMmThreads, kMmSmem, s>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (nrest > 0) {
    a.units = rest;
    a.nunits = nrest;
    a.next = base.next + 1;
    k_mm64<kAtomMax / 8><<<std::min(nrest, kGrid), kMmThreads, kMmSmem, s>>>(a);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace hbx
