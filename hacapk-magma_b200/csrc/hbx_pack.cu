// hbx_pack.cu -- the packed factor stream, laid out on the device
// (the layout of hbx_plan.h; pack_plan in hbx_plan.cpp is the same on the host).
//
// The leaves' words go to the device once, as they lie on the host, and
// k_pack forms every run from them: what bounds it is the two passes over the
// factors in HBM (read 8 bytes a word, write the storage precision), well
// under a millisecond per GB, so the setup is bound by the copy of the leaves
// over PCIe.  Packing on the host cost a zeroed host image of the whole stream
// (its page faults alone 0.4 s for the 1.2 GB of an 81,920-triangle sphere),
// the strided pass of all cores over it, and the same copy.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "hbx_engine.h"
#include "hbx_stage.h"

namespace hbx {
namespace {

// One leaf: word offsets of V (a dense leaf: A) and U in the device image.
struct PackLeaf {
  long long v, u;
  int ndl, ndt, r0, dense;
};

struct PackArgs {
  const double *raw;
  const PackLeaf *leaves;
  const RunRec *recs;
  const CtaInfo *ctas;
  const Block *blocks;
  const Piece *pieces;
  const uint32_t *piece_col;   // block column of each piece's first column
  const uint32_t *group_begin, *group_leaves, *group_row;  // P groups; stacked row of each group leaf's first rank
  uint8_t *stream;
};

constexpr int kPackThreads = 256;
constexpr int kTileCols = 32;
constexpr int kRunsAtOnce = 16;  // CTAs per engine CTA: 148 x 16 blocks of 256 threads, two waves and more

// The last index q in [lo, hi) with key[q] <= x (key ascending, key[lo] <= x).
__device__ __forceinline__ uint32_t last_at(const uint32_t *key, uint32_t lo, uint32_t hi, uint32_t x) {
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (key[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// One run at a time, 32 columns of it at a time through a shared tile: words
// that lie next to each other in a leaf (a row of V^T or of a dense leaf, a
// column of U) are read by neighbouring lanes, and the tile is written out as
// the run's panels, 16 bytes a thread.
template <int kPrec>
__global__ void __launch_bounds__(kPackThreads) k_pack(PackArgs a) {
  __shared__ double tile[kSlabMax][kTileCols + 1];
  __shared__ long long base[kSlabMax];  // P: of each row;  D, U: of each column of the tile
  __shared__ int rstride[kTileCols];    // D columns: words from row to row; U columns: -1; past the block: 0
  constexpr uint32_t G = group_cols(kPrec);
  const CtaInfo ci = a.ctas[blockIdx.x];
  const uint32_t nr = ci.nr_p + ci.nr_d + ci.nr_u;
  const uint32_t tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  for (uint32_t r = blockIdx.y; r < nr; r += gridDim.y) {
    const Run hd = a.recs[ci.rec_begin + r].hdr;
    const Block b = a.blocks[hd.block];
    const uint32_t h = hd.nrow, ncol = G * hd.npanel;
    uint8_t *dst = a.stream + ci.stream_off + hd.pos;
    const bool p = b.kind == kRunP;
    if (p && tid < h) {
      const uint32_t row = b.r0 + tid, q = last_at(a.group_row, a.group_begin[b.a], a.group_begin[b.a + 1], row);
      const PackLeaf &L = a.leaves[a.group_leaves[q]];
      base[tid] = L.v + (long long)(row - a.group_row[q]) * L.ndt;
    }
    for (uint32_t c0 = 0; c0 < ncol; c0 += kTileCols) {
      if (!p && tid < kTileCols) {
        const uint32_t col = hd.col0 + c0 + tid;
        int rs = 0;
        if (col < b.W) {
          const uint32_t q = last_at(a.piece_col, b.piece_begin, b.piece_begin + b.npiece, col);
          const Piece P = a.pieces[q];
          const PackLeaf &L = a.leaves[P.leaf];
          const long long lc = P.c0 + (col - a.piece_col[q]), ro = (long long)hd.out - L.r0;
          rs = L.dense ? L.ndt : -1;
          base[tid] = L.dense ? L.v + lc + ro * L.ndt : L.u + ro + lc * L.ndl;
        }
        rstride[tid] = rs;
      }
      __syncthreads();
      const uint32_t col = hd.col0 + c0 + lane;
      if (p) {
        for (uint32_t i = w; i < h; i += kPackThreads / 32) tile[i][lane] = col < b.W ? a.raw[base[i] + col] : 0.0;
      } else {
        const int rs = rstride[lane];
        if (rs >= 0)
          for (uint32_t i = w; i < h; i += kPackThreads / 32)
            tile[i][lane] = rs > 0 ? a.raw[base[lane] + (long long)i * rs] : 0.0;
        for (uint32_t c = w; c < kTileCols; c += kPackThreads / 32)
          if (rstride[c] < 0 && lane < h) tile[lane][c] = a.raw[base[c] + lane];
      }
      __syncthreads();
      const uint32_t n = min((uint32_t)kTileCols, ncol - c0) / G * h;
      for (uint32_t e = tid; e < n; e += kPackThreads) {
        const uint32_t pn = e / h, i = e % h;
        const double *t = &tile[i][pn * G];
        uint4 v;
        if (kPrec == kFP64) {
          const unsigned long long x = __double_as_longlong(t[0]), y = __double_as_longlong(t[1]);
          v = make_uint4((uint32_t)x, (uint32_t)(x >> 32), (uint32_t)y, (uint32_t)(y >> 32));
        } else if (kPrec == kFP32) {
          v = make_uint4(__float_as_uint((float)t[0]), __float_as_uint((float)t[1]), __float_as_uint((float)t[2]),
                         __float_as_uint((float)t[3]));
        } else {
          auto two = [&](int k) { return (uint32_t)bf16_from_double(t[k]) | ((uint32_t)bf16_from_double(t[k + 1]) << 16); };
          v = make_uint4(two(0), two(2), two(4), two(6));
        }
        reinterpret_cast<uint4 *>(dst)[(size_t)(c0 / G + pn) * h + i] = v;
      }
      __syncthreads();
    }
  }
}

}  // namespace

cudaError_t pack_on_device(const stc_HACApK_leafmtxp *st, const Plan &plan, const RunRec *d_recs, const CtaInfo *d_ctas,
                           uint8_t *d_stream, cudaError_t (*alloc)(void *, size_t)) {
  // the leaves' words, in leaf order: V then U of a low-rank leaf, A of a dense one
  std::vector<PackLeaf> leaves(std::max(1, plan.nlf));
  std::vector<HostPiece> pieces;
  pieces.reserve(2 * (size_t)plan.nlf);
  uint64_t words = 0;
  auto add = [&](const double *src, size_t n) -> long long {
    const uint64_t at = words;
    pieces.push_back(HostPiece{const_cast<double *>(src), at, n});
    words += n;
    return (long long)at;
  };
  for (int ip = 0; ip < plan.nlf; ++ip) {
    const auto *s = reinterpret_cast<const stc_HACApK_leafmtx *>(reinterpret_cast<const char *>(st->st_lf) +
                                                                 (size_t)st->st_lf_stride * ip);
    PackLeaf L{0, 0, s->ndl, s->ndt, s->nstrtl - 1, s->ltmtx == 2 ? 1 : 0};
    if (s->ndl > 0 && s->ndt > 0) {
      if (s->ltmtx == 2) {
        L.v = add(s->a1, (size_t)s->ndl * s->ndt);
      } else if (s->kt > 0) {
        const auto *u = reinterpret_cast<const double *>(reinterpret_cast<const char *>(s->a1) + s->a1size);
        L.v = add(s->a1, (size_t)s->ndt * s->kt);
        L.u = add(u, (size_t)s->ndl * s->kt);
      }
    }
    leaves[ip] = L;
  }
  if (words == 0 || plan.recs.empty()) return cudaSuccess;
  std::vector<uint32_t> pcol(std::max<size_t>(1, plan.pieces.size()), 0), grow(std::max<size_t>(1, plan.group_leaves.size()), 0);
  for (const Block &b : plan.blocks) {
    uint32_t c = 0;
    for (uint32_t q = b.piece_begin; q < b.piece_begin + b.npiece; ++q) {
      pcol[q] = c;
      c += plan.pieces[q].n;
    }
  }
  for (size_t g = 0; g + 1 < plan.group_leaf_begin.size(); ++g) {
    const uint32_t q0 = plan.group_leaf_begin[g], q1 = plan.group_leaf_begin[g + 1];
    for (uint32_t q = q0; q < q1; ++q) grow[q] = (uint32_t)(plan.zoff[plan.group_leaves[q]] - plan.zoff[plan.group_leaves[q0]]);
  }
  // one temporary allocation: the leaf words, then the tables
  size_t bytes = words * sizeof(double);
  auto place = [&](size_t n) {
    const size_t at = (bytes + 255) & ~(size_t)255;
    bytes = at + n;
    return at;
  };
  const size_t o_leaf = place(leaves.size() * sizeof(PackLeaf)), o_blk = place(plan.blocks.size() * sizeof(Block)),
               o_pc = place(plan.pieces.size() * sizeof(Piece)), o_col = place(pcol.size() * 4),
               o_gb = place(plan.group_leaf_begin.size() * 4), o_gl = place(plan.group_leaves.size() * 4),
               o_gr = place(grow.size() * 4);
  struct Temp {
    uint8_t *p = nullptr;
    ~Temp() { cudaFree(p); }
  } temp;
  cudaError_t e = alloc(&temp.p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return e;
  }
  uint8_t *d = temp.p;
  std::vector<uint8_t> tab(bytes - o_leaf);  // the tables, uploaded at once
  auto put = [&](size_t at, const void *src, size_t n) {
    if (n > 0) std::memcpy(tab.data() + (at - o_leaf), src, n);
  };
  put(o_leaf, leaves.data(), leaves.size() * sizeof(PackLeaf));
  put(o_blk, plan.blocks.data(), plan.blocks.size() * sizeof(Block));
  put(o_pc, plan.pieces.data(), plan.pieces.size() * sizeof(Piece));
  put(o_col, pcol.data(), pcol.size() * 4);
  put(o_gb, plan.group_leaf_begin.data(), plan.group_leaf_begin.size() * 4);
  put(o_gl, plan.group_leaves.data(), plan.group_leaves.size() * 4);
  put(o_gr, grow.data(), grow.size() * 4);
  e = cudaMemcpy(d + o_leaf, tab.data(), tab.size(), cudaMemcpyHostToDevice);
  Stager stager;
  if (e == cudaSuccess) e = stager.to_device(pieces, words, reinterpret_cast<double *>(d));
  if (e == cudaSuccess) {
    const PackArgs a{reinterpret_cast<const double *>(d),
                     reinterpret_cast<const PackLeaf *>(d + o_leaf),
                     d_recs,
                     d_ctas,
                     reinterpret_cast<const Block *>(d + o_blk),
                     reinterpret_cast<const Piece *>(d + o_pc),
                     reinterpret_cast<const uint32_t *>(d + o_col),
                     reinterpret_cast<const uint32_t *>(d + o_gb),
                     reinterpret_cast<const uint32_t *>(d + o_gl),
                     reinterpret_cast<const uint32_t *>(d + o_gr),
                     d_stream};
    const dim3 grid((unsigned)plan.num_ctas, kRunsAtOnce);
    if (plan.precision == kBF16) k_pack<kBF16><<<grid, kPackThreads>>>(a);
    else if (plan.precision == kFP32) k_pack<kFP32><<<grid, kPackThreads>>>(a);
    else k_pack<kFP64><<<grid, kPackThreads>>>(a);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
  }
  return e;
}

}  // namespace hbx
