// hbx_mrhs_solve.cu -- vector kernels of the multi-RHS BiCGSTAB (no
// counterpart in the reference).  Every vector is nd x kNrhs doubles,
// row-major (the kNrhs right-hand sides of a row adjacent); each right-hand
// side j runs its own BiCGSTAB recurrence of HACApK_SOLVER.c:602-732 with its
// own scalars and stops on its own (a convergence mask): a finished RHS keeps
// its x and r, and its p is fed to the product as zeros.
//
// Layout: a warp takes whole rows, lane l the right-hand sides 2l and 2l + 1
// (16 bytes a lane, the scalars of its two in registers for the whole launch);
// the warps of the grid take rows in turn.  A dot product is summed per lane,
// then over the block's warps in warp order, then over the blocks by the block
// that finishes last (16 lanes per right-hand side, each every sixteenth block,
// added in lane order): the same order on every run, and the scalar that
// follows from the dots is formed there, so a step is five launches beside its
// two products.  One block of 32 warps per SM: the last block's sum over the
// blocks is a chain of round trips to L2, and 148 blocks make it short.  Per
// step on 20,480 unknowns: one thread per element with its scalars read for
// each, 296 blocks of 256, and single-block launches for the scalars 72 us;
// this with 296 blocks of 16 warps 54; with 148 of 32 44 (the bytes take 30).
#include <algorithm>
#include <cmath>

#include "../../include/hacapk_b200.h"
#include "hbx_engine.h"

namespace hbx {
namespace {

constexpr int kMrWarps = 32;
constexpr int kMrThreads = 32 * kMrWarps;
constexpr int kSumLanes = kMrThreads / kNrhs;  // lanes per right-hand side over the blocks

// Right-hand sides 2 lane and 2 lane + 1 of row i; `vec`: v lies on a 16-byte
// boundary (the solver's own vectors always do, a caller's need not).
__device__ __forceinline__ double2 ld_pair(const double *v, size_t i, bool vec) {
  const double *p = v + i * kNrhs + 2 * (threadIdx.x & 31);
  if (vec) return *reinterpret_cast<const double2 *>(p);
  return make_double2(p[0], p[1]);
}
__device__ __forceinline__ void st_pair(double *v, size_t i, double2 x) {
  *reinterpret_cast<double2 *>(v + i * kNrhs + 2 * (threadIdx.x & 31)) = x;
}

// use(i, v) for every row i of the calling warp, v = the row's pairs of the N
// vectors; kRowsAtOnce rows are loaded before the first is used (the stores of
// a row would otherwise hold back the next row's loads).
constexpr int kRowsAtOnce = 2;
template <int N, class F>
__device__ __forceinline__ void for_rows(int nd, const double *const (&vec)[N], bool on16, F use) {
  const int step = gridDim.x * kMrWarps;
  for (int i0 = blockIdx.x * kMrWarps + (threadIdx.x >> 5); i0 < nd; i0 += step * kRowsAtOnce) {
    double2 v[kRowsAtOnce][N];
#pragma unroll
    for (int u = 0; u < kRowsAtOnce; ++u)
#pragma unroll
      for (int k = 0; k < N; ++k)
        v[u][k] = i0 + u * step < nd ? ld_pair(vec[k], (size_t)(i0 + u * step), on16) : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < kRowsAtOnce; ++u)
      if (i0 + u * step < nd) use((size_t)(i0 + u * step), v[u]);
  }
}

// acc[q]: the calling lane's sums of dot q over its rows, for its two
// right-hand sides.  True in the block that finishes last, with tot[q] the
// totals of right-hand side threadIdx.x in threads 0..kNrhs-1.
template <int NQ>
__device__ __forceinline__ bool totals(const double2 (&acc)[NQ], double *part, unsigned *ticket, double (&tot)[NQ]) {
  __shared__ double red[kMrWarps][kNrhs];
  __shared__ bool last;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, j = threadIdx.x % kNrhs, l = threadIdx.x / kNrhs;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    red[w][2 * lane] = acc[q].x;
    red[w][2 * lane + 1] = acc[q].y;
    __syncthreads();
    if (threadIdx.x < kNrhs) {
      double v = red[0][j];
#pragma unroll
      for (int k = 1; k < kMrWarps; ++k) v += red[k][j];
      part[((size_t)blockIdx.x * NQ + q) * kNrhs + j] = v;
      __threadfence();
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const unsigned t = atomicAdd(ticket, 1u);
    last = t == gridDim.x - 1;
    if (last) *ticket = 0;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double v = 0.0;
#pragma unroll 8
    for (int b = l; b < (int)gridDim.x; b += kSumLanes) v += __ldcg(part + ((size_t)b * NQ + q) * kNrhs + j);
    red[l][j] = v;
    __syncthreads();
    if (l == 0) {
      tot[q] = red[0][j];
#pragma unroll
      for (int k = 1; k < kSumLanes; ++k) tot[q] += red[k][j];
    }
    __syncthreads();
  }
  return true;
}
static_assert(kSumLanes <= kMrWarps, "totals() sums its lanes in the warps' array");

// *any_active = some right-hand side runs on (the last block, every thread).
__device__ __forceinline__ void set_any(bool active, int *any_active) {
  const int any = __syncthreads_or(active ? 1 : 0);
  if (threadIdx.x == 0) *any_active = any;
}

__device__ __forceinline__ void add_prod(double2 &a, double2 x, double2 y) {
  a.x = fma(x.x, y.x, a.x);
  a.y = fma(x.y, y.y, a.y);
}

// out[j] = ||v_j||^2 (the outer loop)
__global__ void __launch_bounds__(kMrThreads) k_mr_norms(int nd, const double *v, bool vec, double *part,
                                                         unsigned *ticket, double *out) {
  double2 acc[1] = {{0.0, 0.0}};
  for_rows<1>(nd, {v}, vec, [&](size_t, const double2 (&x)[1]) { add_prod(acc[0], x[0], x[0]); });
  double tot[1];
  if (totals<1>(acc, part, ticket, tot) && threadIdx.x < kNrhs) out[threadIdx.x] = tot[0];
}

// The start of an inner solve: r = rh = R, x = 0, and the first scalars,
// rho = rh.r = r.r; an RHS runs while its mask is set and ||r|| is above its
// threshold.  (p and Ap are first written by the first step.)
__global__ void __launch_bounds__(kMrThreads) k_mr_setup(int nd, const double *R, double *r, double *rh, double *x,
                                                         const double *thresh, const int *mask, MrScal *s,
                                                         double *part, unsigned *ticket, int *any_active) {
  double2 acc[1] = {{0.0, 0.0}};
  for_rows<1>(nd, {R}, true, [&](size_t i, const double2 (&v)[1]) {
    st_pair(r, i, v[0]);
    st_pair(rh, i, v[0]);
    st_pair(x, i, make_double2(0.0, 0.0));
    add_prod(acc[0], v[0], v[0]);
  });
  double tot[1];
  if (!totals<1>(acc, part, ticket, tot)) return;
  bool active = false;
  if (threadIdx.x < kNrhs) {
    const int j = threadIdx.x;
    MrScal q{};
    q.rho = tot[0];
    q.rr = tot[0];
    q.rtol = thresh[j];
    active = mask[j] && std::sqrt(tot[0]) > q.rtol;
    q.active = active ? 1 : 0;
    q.status = 0;
    s[j] = q;
  }
  set_any(active, any_active);
}

// p = r + beta (p - zeta ap) (p = r on an RHS's first step); p32 = p as
// float, zero for a finished RHS.
__global__ void __launch_bounds__(kMrThreads) k_mr_p(int nd, const MrScal *s, const int *any, const double *r, double *p,
                                                     const double *ap, float *p32) {
  if (!*any) return;
  const int lane = threadIdx.x & 31;
  const MrScal a = s[2 * lane], b = s[2 * lane + 1];
  for_rows<3>(nd, {r, p, ap}, true, [&](size_t i, const double2 (&v)[3]) {
    double2 pv = make_double2(0.0, 0.0);
    if (a.active || b.active) {
      const double2 rv = v[0], po = v[1], av = v[2];
      pv.x = !a.active ? po.x : a.iters == 0 ? rv.x : fma(a.beta, fma(-a.zeta, av.x, po.x), rv.x);
      pv.y = !b.active ? po.y : b.iters == 0 ? rv.y : fma(b.beta, fma(-b.zeta, av.y, po.y), rv.y);
      st_pair(p, i, pv);
    }
    *reinterpret_cast<float2 *>(p32 + i * kNrhs + 2 * lane) =
        make_float2(a.active ? (float)pv.x : 0.0f, b.active ? (float)pv.y : 0.0f);
  });
}

// rh . Ap and alpha = rho / (rh . Ap)
__global__ void __launch_bounds__(kMrThreads) k_mr_alpha(int nd, MrScal *s, const int *any, const double *rh,
                                                         const double *ap, double *part, unsigned *ticket) {
  if (!*any) return;
  double2 acc[1] = {{0.0, 0.0}};
  for_rows<2>(nd, {rh, ap}, true, [&](size_t, const double2 (&v)[2]) { add_prod(acc[0], v[0], v[1]); });
  double tot[1];
  if (!totals<1>(acc, part, ticket, tot) || threadIdx.x >= kNrhs) return;
  MrScal &q = s[threadIdx.x];
  if (!q.active) return;
  const double alpha = q.rho / tot[0];
  if (tot[0] == 0.0 || !isfinite(alpha)) {
    q.active = 0;
    q.status = HBX_ERR_BREAKDOWN;
    return;
  }
  q.alpha = alpha;
}

// t = r - alpha Ap, in r's place (a finished RHS keeps its r); t32 = t as
// float (zero for a finished RHS)
__global__ void __launch_bounds__(kMrThreads) k_mr_t(int nd, const MrScal *s, const int *any, double *r,
                                                     const double *ap, float *t32) {
  if (!*any) return;
  const int lane = threadIdx.x & 31;
  const MrScal a = s[2 * lane], b = s[2 * lane + 1];
  for_rows<2>(nd, {r, ap}, true, [&](size_t i, const double2 (&v)[2]) {
    double2 tv = make_double2(0.0, 0.0);
    if (a.active || b.active) {
      const double2 rv = v[0], av = v[1];
      if (a.active) tv.x = fma(-a.alpha, av.x, rv.x);
      if (b.active) tv.y = fma(-b.alpha, av.y, rv.y);
      st_pair(r, i, make_double2(a.active ? tv.x : rv.x, b.active ? tv.y : rv.y));
    }
    *reinterpret_cast<float2 *>(t32 + i * kNrhs + 2 * lane) = make_float2((float)tv.x, (float)tv.y);
  });
}

// At . t, At . At and zeta = (At . t) / (At . At)
__global__ void __launch_bounds__(kMrThreads) k_mr_zeta(int nd, MrScal *s, const int *any, const double *at,
                                                        const double *t, double *part, unsigned *ticket) {
  if (!*any) return;
  double2 acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
  for_rows<2>(nd, {at, t}, true, [&](size_t, const double2 (&v)[2]) {
    add_prod(acc[0], v[0], v[1]);
    add_prod(acc[1], v[0], v[0]);
  });
  double tot[2];
  if (!totals<2>(acc, part, ticket, tot) || threadIdx.x >= kNrhs) return;
  MrScal &q = s[threadIdx.x];
  if (!q.active) return;
  const double zeta = tot[1] != 0.0 ? tot[0] / tot[1] : 0.0;
  if (!isfinite(zeta)) {
    q.active = 0;
    q.status = HBX_ERR_BREAKDOWN;
    return;
  }
  q.zeta = zeta;
}

// x += alpha p + zeta t;  r = t - zeta At (t lies in r);  then rho_new = rh . r, rr = r . r;
// the stop test; beta for the next step
__global__ void __launch_bounds__(kMrThreads) k_mr_xr(int nd, MrScal *s, const double *p, const double *at,
                                                      const double *rh, double *x, double *r,
                                                      int max_iter, double *part, unsigned *ticket, int *any_active) {
  if (!*any_active) return;
  const int lane = threadIdx.x & 31;
  double2 acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
  {
    const MrScal a = s[2 * lane], b = s[2 * lane + 1];
    if (a.active || b.active)
      for_rows<5>(nd, {r, p, at, rh, x}, true, [&](size_t i, const double2 (&v)[5]) {
        const double2 tv = v[0], pv = v[1], av = v[2], hv = v[3];
        double2 xv = v[4], rv = tv;
        if (a.active) {
          xv.x = fma(a.zeta, tv.x, fma(a.alpha, pv.x, xv.x));
          rv.x = fma(-a.zeta, av.x, tv.x);
        }
        if (b.active) {
          xv.y = fma(b.zeta, tv.y, fma(b.alpha, pv.y, xv.y));
          rv.y = fma(-b.zeta, av.y, tv.y);
        }
        st_pair(x, i, xv);
        st_pair(r, i, rv);
        add_prod(acc[0], hv, rv);
        add_prod(acc[1], rv, rv);
      });
  }
  double tot[2];
  if (!totals<2>(acc, part, ticket, tot)) return;
  bool active = false;
  if (threadIdx.x < kNrhs && s[threadIdx.x].active) {
    MrScal q = s[threadIdx.x];
    const double rho_new = tot[0], rr = tot[1];
    q.iters += 1;
    q.rr = rr;
    if (!isfinite(rr)) {
      q.active = 0;
      q.status = HBX_ERR_BREAKDOWN;
    } else if (std::sqrt(rr) <= q.rtol) {
      q.active = 0;
    } else if (q.iters >= max_iter) {
      q.active = 0;
      q.status = HBX_ERR_NOT_CONVERGED;
    } else {
      const double beta = (q.alpha / q.zeta) * (rho_new / q.rho);
      if (q.zeta == 0.0 || !isfinite(beta)) {
        q.active = 0;
        q.status = HBX_ERR_BREAKDOWN;
      } else {
        q.beta = beta;
        q.rho = rho_new;
      }
    }
    s[threadIdx.x] = q;
    active = q.active != 0;
  }
  set_any(active, any_active);
}

// out (cols x rows) = in (rows x cols), 32 x 32 tiles
__global__ void k_mr_transpose(int rows, int cols, const double *in, double *out) {
  __shared__ double tile[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int r = by + k, c = bx + threadIdx.x;
    if (r < rows && c < cols) tile[k][threadIdx.x] = in[(size_t)r * cols + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int c = bx + k, r = by + threadIdx.x;
    if (r < rows && c < cols) out[(size_t)c * rows + r] = tile[threadIdx.x][k];
  }
}

// R (nd x kNrhs) = B - (HU)^T where HU is kNrhs x nd (one product per row)
__global__ void k_mr_resid(int nd, const double *B, const double *HU, double *R) {
  __shared__ double tile[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;  // bx: rows of R, by: RHS
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int j = by + k, i = bx + threadIdx.x;
    if (j < kNrhs && i < nd) tile[k][threadIdx.x] = HU[(size_t)j * nd + i];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int i = bx + k, j = by + threadIdx.x;
    if (i < nd && j < kNrhs) {
      const size_t e = (size_t)i * kNrhs + j;
      R[e] = B[e] - tile[threadIdx.x][k];
    }
  }
}

// U += D on the RHS whose mask is set
__global__ void __launch_bounds__(256) k_mr_add(size_t n, const int *mask, const double *D, double *U) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    if (mask[e % kNrhs]) U[e] += D[e];
}

bool on16(const double *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

int mr_row_blocks(int nd) { return std::max(1, std::min(148, (nd + kMrWarps - 1) / kMrWarps)); }

cudaError_t mr_launch_norms(int nd, const double *v, double *part, unsigned *ticket, double *out, cudaStream_t s) {
  k_mr_norms<<<mr_row_blocks(nd), kMrThreads, 0, s>>>(nd, v, on16(v), part, ticket, out);
  return cudaGetLastError();
}

cudaError_t mr_launch_setup(const MrStep &a, const double *R, const double *thresh, const int *mask, cudaStream_t s) {
  k_mr_setup<<<mr_row_blocks(a.nd), kMrThreads, 0, s>>>(a.nd, R, a.r, a.rh, a.x, thresh, mask, a.sc, a.part, a.ticket,
                                                        a.any_active);
  return cudaGetLastError();
}

cudaError_t mr_launch_step(const MrStep &a, cudaStream_t s) {
  const int nblk = mr_row_blocks(a.nd);
  cudaError_t e;
  k_mr_p<<<nblk, kMrThreads, 0, s>>>(a.nd, a.sc, a.any_active, a.r, a.p, a.ap, a.f32);
  if ((e = a.matmat(a.ctx, a.f32, a.ap, s)) != cudaSuccess) return e;
  k_mr_alpha<<<nblk, kMrThreads, 0, s>>>(a.nd, a.sc, a.any_active, a.rh, a.ap, a.part, a.ticket);
  k_mr_t<<<nblk, kMrThreads, 0, s>>>(a.nd, a.sc, a.any_active, a.r, a.ap, a.f32);
  if ((e = a.matmat(a.ctx, a.f32, a.at, s)) != cudaSuccess) return e;
  k_mr_zeta<<<nblk, kMrThreads, 0, s>>>(a.nd, a.sc, a.any_active, a.at, a.r, a.part, a.ticket);
  k_mr_xr<<<nblk, kMrThreads, 0, s>>>(a.nd, a.sc, a.p, a.at, a.rh, a.x, a.r, a.max_iter, a.part, a.ticket, a.any_active);
  return cudaGetLastError();
}

cudaError_t mr_launch_transpose(int rows, int cols, const double *in, double *out, cudaStream_t s) {
  dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
  k_mr_transpose<<<grid, block, 0, s>>>(rows, cols, in, out);
  return cudaGetLastError();
}

cudaError_t mr_launch_resid(int nd, const double *B, const double *HU, double *R, cudaStream_t s) {
  dim3 grid((nd + 31) / 32, (kNrhs + 31) / 32), block(32, 8);
  k_mr_resid<<<grid, block, 0, s>>>(nd, B, HU, R);
  return cudaGetLastError();
}

cudaError_t mr_launch_add(int nd, const int *mask, const double *D, double *U, cudaStream_t s) {
  const size_t n = (size_t)nd * kNrhs;
  k_mr_add<<<(int)std::min<size_t>((n + 255) / 256, 148 * 16), 256, 0, s>>>(n, mask, D, U);
  return cudaGetLastError();
}

}  // namespace hbx
