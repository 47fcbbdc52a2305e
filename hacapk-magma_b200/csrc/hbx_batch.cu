// hbx_batch.cu -- vector kernels of the batched BiCGSTAB over many
// independent H-matrices packed as one block-diagonal H (no counterpart in
// the reference, which solves one body per run).  Instance k owns rows
// [off[k], off[k+1]) of every vector; each instance runs the recurrence of
// HACApK_SOLVER.c:602-732 with its own scalars (MrScal, one per instance) and
// its own stop test ||r||/||b|| < tol, checked before every step as
// HACApK_SOLVER.c:631 does.  A finished instance keeps u and r, and its p and
// t are zero so its rows of the block-diagonal products are zero.
//
// An instance's dots need its rows alone, so a group of CTAs takes an
// instance and goes from the product to the next product's input in one
// launch: k_bt_mid forms alpha and t, k_bt_end zeta, u, r, beta and p, the
// float copy of t or p that an FP32 or BF16 product reads included.  Two
// launches and two products a step; what bounds them is their chain of
// reductions (one or two, through the cluster's shared memory), and the
// group's size (1, 2, 4 or 8 CTAs by the instance's own rows) keeps at most four
// rows per thread up to 16,384 rows.  The step of 24 bodies of 320 to 5,120
// rows took 17 launches beside the products before (dots, scalars, updates,
// float copies, prefix counts: 40 us, and the host could not launch them fast
// enough); these two take 12.
//
// The launch's clusters are of the largest group's size, and smaller groups
// share one (the groups lie in descending size, so none straddles two).  A
// cluster barrier then takes in more than its group, and a group that has
// returned no longer counts: no group waits for anything but the others' next
// barrier or end.
//
// Dot products are compensated (Dot2), as the single-body solver's: each
// thread in row order, a warp butterfly, the CTA's warps in order, the
// cluster's CTAs in order, so every run sums in the same order.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "../../include/hacapk_b200.h"
#include "hbx_device.cuh"
#include "hbx_engine.h"

namespace hbx {
namespace {

namespace cg = cooperative_groups;

constexpr int kBt = 512;       // threads of a CTA
constexpr int kBtRows = 2048;  // rows that a CTA takes before its instance gets twice as many CTAs: 4 a thread
constexpr int kMaxCluster = 8;

// The calling CTA's place and the rows of the calling thread: its instance's,
// in turn over the group's CTAs.
struct Rows {
  int k;        // instance (-1: a CTA past the last group)
  int size, rank, base;  // CTAs of the group, this one's place, the first one's rank in the cluster
  int i1;       // end row of the instance
  int first, step;
};
__device__ __forceinline__ Rows my_rows(const BtCta *map, const int *off) {
  const BtCta c = map[blockIdx.x];
  Rows R{c.k, c.size, c.rank, c.base, 0, 0, kBt};
  if (c.k < 0) return R;
  R.i1 = off[c.k + 1];
  R.first = off[c.k] + c.rank * kBt + (int)threadIdx.x;
  R.step = c.size * kBt;
  return R;
}
__device__ __forceinline__ void group_sync(const Rows &R, cg::cluster_group &cl) {
  if (R.size > 1) cl.sync();
  else __syncthreads();
}

// tot[q]: the sums of acc[q] over the group, the same in every thread.
// `sh` is written again only after another group_sync.
template <int NQ>
struct ClusterSums {
  Acc2 warp[kBt / 32][NQ];
  Acc2 cta[NQ];
};
template <int NQ>
__device__ __forceinline__ void group_totals(const Rows &R, cg::cluster_group &cl, const Acc2 (&acc)[NQ],
                                             ClusterSums<NQ> &sh, double (&tot)[NQ]) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const Acc2 m = warp_merge(acc[q]);
    if (lane == 0) sh.warp[w][q] = m;
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    Acc2 t = sh.warp[0][threadIdx.x];
    for (int k = 1; k < kBt / 32; ++k) t = acc2_merge(t, sh.warp[k][threadIdx.x]);
    sh.cta[threadIdx.x] = t;
  }
  group_sync(R, cl);
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    Acc2 t = *cl.map_shared_rank(&sh.cta[q], R.base);
    for (int c = 1; c < R.size; ++c) t = acc2_merge(t, *cl.map_shared_rank(&sh.cta[q], R.base + c));
    tot[q] = t.s + t.c;
  }
}

// The CTA that finishes last in the grid (one thread of each calls with its
// results written) counts the active instances: pre[k] = those below k,
// flags: any_active, done.
__device__ __forceinline__ void count_active(int count, const MrScal *s, int *pre, BtFlags *f) {
  __shared__ bool last;
  __shared__ int part[kBt];
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned t = atomicAdd(&f->ticket, 1u);
    last = t == gridDim.x - 1;
    if (last) f->ticket = 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int t = threadIdx.x, per = (count + kBt - 1) / kBt;
  const int k0 = min(count, t * per), k1 = min(count, k0 + per);
  int c = 0;
  for (int k = k0; k < k1; ++k) c += __ldcg(&s[k].active) ? 1 : 0;
  part[t] = c;
  __syncthreads();
  for (int o = 1; o < kBt; o <<= 1) {
    const int v = t >= o ? part[t - o] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  if (pre) {
    int run = part[t] - c;  // active instances below k0
    for (int k = k0; k < k1; ++k) {
      pre[k] = run;
      run += __ldcg(&s[k].active) ? 1 : 0;
    }
    if (t == kBt - 1) pre[count] = part[t];
  }
  if (t == kBt - 1) {
    f->any = part[t] > 0;
    f->done = part[t] == 0;
  }
}

// out[k] = x . x over the rows of instance k
__global__ void __launch_bounds__(kBt) k_bt_norms(const BtCta *map, const int *off, const double *x, double *out) {
  cg::cluster_group cl = cg::this_cluster();
  __shared__ ClusterSums<1> sh;
  const Rows R = my_rows(map, off);
  if (R.k < 0) return;
  Acc2 acc[1] = {{0.0, 0.0}};
  for (int i = R.first; i < R.i1; i += R.step) dot2_add(acc[0], x[i], x[i]);
  double tot[1];
  group_totals<1>(R, cl, acc, sh, tot);
  if (R.rank == 0 && threadIdx.x == 0) out[R.k] = tot[0];
  group_sync(R, cl);  // every CTA has read the others' sums
}

// Start of the solve, r = b - H u formed: rh = r, p = r, the stop test; an
// instance runs while ||r||/||b|| >= tol (rtol: per instance).
__global__ void __launch_bounds__(kBt) k_bt_init(BtStep a, const double *b, double tol, const double *rtol) {
  cg::cluster_group cl = cg::this_cluster();
  __shared__ ClusterSums<2> sh;
  const Rows R = my_rows(a.grid.map, a.off);
  if (R.k < 0) {
    count_active(a.count, a.sc, a.pre, a.flags);
    return;
  }
  Acc2 acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int i = R.first; i < R.i1; i += R.step) {
    const double rv = a.r[i], bv = b[i];
    a.rh[i] = rv;
    dot2_add(acc[0], rv, rv);
    dot2_add(acc[1], bv, bv);
  }
  double tot[2];
  group_totals<2>(R, cl, acc, sh, tot);
  const double rr = tot[0], bn = std::sqrt(tot[1]);
  MrScal q{};
  q.rho = rr;
  q.rr = rr;
  const double rel = bn > 0.0 ? std::sqrt(rr) / bn : 0.0;
  if (rtol) tol = rtol[R.k];  // per-instance tolerance (the inner solves of a refined batch)
  q.rtol = tol;
  q.status = 0;
  if (!isfinite(rel)) q.status = HBX_ERR_BREAKDOWN;
  else if (rel >= tol) q.active = a.max_iter > 0 ? 1 : 0;
  if (rel >= tol && a.max_iter <= 0) q.status = HBX_ERR_NOT_CONVERGED;
  for (int i = R.first; i < R.i1; i += R.step) {
    const double pv = q.active ? a.r[i] : 0.0;
    a.p[i] = pv;
    if (a.x32) a.x32[i] = (float)pv;
    if (!q.active) a.t[i] = 0.0;
  }
  if (R.rank == 0 && threadIdx.x == 0) {
    a.bnorm[R.k] = bn;
    a.sc[R.k] = q;
  }
  group_sync(R, cl);
  count_active(a.count, a.sc, a.pre, a.flags);
}

// After Ap: alpha = rho / (rh . Ap), t = r - alpha Ap
__global__ void __launch_bounds__(kBt) k_bt_mid(BtStep a) {
  cg::cluster_group cl = cg::this_cluster();
  __shared__ ClusterSums<1> sh;
  if (*(volatile const int *)&a.flags->done) return;
  const Rows R = my_rows(a.grid.map, a.off);
  if (R.k < 0) return;
  MrScal &S = a.sc[R.k];
  if (!S.active) return;  // the same in the whole group
  const double rho = S.rho;
  Acc2 acc[1] = {{0.0, 0.0}};
  for (int i = R.first; i < R.i1; i += R.step) dot2_add(acc[0], a.rh[i], a.ap[i]);
  double tot[1];
  group_totals<1>(R, cl, acc, sh, tot);
  const double alpha = rho / tot[0];
  const bool bad = tot[0] == 0.0 || !isfinite(alpha);
  for (int i = R.first; i < R.i1; i += R.step) {
    const double tv = bad ? 0.0 : fma(-alpha, a.ap[i], a.r[i]);
    a.t[i] = tv;
    if (a.x32) a.x32[i] = (float)tv;
    if (bad) a.p[i] = 0.0;
  }
  group_sync(R, cl);  // the others' sums and S are read
  if (R.rank == 0 && threadIdx.x == 0) {
    if (bad) {
      S.active = 0;
      S.status = HBX_ERR_BREAKDOWN;
    } else {
      S.alpha = alpha;
    }
  }
}

// After At: zeta = (At . t) / (At . At), u += alpha p + zeta t, r = t - zeta
// At, rho_new = rh . r, rr = r . r; the stop test; p = r + beta (p - zeta Ap).
// At . At == 0 means At = 0: zeta = 0 keeps the step's BiCG half (u += alpha p,
// r = t); the stop test then ends the instance as converged when that r is
// below the tolerance and as a breakdown otherwise, before any further step.
__global__ void __launch_bounds__(kBt) k_bt_end(BtStep a) {
  cg::cluster_group cl = cg::this_cluster();
  __shared__ ClusterSums<2> sh, sh2;
  if (*(volatile const int *)&a.flags->done) return;
  const Rows R = my_rows(a.grid.map, a.off);
  MrScal q{};
  if (R.k >= 0) q = a.sc[R.k];
  if (q.active) {
    Acc2 acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (int i = R.first; i < R.i1; i += R.step) {
      const double av = a.at[i];
      dot2_add(acc[0], av, a.t[i]);
      dot2_add(acc[1], av, av);
    }
    double tot[2];
    group_totals<2>(R, cl, acc, sh, tot);
    const double zeta = tot[1] != 0.0 ? tot[0] / tot[1] : 0.0;
    bool run = isfinite(zeta);
    if (!run) {
      q.status = HBX_ERR_BREAKDOWN;  // u and r of the previous step stay
    } else {
      q.zeta = zeta;
      acc[0] = acc[1] = Acc2{0.0, 0.0};
      for (int i = R.first; i < R.i1; i += R.step) {
        const double tv = a.t[i];
        a.u[i] = fma(zeta, tv, fma(q.alpha, a.p[i], a.u[i]));
        const double rv = fma(-zeta, a.at[i], tv);
        a.r[i] = rv;
        dot2_add(acc[0], a.rh[i], rv);
        dot2_add(acc[1], rv, rv);
      }
      group_totals<2>(R, cl, acc, sh2, tot);
      const double rho_new = tot[0], rr = tot[1], bn = a.bnorm[R.k];
      q.iters += 1;
      q.rr = rr;
      const double rel = bn > 0.0 ? std::sqrt(rr) / bn : 0.0;
      if (!isfinite(rel)) {
        run = false;
        q.status = HBX_ERR_BREAKDOWN;
      } else if (rel < q.rtol) {
        run = false;
      } else if (q.iters >= a.max_iter) {
        run = false;
        q.status = HBX_ERR_NOT_CONVERGED;
      } else {
        const double beta = (q.alpha / q.zeta) * (rho_new / q.rho);
        if (q.zeta == 0.0 || !isfinite(beta)) {
          run = false;
          q.status = HBX_ERR_BREAKDOWN;
        } else {
          q.beta = beta;
          q.rho = rho_new;
        }
      }
    }
    q.active = run ? 1 : 0;
    for (int i = R.first; i < R.i1; i += R.step) {
      const double pv = run ? fma(q.beta, fma(-q.zeta, a.ap[i], a.p[i]), a.r[i]) : 0.0;
      a.p[i] = pv;
      if (a.x32) a.x32[i] = (float)pv;
      if (!run) a.t[i] = 0.0;
    }
    group_sync(R, cl);  // the others' sums and scalars are read
    if (R.rank == 0 && threadIdx.x == 0) a.sc[R.k] = q;
  }
  count_active(a.count, a.sc, a.pre, a.flags);
}

// r[i] = 0 for the rows of instances whose flag is 0
__global__ void k_bt_mask(size_t n, const int *rinst, const int *flag, double *r) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    if (!flag[rinst[i]]) r[i] = 0.0;
}

template <class... P, class... A>
cudaError_t launch_clusters(void (*kern)(P...), int ctas, int cluster, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kBt);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

}  // namespace

// Each instance's group by its own rows: with every group sized by the largest
// instance, a step of 1,000 bodies of 320 rows beside one of 20,480 took 773 us,
// more than the 17 launches (580); this way it takes 533 where those take 622
// (another draw of the bodies).  One body of 1,280 rows alone 90 -> 61 us a step,
// 20,480 183 -> 139, 81,920 534 -> 464, 327,680 (80 rows a thread) 2,142 -> 2,038.
int bt_map(const std::vector<int> &off, std::vector<BtCta> &map) {
  const int count = (int)off.size() - 1;
  auto size_of = [&](int k) {
    int c = 1;
    while (c < kMaxCluster && off[k + 1] - off[k] > c * kBtRows) c *= 2;
    return c;
  };
  int cluster = 1;
  for (int k = 0; k < count; ++k) cluster = std::max(cluster, size_of(k));
  map.clear();
  for (int c = cluster; c > 0; c /= 2)
    for (int k = 0; k < count; ++k)
      if (size_of(k) == c)
        for (int r = 0; r < c; ++r)
          map.push_back(BtCta{k, (uint8_t)c, (uint8_t)r, (uint8_t)((map.size() - r) % cluster), 0});
  while (map.size() % cluster) map.push_back(BtCta{-1, 1, 0, 0, 0});
  return cluster;
}

cudaError_t bt_launch_norms(const BtGrid &g, const int *off, const double *x, double *out, cudaStream_t s) {
  return launch_clusters(k_bt_norms, g.ctas, g.cluster, s, g.map, off, x, out);
}

cudaError_t bt_launch_init(const BtStep &a, const double *b, double tol, const double *rtol, cudaStream_t s) {
  return launch_clusters(k_bt_init, a.grid.ctas, a.grid.cluster, s, a, b, tol, rtol);
}

cudaError_t bt_launch_mask(size_t n, const int *rinst, const int *flag, double *r, cudaStream_t s) {
  k_bt_mask<<<(int)std::min<size_t>((n + 255) / 256, 148 * 8), 256, 0, s>>>(n, rinst, flag, r);
  return cudaGetLastError();
}

cudaError_t bt_launch_step(const BtStep &a, cudaStream_t s) {
  cudaError_t e;
  if ((e = a.matvec(a.ctx, a.p, a.ap, s)) != cudaSuccess) return e;
  if ((e = launch_clusters(k_bt_mid, a.grid.ctas, a.grid.cluster, s, a)) != cudaSuccess) return e;
  if ((e = a.matvec(a.ctx, a.t, a.at, s)) != cudaSuccess) return e;
  return launch_clusters(k_bt_end, a.grid.ctas, a.grid.cluster, s, a);
}

}  // namespace hbx
