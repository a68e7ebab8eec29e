// CG with the diagonal preconditioner on small grids: the whole solve in one
// launch of one thread-block cluster.
//
// As kernels of their own a CG iteration's three passes cost about 5 us each
// on a few thousand cells, all of it launch latency and the reductions' last
// block; the levels of an additive-correction cycle run hundreds of such
// iterations. Here a block keeps its cells' r, x, p and 1/c in registers,
// their couplings and p in shared memory, and reads neighbours of other
// blocks from theirs; an iteration is three cluster barriers. What bounds it:
// those barriers and the two block reductions. Measured an iteration: one block
// (up to kSmallCells cells, no cluster barrier) 1.8 us at 512 cells, 2.8 us at
// 2048; eight blocks 3.3 us at 4096 cells, 4.4 us at 16384. As kernels of their
// own the passes take 19 us an iteration at 32768 cells.
//
// Per element the arithmetic is CG::solve's (cg.cpp:10-182) in its order, as
// in k_cg_init / k_cg_p / k_cg_q / k_cg_xr; the sums are in tree order.
#pragma once

#include <cooperative_groups.h>

#include "pbg_ref_kernels.cuh"

namespace pbg {

constexpr int kSmallThreads = 512;
constexpr int kSmallPer = 4;                              // cells a thread
constexpr int kSmallCells = kSmallThreads * kSmallPer;    // cells a block
constexpr int kSmallCluster = 8;                          // blocks of the larger form

// Shared memory: seven coupling arrays and p (one more entry, kept at zero,
// for neighbours outside the domain).
inline size_t small_cg_smem() { return sizeof(double) * (8 * (size_t)kSmallCells + 2); }

template <int CL>
__device__ __forceinline__ void small_sync() {
  if constexpr (CL == 1) __syncthreads();
  else cooperative_groups::this_cluster().sync();
}

// Sums of NV values over the cluster, the same for every thread. part holds
// CL partials a value in every block.
template <int NV, int CL>
__device__ __forceinline__ void small_sum(double (&v)[NV], double (*warp)[kSmallThreads / 32], double (*part)[CL]) {
  constexpr int NW = kSmallThreads / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) warp[q][wid] = v[q];
  __syncthreads();
  if constexpr (CL == 1) {
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = warp[q][lane & (NW - 1)];
#pragma unroll
    for (int off = NW / 2; off > 0; off >>= 1)
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
    __syncthreads();   // warp is free again
  } else {
    auto cl = cooperative_groups::this_cluster();
    if (wid == 0) {
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        double s = warp[q][lane & (NW - 1)];
#pragma unroll
        for (int off = NW / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane < CL) *cl.map_shared_rank(&part[q][cl.block_rank()], lane) = s;
      }
    }
    cl.sync();
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double s = part[q][0];
#pragma unroll
      for (int c = 1; c < CL; ++c) s += part[q][c];
      v[q] = s;
    }
  }
}

template <int CL>
__global__ void __launch_bounds__(kSmallThreads, 1) k_cg_small(MatView<double> A, double *__restrict__ x,
                                                               const double *__restrict__ b, KrylovParams pr,
                                                               KrylovState *st, double *hist) {
  namespace cg = cooperative_groups;
  extern __shared__ double sh[];
  __shared__ double warp[2][kSmallThreads / 32], part[2][2][CL];
  __shared__ double stale[kStaleMax];
  __shared__ int stop_flag;
  const int rank = CL == 1 ? 0 : (int)cg::this_cluster().block_rank();
  const long long N = A.ncell();
  const int m = (int)((N + CL - 1) / CL);   // cells of a block
  const int first = rank * m;
  double *cf = sh, *ps = sh + 7 * (size_t)kSmallCells;
  const KnownDiv dV(pr.dV);
  const double nc = (double)N;
  auto res_of = [&](double d) { return res_norm(d, nc, pr.scale); };

  // own cells: e = threadIdx + 512 u; neighbours' p by their address in the
  // cluster's shared memory
  double r[kSmallPer], xv[kSmallPer], p[kSmallPer], mc[kSmallPer];
  const double *nb[kSmallPer][6];
  if (threadIdx.x == 0) { ps[kSmallCells] = 0.0; stop_flag = 0; }
  double v2[2] = {0.0, 0.0};
#pragma unroll
  for (int u = 0; u < kSmallPer; ++u) {
    const int e = threadIdx.x + kSmallThreads * u;
    const long long g = first + e;
    r[u] = xv[u] = p[u] = mc[u] = 0.0;
#pragma unroll
    for (int f = 0; f < 6; ++f) nb[u][f] = ps + kSmallCells;
    if (e < m && g < N) {
      const Pos q = pos_of(g, A.ny, A.nz);
      const Nb<double> a = coeffs(A, g, q);
      const NbIdx n = nb_index(A, g, q);
      const double c = A.c[g];
      const double av[6] = {a.w, a.e, a.s, a.n, a.b, a.t};
      const long long ni[6] = {n.w, n.e, n.s, n.n, n.b, n.t};
      cf[e] = c;
#pragma unroll
      for (int f = 0; f < 6; ++f) {
        cf[(f + 1) * kSmallCells + e] = av[f];
        if (ni[f] >= 0) {
          const int owner = (int)(ni[f] / m);
          double *at = ps + (ni[f] - (long long)owner * m);
          if constexpr (CL == 1) nb[u][f] = at;
          else nb[u][f] = cg::this_cluster().map_shared_rank(at, owner);
        }
      }
      // r = b - A x in y_m_A_x's order (scalar_operators.cpp:22-46)
      double xs[6];
#pragma unroll
      for (int f = 0; f < 6; ++f) xs[f] = ni[f] >= 0 ? x[ni[f]] : 0.0;
      xv[u] = x[g];
      double t = __dsub_rn(b[g], __dmul_rn(c, xv[u]));
      t = __dadd_rn(t, __dadd_rn(__dmul_rn(a.w, xs[0]), __dmul_rn(a.e, xs[1])));
      t = __dadd_rn(t, __dadd_rn(__dmul_rn(a.s, xs[2]), __dmul_rn(a.n, xs[3])));
      t = __dadd_rn(t, __dadd_rn(__dmul_rn(a.b, xs[4]), __dmul_rn(a.t, xs[5])));
      r[u] = t;
      mc[u] = __ddiv_rn(1.0, c);
      v2[0] += voldiv(t, t, dV);
      v2[1] += __dmul_rn(t, __dmul_rn(t, mc[u]));
    }
  }
  if constexpr (CL > 1) small_sync<CL>();   // every block runs before its shared memory is written
  small_sum<2, CL>(v2, warp, part[1]);      // its barrier: every block has read x
  const double res0 = res_of(v2[0]);
  double res = res0, rho = v2[1], rho_old = 0.0, alfa = 0.0, beta = 0.0, pq = 0.0;
  int iterations = 0, it = 0, status = ST_RUNNING, converged = 0;
  const int ns = stale_entries(pr.stalecount);
  if (threadIdx.x == 0 && ns > 0) {
    for (int q = 0; q < ns; ++q) stale[q] = 1.0e24;   // boil::unreal
    stale[ns - 1] = res0;
  }
  if (res0 < pr.res_tol) { status = ST_INITIAL; converged = 1; }
  else if (pr.maxit <= 0) status = ST_MAXITER;
  while (status == ST_RUNNING) {
    beta = it == 0 ? 0.0 : __ddiv_rn(rho, rho_old);
#pragma unroll
    for (int u = 0; u < kSmallPer; ++u) {
      const double z = __dmul_rn(r[u], mc[u]);
      p[u] = it == 0 ? z : __dadd_rn(z, __dmul_rn(beta, p[u]));
      if (threadIdx.x + kSmallThreads * u < m) ps[threadIdx.x + kSmallThreads * u] = p[u];
    }
    small_sync<CL>();
    double q[kSmallPer], v1[1] = {0.0};
#pragma unroll
    for (int u = 0; u < kSmallPer; ++u) {
      const int e = threadIdx.x + kSmallThreads * u;
      q[u] = 0.0;
      if (e >= m) continue;
      const double *c = cf + e;   // A p in A_x's order (scalar_operators.cpp:49-72)
      double y = __dmul_rn(c[0], p[u]);
      y = __dsub_rn(y, __dadd_rn(__dmul_rn(c[kSmallCells], *nb[u][0]), __dmul_rn(c[2 * kSmallCells], *nb[u][1])));
      y = __dsub_rn(y, __dadd_rn(__dmul_rn(c[3 * kSmallCells], *nb[u][2]), __dmul_rn(c[4 * kSmallCells], *nb[u][3])));
      y = __dsub_rn(y, __dadd_rn(__dmul_rn(c[5 * kSmallCells], *nb[u][4]), __dmul_rn(c[6 * kSmallCells], *nb[u][5])));
      if (first + e >= N) y = 0.0;
      q[u] = y;
      v1[0] += __dmul_rn(p[u], y);
    }
    small_sum<1, CL>(v1, warp, part[0]);
    pq = v1[0];
    alfa = __ddiv_rn(rho, pq);
    v2[0] = v2[1] = 0.0;
#pragma unroll
    for (int u = 0; u < kSmallPer; ++u) {
      xv[u] = __dadd_rn(xv[u], __dmul_rn(alfa, p[u]));
      r[u] = __dsub_rn(r[u], __dmul_rn(alfa, q[u]));
      if (first + threadIdx.x + kSmallThreads * u < N && threadIdx.x + kSmallThreads * u < m) {
        v2[0] += voldiv(r[u], r[u], dV);
        v2[1] += __dmul_rn(r[u], __dmul_rn(r[u], mc[u]));
      }
    }
    small_sum<2, CL>(v2, warp, part[1]);
    res = res_of(v2[0]);
    if (rank == 0 && threadIdx.x == 0 && hist && it < pr.hist_cap) hist[it] = res;
    iterations = it + 1;
    const bool minok = it >= pr.mini - 1;
    if ((res < pr.res_tol && minok) || (res < res0 * pr.res_rat && minok)) {
      converged = 1; status = ST_CONVERGED;
      break;
    }
    if (ns > 0) {   // the staleness window (cg.cpp:138-160), the same in every block
      if (threadIdx.x == 0) stop_flag = stale_step(stale, ns, res);
      __syncthreads();
      if (stop_flag) { status = ST_STALE; break; }
    }
    if (!(res == res)) { status = ST_NAN; break; }
    rho_old = rho;
    rho = v2[1];
    ++it;
    if (it >= pr.maxit) status = ST_MAXITER;
  }
  small_sync<CL>();   // no block leaves while its shared memory may be read
#pragma unroll
  for (int u = 0; u < kSmallPer; ++u) {
    const int e = threadIdx.x + kSmallThreads * u;
    if (e < m && first + e < N && status != ST_INITIAL) x[first + e] = xv[u];
  }
  if (rank == 0 && threadIdx.x == 0) {
    st->res0 = res0; st->res = res; st->rho = rho; st->rho_old = rho_old;
    st->alfa = alfa; st->beta = beta; st->pq = pq; st->ncell = nc;
    st->iter = it; st->iterations = iterations; st->converged = converged;
    st->status = status; st->done = 1; st->pending_x = 0;
  }
}

// The form for this grid: blocks of the cluster, 0 where it does not fit.
inline int small_cg_blocks(const MatView<double> &A, int solver, int prec, bool exact) {
  if (solver != 0 || prec != 0 || exact) return 0;
  if (A.ncell() <= kSmallCells) return 1;
  if (A.ncell() <= (long long)kSmallCells * kSmallCluster) return kSmallCluster;
  return 0;
}

inline void enqueue_small_cg(const MatView<double> &A, double *x, const double *b, const KrylovParams &pr,
                             int blocks, KrylovState *st, double *hist, cudaStream_t s) {
  const size_t smem = small_cg_smem();
  auto go = [&](auto kern) {
    PBG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PBG_CUDA(cudaLaunchKernelEx(&cfg, kern, A, x, b, pr, st, hist));
    note_launch();
  };
  if (blocks == 1) go(k_cg_small<1>);
  else go(k_cg_small<kSmallCluster>);
}

}  // namespace pbg
