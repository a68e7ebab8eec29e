// Reference-parity solvers: host drivers and the kernels the C-ABI calls
// directly. See pbg_ref_kernels.cu.
#pragma once

#include <vector>

#include "pbg_common.cuh"
#include "pbg_session.h"
#include "pbg_sweeps.cuh"

namespace pbg {

// element of Scalar::dot_voldiv_avg: x*y/dV/dV (scalar.h:317-326). Two FP64
// divisions a cell (125 cycles each) bounded the kernels that form this sum;
// the corrected products give the same bits.
__device__ __forceinline__ double voldiv(double x, double y, const KnownDiv &dV) {
  return dV(dV(__dmul_rn(x, y)));
}

// res = sqrt(d/N/N)/scale (cg.cpp:68 and :115)
__device__ __forceinline__ double res_norm(double d, double ncell, double scale) {
  return __ddiv_rn(__dsqrt_rn(__ddiv_rn(__ddiv_rn(d, ncell), ncell)), scale);
}

// The staleness window of n residuals (cg.cpp:138-160): true if res is below
// none of them, else res takes the place of the oldest.
__device__ __forceinline__ int stale_entries(int stalecount) { return stalecount > kStaleMax ? kStaleMax : stalecount; }
__device__ __forceinline__ bool stale_step(double *win, int n, double res) {
  if (n <= 0) return false;
  bool stale = true;
  for (int q = 0; q < n; ++q)
    if (res < win[q]) { stale = false; break; }
  if (stale) return true;
  for (int q = 0; q < n - 1; ++q) win[q] = win[q + 1];
  win[n - 1] = res;
  return false;
}

// IC3 factor (compact arrays), run one launch per plane h = 5 i + 2 j + k.
// The other sweeps (IC0, IC2, Gauss-Seidel) are in pbg_sweeps.cuh.
struct Ic3Factor {
  double *c, *w, *s, *b, *tw, *ts, *nw;
};

struct KrylovParams {
  int prec = 0;            // Prec code: 0 diagonal, 1 IC0, 2 IC2, 3 IC3
  int mini, maxit, stalecount, hist_cap;
  double res_rat, res_tol, scale, dV;
  double *seq = nullptr;   // exact-order reduction terms (2 x ncell), null: tree
  const double *ci = nullptr;  // Jacobi / Gauss-Seidel: the matrix's stored 1/c (null: 1/c here)
};

// solver codes of the drivers below: 0 CG, 1 BiCGS, 2 CGS, 3 Jacobi,
// 4 Gauss-Seidel
struct RefKrylovWork {
  DBuf<double> r, q, pA, pB, rt, ph, v, s, sh, t, u;
  DBuf<double> mcd;                               // 1 / c (the diagonal preconditioner)
  DBuf<double> xold;                              // Gauss-Seidel: x before the sweep (periodic)
  const double *rhs = nullptr, *ci = nullptr;     // Jacobi / Gauss-Seidel operands of a solve
  DBuf<double> z, mc, mw, ms, mb, mtw, mts, mnw;  // IC preconditioner: z, and IC3's factor
  DBuf<double> mo;                                // sweeps: operands in march order
  DBuf<TagWord> words;                          // sweeps: exchange between tiles
  DBuf<unsigned> ticket;                          // sweeps: tickets [0..1], the stuck flag [2]
  unsigned long long epoch = 0;                   // sweeps: the last launch's epoch
  int *hstuck = nullptr;                          // pinned copy of the stuck flag
  ~RefKrylovWork();
  void ensure(size_t n, int solver);
  Ic3Factor ic3(size_t n);
  bool gs_march = false;                          // this Gauss-Seidel solve runs k_gs_sweep
  double *march(const SweepGeo &g, int planes);
  bool gs_alloc(const SweepGeo &g, cudaStream_t s);
  void sweep_alloc(size_t words_needed, cudaStream_t s);
  SweepSync sweep() {
    return {words.p, ticket.p, reinterpret_cast<int *>(ticket.p + 2), ++epoch};
  }
  // enqueue the copy of the stuck flag / after a synchronisation, throw if it is set
  void sweep_check_enqueue(cudaStream_t s);
  void sweep_check();
};

struct RefKrylovResult {
  int converged, status, iterations;
  double res0, res;
};

__global__ void k_spmv_ref(MatView<double> A, const double *__restrict__ x, double *__restrict__ y);
__global__ void k_resid_ref(MatView<double> A, const double *__restrict__ x,
                            const double *__restrict__ b, double *__restrict__ r);
__global__ void k_seq_sum(long long N, const double *__restrict__ a, const double *__restrict__ b,
                          double *seq, unsigned *count, double *out);
// Lays out an exact-order reduction scratch of exact_scratch_doubles(ncell)
// doubles at base (header, records, zeroed flags and counters).
void exact_scratch_init(double *base, long long ncell, cudaStream_t s);
__global__ void k_dot2(long long N, const double *__restrict__ x, const double *__restrict__ y,
                       double dV, double *part, unsigned *count, double *out);

void enqueue_ref_setup(const MatView<double> &A, double *x, const double *b, const KrylovParams &pr,
                       int solver, RefKrylovWork &w, const RedPool &red, KrylovState *st,
                       cudaStream_t s);
void enqueue_ref_iters(const MatView<double> &A, double *x, int solver, int count,
                       RefKrylovWork &w, const RedPool &red, KrylovState *st, double *hist,
                       cudaStream_t s, bool exact, int prec);
RefKrylovResult ref_krylov_solve(const MatView<double> &A, double *x, const double *b,
                                 const KrylovParams &pr, int solver, RefKrylovWork &w,
                                 const RedPool &red, KrylovState *st, KrylovState *hst,
                                 double *hist, cudaStream_t s);

struct RefACLevel {
  int nx = 0, ny = 0, nz = 0, CI = 1, CJ = 1, CK = 1;
  double dV = 0;
  Mat64 A;                 // coarse levels: general storage
  DBuf<double> phi, fnew;
  DBuf<uint8_t> aflag;
};

struct RefACParams {
  int init, loop;          // -1 none, 1 V, 2 F, 4 W, 5 flex (loop -1: "just solve")
  double toler, factor;
  int max_cyc, min_cyc, stop_if_div, priority_min_cyc;
  int mv[3], ms[3];
  double resrat_val, restol_val;
  bool use_linf = false;
  long long flex_visits = 1000000;
};

struct RefACResult {
  int converged, cycles, diverged, nhist;
  double res0, res;
  int visits;              // smoother calls of the last flex cycle
  int flex_capped;         // a flex cycle stopped at its visit bound
};

struct RefACCtx {
  cudaStream_t s;
  RefKrylovWork *w;
  RedPool *red;
  KrylovState *st;
  KrylovState *hst = nullptr;   // pinned host copy of st (flex: the smoother's converged flag)
  long long flex_visits = 1000000;
  double *dscal, *dmean, *hbuf;
  unsigned long long *dlinf;
  int mv[3], ms[3];
  double resrat_val, restol_val;
};

class RefAC {
 public:
  std::vector<RefACLevel> L;
  DBuf<double> fold;
  double *seq = nullptr;   // exact-order reduction terms, or null
  MatView<double> A0v{};
  // the smoother of every level (the Centered object's Linear): solver code
  // of the drivers above, its Prec code, and level 0's stored ci (or null)
  int sm_kind = 0, sm_prec = 0;
  const double *sm_ci0 = nullptr;
  // AC's own solver for call_solver (post-smoothing, coarsest level):
  // sol_kind -1 = the levels' smoother
  int sol_kind = -1, sol_prec = 0;
  // the level solvers' scale (dti * scale) and the dt of AC's residual measure
  double sm_scale = 1.0, res_dt = 1.0;

  void build(const MatView<double> &A0, const uint8_t *aflag0, double h, cudaStream_t s);
  MatView<double> view(int l) const;
  void coarsen_all(cudaStream_t s);
  RefACResult cycle(double *x, const double *b, const RefACParams &pa, RefACCtx &cx,
                    double *res_hist, int hist_cap);
  int nlevels() const { return (int)L.size(); }

 private:
  double residual(RedPool &red, double *dscal, unsigned long long *dlinf, double *hbuf,
                  cudaStream_t s, double *linf);
  void smooth(int l, int mi, double res_rat, double res_tol, int ms, RefKrylovWork &w,
              RedPool &red, KrylovState *st, cudaStream_t s, bool as_solver = false);
  void solve_l(int l, int mi, double res_rat, double res_tol, int ms, RefACCtx &cx);
  bool smooth_converged(int l, int mi, double res_rat, double res_tol, int ms, RefACCtx &cx);
  void restrict_to(int l, RedPool &red, double *dmean, cudaStream_t s);
  void interp_from(int l, cudaStream_t s);
  void run(int kind, int l, RefACCtx &cx);
  void v_cycle(int l, RefACCtx &cx);
  void fw_cycle(int l, RefACCtx &cx, bool w);
  void flex_cycle(int l, RefACCtx &cx);
  void full_cycle(int l, int kind, RefACCtx &cx);
  long long flex_calls_ = 0;
  bool flex_capped_ = false;
};

}  // namespace pbg
