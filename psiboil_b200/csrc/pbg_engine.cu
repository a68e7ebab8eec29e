// Host side of the engine solver (hierarchy set-up, K-cycle recursion,
// flexible CG and the mixed-precision refinement loop).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "pbg_engine.cuh"
#include "pbg_engine_kernels.cuh"
#include "pbg_vec.cuh"

namespace pbg {

// ---------------------------------------------------------------- hierarchy set-up kernels
// Output arrays of one level's numeric set-up: the FP64 operator, its
// inverse diagonal and, in the mixed path (c32 != nullptr), the FP32
// operator in edge form (c32 = diagonal excess, see kEdgeForm).
struct LevelOut {
  double *c, *w, *s, *b, *d;
  float *c32, *w32, *s32, *b32, *d32;
};

// Inverse diagonal and FP32 copies of a level whose FP64 operator is set.
__global__ void k_level_finish(EMat<double> A, LevelOut o) {
  GRID_LOOP(p, A.g.n) {
    const double c = A.c[p];
    // A pad cell (RowPad) has no diagonal and no couplings: its right-hand side
    // and A times anything are zero there, so whatever the prolongation leaves
    // in it reaches neither a dot product nor another cell.
    const double d = c != 0.0 ? 1.0 / c : 0.0;
    o.d[p] = d;
    if (o.c32) {
      const Pos q = A.g.pos(p);
      const double sum = offdiag(A, p, q, [](uint32_t) { return 1.0; });
      o.c32[p] = (float)(c - sum);
      o.w32[p] = (float)A.w[p]; o.s32[p] = (float)A.s[p]; o.b32[p] = (float)A.b[p];
      o.d32[p] = (float)d;
    }
  }
}

// Level 0 of the hierarchy in padded rows (RowPad) from the caller's: in 2-D
// the j couplings become the row's.
__global__ void k_pad_matrix(EMat<double> A, RowPad P, uint32_t rows, FastDiv dFP, double *__restrict__ c,
                             double *__restrict__ w, double *__restrict__ s, double *__restrict__ b) {
  GRID_LOOP(pp, rows * (uint32_t)P.FP) {
    const uint32_t row = dFP.div(pp);
    const int f = (int)(pp - row * (uint32_t)P.FP);
    const bool in = f < P.F;
    const uint32_t p = row * (uint32_t)P.F + (in ? f : 0);
    c[pp] = in ? A.c[p] : 0.0;
    w[pp] = in ? A.w[p] : 0.0;
    s[pp] = in && !P.two_d ? A.s[p] : 0.0;
    b[pp] = in ? (P.two_d ? A.s[p] : A.b[p]) : 0.0;
  }
}

// Galerkin coarse operator P^T A P for piecewise-constant aggregation by 2
// per direction (the sum over a block of every entry of A; each internal
// coupling enters the block's diagonal twice), FP64.
__global__ void k_galerkin(EMat<double> A, Geo H, LevelOut o) {
  const int fx = A.nx > 1 ? 2 : 1, fy = A.ny > 1 ? 2 : 1, fz = A.nz > 1 ? 2 : 1;
  GRID_LOOP(P, H.n) {
    Pos Q = H.pos(P);
    double c = 0.0, w = 0.0, s = 0.0, b = 0.0;
    const int i0 = Q.i * fx, j0 = Q.j * fy, k0 = Q.k * fz;
    for (int a = 0; a < fx && i0 + a < A.nx; ++a)
      for (int bb = 0; bb < fy && j0 + bb < A.ny; ++bb)
        for (int cc = 0; cc < fz && k0 + cc < A.nz; ++cc) {
          const uint32_t p = ((uint32_t)(i0 + a) * A.ny + (j0 + bb)) * A.nz + (k0 + cc);
          c += A.c[p];
          if (a == 0) w += A.w[p]; else c -= 2.0 * A.w[p];
          if (bb == 0) s += A.s[p]; else c -= 2.0 * A.s[p];
          if (cc == 0) b += A.b[p]; else c -= 2.0 * A.b[p];
        }
    o.c[P] = c; o.w[P] = w; o.s[P] = s; o.b[P] = b;
  }
}

// ---------------------------------------------------------------- dense coarsest
// Dense n x n matrix of the coarsest symmetric 7-point operator (D zeroed
// beforehand).
__global__ void k_dense_fill(EMat<double> A, double *__restrict__ D) {
  const uint32_t n = A.g.n, SI = A.g.nynz, SJ = (uint32_t)A.nz;
  GRID_LOOP(p, n) {
    Pos q = A.g.pos(p);
    D[(size_t)p * n + p] = A.c[p];
    if (q.i > 0) { D[(size_t)p * n + p - SI] = -A.w[p]; D[(size_t)(p - SI) * n + p] = -A.w[p]; }
    if (q.j > 0) { D[(size_t)p * n + p - SJ] = -A.s[p]; D[(size_t)(p - SJ) * n + p] = -A.s[p]; }
    if (q.k > 0) { D[(size_t)p * n + p - 1] = -A.b[p]; D[(size_t)(p - 1) * n + p] = -A.b[p]; }
  }
}

// Largest diagonal entry, for the pivot threshold (one block of 1024).
__global__ void k_dense_dmax(int n, const double *__restrict__ D, double *dmax) {
  double m = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, D[(size_t)i * n + i]);
  for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
  __shared__ double wm[32];
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) m = fmax(m, wm[q]);
    *dmax = fmax(m, wm[0]);
  }
}

constexpr int kGjB = 32;     // pivots per block step
constexpr int kGjRows = 32;  // rows per CTA
constexpr int kGjCols = 128; // columns per CTA at a time, two threads a column
constexpr int kGjGrid = 296; // CTAs at most: one wave, two an SM

// One blocked Gauss-Jordan exchange on the pivots k0 .. k0+kb-1 (out of
// place, A -> B). With A11 the pivot block, G = A11^-1 (by scalar
// Gauss-Jordan in shared memory, every CTA redundantly):
//   B11 = G, B12 = G A12, B21 = -A21 G, B22 = A22 - A21 G A12.
// After the last block B = A^-1. A pivot not above rel_tol * dmax (a
// solid-only aggregate, or the constant mode of an all-Neumann problem)
// is skipped: its row and column become zero, i.e. that unknown is held at
// zero, which gives a generalised inverse of a consistent singular system
// (in a positive semi-definite matrix a zero Schur pivot has a zero row
// and column, so nothing else changes).
// Every CTA forms G, so a small step is bound by it: 32 dependent exchanges,
// each a barrier, a shared load, a division and two multiply-adds. A thread
// holds four entries (row w + 8 u, column lane): the pivot column comes by
// shuffle, the pivot row from shared memory in two buffers by turns, which
// makes one barrier do (8 us a step where two barriers and a round trip of
// every entry through shared memory took 21). The columns of a CTA's 32 rows
// are shared out over CTAs as far as one wave of them goes, and a CTA takes
// the rest 128 at a time; a thread loads eight rows' entries before their
// sums, as the loads' latency bounds large steps. Time per step of 32 pivots:
//   n                                          512   720  1000  1872  4096
//   32 rows x 128 columns a CTA, one a column tile
//                                               31    30    34    73   335 us
//   one wave of CTAs                            24    24    28    43   187 us
//   and G in registers, loads in eights         15    14    18    32   121 us
__global__ void __launch_bounds__(256, 2) k_gj_block(int n, int k0, const double *__restrict__ A,
                                                     double *__restrict__ B, const double *dmax,
                                                     double rel_tol) {
  constexpr int GR = kGjB / 8, AHEAD = 8;
  __shared__ double G[kGjB][kGjB + 1];
  __shared__ __align__(16) double U[kGjRows][kGjB + 2];
  __shared__ __align__(16) double S[kGjRows][kGjB + 2];
  __shared__ double rowb[2][kGjB];
  const int kb = min(kGjB, n - k0);
  const double thr = rel_tol * (*dmax);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i0 = blockIdx.x * kGjRows;
  double g[GR];
#pragma unroll
  for (int u = 0; u < GR; ++u) {
    const int i = w + 8 * u;
    g[u] = i < kb && lane < kb ? A[(size_t)(k0 + i) * n + k0 + lane] : 0.0;
    S[i][lane] = i0 + i < n && lane < kb ? A[(size_t)(i0 + i) * n + k0 + lane] : 0.0;   // the rows' pivot-column entries
  }
  if (w == 0) rowb[0][lane] = g[0];
  __syncthreads();
#pragma unroll
  for (int ku = 0; ku < GR; ++ku)
    for (int kw = 0; kw < 8; ++kw) {
      const int k = 8 * ku + kw;
      if (k >= kb) break;
      const double rk = rowb[k & 1][lane], akk = rowb[k & 1][k];
      const bool sk = !(akk > thr);
      const double piv = sk ? 0.0 : 1.0 / akk;
#pragma unroll
      for (int u = 0; u < GR; ++u) {
        const double c = __shfl_sync(0xffffffffu, g[u], k);
        const bool ik = u == ku && w == kw, jk = lane == k;
        double v;
        if (sk) v = ik || jk ? 0.0 : g[u];
        else if (ik) v = jk ? piv : rk * piv;
        else v = jk ? -c * piv : g[u] - c * rk * piv;
        g[u] = v;
      }
      // the row of pivot k + 1, into the buffer that step k - 1 read
      if (kw < 7) {
        if (w == kw + 1) rowb[(k + 1) & 1][lane] = g[ku];
      } else if (ku + 1 < GR && w == 0) {
        rowb[(k + 1) & 1][lane] = g[ku + 1 < GR ? ku + 1 : 0];
      }
      __syncthreads();
    }
#pragma unroll
  for (int u = 0; u < GR; ++u) G[w + 8 * u][lane] = g[u];
  __syncthreads();
  // U: the row coefficients on the pivot rows
  double acc[GR] = {};
#pragma unroll 4
  for (int m = 0; m < kGjB; m += 2) {
    const double g0 = G[m][lane], g1 = G[m + 1][lane];
#pragma unroll
    for (int u = 0; u < GR; ++u) {
      const double2 sv = *reinterpret_cast<const double2 *>(&S[w + 8 * u][m]);
      acc[u] += sv.x * g0;
      acc[u] += sv.y * g1;
    }
  }
#pragma unroll
  for (int u = 0; u < GR; ++u) {
    const int i = i0 + w + 8 * u;
    U[w + 8 * u][lane] = i >= k0 && i < k0 + kb ? G[i - k0][lane] : acc[u];
  }
  __syncthreads();
  const int half = threadIdx.x / kGjCols * (kGjRows / 2);
  for (int j = blockIdx.y * kGjCols + threadIdx.x % kGjCols; j < n; j += gridDim.y * kGjCols) {
    const bool jin = j >= k0 && j < k0 + kb;
    double a[kGjB];
#pragma unroll
    for (int l = 0; l < kGjB; ++l) a[l] = !jin && l < kb ? A[(size_t)(k0 + l) * n + j] : 0.0;
    for (int r0 = half; r0 < half + kGjRows / 2; r0 += AHEAD) {
      double o[AHEAD];
#pragma unroll
      for (int r = 0; r < AHEAD; ++r) {
        const int i = i0 + r0 + r;
        o[r] = i < n && !jin && !(i >= k0 && i < k0 + kb) ? A[(size_t)i * n + j] : 0.0;
      }
#pragma unroll
      for (int r = 0; r < AHEAD; ++r) {
        const int ii = r0 + r, i = i0 + ii;
        if (i >= n) continue;
        const bool iin = i >= k0 && i < k0 + kb;
        double v;
        if (jin) v = iin ? U[ii][j - k0] : -U[ii][j - k0];
        else {
          double sum = 0.0;
#pragma unroll
          for (int l = 0; l < kGjB; l += 2) {
            const double2 q = *reinterpret_cast<const double2 *>(&U[ii][l]);
            sum += q.x * a[l];
            sum += q.y * a[l + 1];
          }
          v = iin ? sum : o[r] - sum;
        }
        B[(size_t)i * n + j] = v;
      }
    }
  }
}

// Grids whose rows are padded: below kPadMin the passes are bound by their
// chains of loads whatever the rows, and the pad cells would be a larger
// share of the level; above kPadMax the copy of the operator (32 bytes a
// cell) could cost a grid its place in device memory.
constexpr long long kPadMin = 4096, kPadMax = 1ll << 28;
// Cells of the coarsest level at most, unless the caller has chosen: a level
// of 513 to 1024 cells is inverted rather than coarsened once more. It is
// visited 2^(l-1) times an iteration, so the deeper it lies the more the inverse
// saves, while its set-up (15 to 20 us for each 32 cells) is paid once for a
// matrix. Measured against coarsening on, ms of a solve on a known matrix / of a
// step with a new one: level 1 of 720 cells 1.24 -> 0.80 / 0.90 -> 1.10; of 1000
// cells 0.99 -> 0.67 / 0.87 -> 1.25; level 2 of 1000 cells 1.83 -> 1.08 / 1.46 ->
// 1.59; level 3 of 1000 cells 6.0 -> 3.7 / 3.2 -> 2.7; level 4 of 1000 cells 14.1
// -> 10.1 / 8.1 -> 6.4. So levels 0 and 1 end at 768 cells, where a step with a
// new matrix takes no longer than it did with an end at 512 and the cycle's former
// weights.
constexpr int kCoarseAuto = 1024, kCoarseAutoTop = 768;

// Stored cells of a row of n: whole FP32 vectors in both precisions (a
// hierarchy serves mixed and FP64 solves, and an FP64 solve's bits do not
// depend on which came first), where that adds at most a seventh. Measured
// there: 7, 14, 22 and 30 cells a row mixed 2 to 7% faster, FP64 from 1.4%
// slower to even. Above: 10, 13 and 17 cells mixed 2% faster, FP64 3 to 4.5%
// slower; 5 and 6 cells mixed within 3% either way, FP64 12% slower; 2 cells
// (512x512) mixed 2.7 -> 3.1 ms, FP64 2.7 -> 3.7 ms.
constexpr int kRowVec = VecTraits<float>::V;
static int padded_row(int n) {
  const int up = (n + kRowVec - 1) / kRowVec * kRowVec;
  return 7ll * up <= 8ll * n ? up : n;
}

template <typename T>
void EWork<T>::ensure(const std::vector<ELevel> &lv) {
  if (L.size() == lv.size() && x0.n == (size_t)lv[0].ncell()) return;
  drop_graph();
  x0.release();   // the last one allocated: its size says that all are there
  L.clear();
  L.resize(lv.size());
  for (size_t l = 0; l < lv.size(); ++l) {
    size_t n = (size_t)lv[l].ncell();
    Lv &v = L[l];
    v.b.alloc(n); v.x.alloc(n); v.xa.alloc(n); v.xb.alloc(n);
    if (l > 0) { v.z1.alloc(n); v.z2.alloc(n); v.q1.alloc(n); v.r1.alloc(n); v.v.alloc(n); }
  }
  size_t n0 = (size_t)lv[0].ncell();
  r0.alloc(n0); z0.alloc(n0); pA.alloc(n0); pB.alloc(n0); q0.alloc(n0);
  q0b.alloc(n0);
  ks.alloc(lv.size());
  fs.alloc(1);
  PBG_CUDA(cudaMemset(fs.p, 0, sizeof(FcgScal)));
  // the refinement's residual is written to the cells of padded rows only
  PBG_CUDA(cudaMemset(L[0].b.p, 0, L[0].b.bytes()));
  PBG_CUDA(cudaStreamSynchronize(0));
  x0.alloc(n0);
}

template <typename T>
void EWork<T>::drop_graph() {
  if (iter_graph) cudaGraphExecDestroy(iter_graph);
  if (loop_graph) cudaGraphExecDestroy(loop_graph);
  iter_graph = nullptr;
  loop_graph = nullptr;
  iter_nodes = 0;
}

// Programmatic dependent launch measured no gain inside the captured
// iteration (20.0 against 20.2 ms at 256^3), so it is off unless PBG_PDL=1.
bool pdl_enabled() {
  static const bool on = [] {
    const char *e = getenv("PBG_PDL");
    return e && atoi(e) == 1;
  }();
  return on;
}

// End of one FCG iteration in the device-side loop (a conditional WHILE
// node of a CUDA graph): continue while the solve is running, and never
// more than maxit times, whatever the flags say.
__global__ void k_fcg_continue(cudaGraphConditionalHandle h, FcgScal *fs) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int n = ++fs->loops;
  cudaGraphSetConditional(h, (!fs->done && n < fs->maxit) ? 1u : 0u);
}

// Start of the device-side loop: enter it only if the solve has not
// converged at the start (k_fcg_init sets done when |r0| is already below
// the tolerance). With this gate in front of the WHILE node, no kernel of
// the loop body runs once the solve is done, so the body's kernels are
// captured without the done flag and do not load it before their work.
__global__ void k_fcg_gate(cudaGraphConditionalHandle h, const FcgScal *fs) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  cudaGraphSetConditional(h, (!fs->done && fs->loops < fs->maxit) ? 1u : 0u);
}

// The FCG iterations of a refinement sweep run as a device-side loop (a
// conditional WHILE graph node) unless PBG_GRAPH_LOOP=0, which replays the
// one-iteration graph in host-polled chunks instead.
static bool graph_loop_enabled() {
  static const bool on = [] {
    const char *e = getenv("PBG_GRAPH_LOOP");
    return !(e && atoi(e) == 0);
  }();
  return on;
}

// Tuning knobs (environment): PBG_COARSE_MAX sets the size of the dense
// coarsest level, PBG_KC_MAX the deepest level that runs a K-cycle,
// PBG_OMEGA one damped-Jacobi weight for every sweep (0 < omega < 1).
EngineOpts::EngineOpts() {
  const char *c = getenv("PBG_COARSE_MAX");
  if (c && atoi(c) > 0) { coarse_max = atoi(c); coarse_auto = false; }
  const char *k = getenv("PBG_KC_MAX");
  if (k && atoi(k) > 0) kc_max = atoi(k);
  const char *o = getenv("PBG_OMEGA");
  if (o && atof(o) > 0.0 && atof(o) < 1.0) omega_a = omega_b = atof(o);
}

template struct EWork<double>;
template struct EWork<float>;

Engine::~Engine() {
  if (hsc) cudaFreeHost(hsc);
}

template <> EMat<double> Engine::mat<double>(int l) const { return L[l].m64; }
template <> EMat<float> Engine::mat<float>(int l) const { return L[l].m32; }
template <> const void *Engine::ainv<double>() const { return Ainv; }
template <> const void *Engine::ainv<float>() const { return Ainv32; }

// Row-scaled FP16 copy of the dense inverse: row i is stored as a / s_i with
// s_i = max_j |a_ij|, so every entry lies in [-1, 1] (one warp per row).
__global__ void k_to_half_rows(int n, const double *__restrict__ a, __half *__restrict__ o,
                               float *__restrict__ sc) {
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= n) return;
  const double *ar = a + (long long)row * n;
  double m = 0.0;
  for (int c = lane; c < n; c += 32) m = fmax(m, fabs(ar[c]));
  for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
  const double inv = m > 0.0 ? 1.0 / m : 0.0;
  for (int c = lane; c < n; c += 32) o[(long long)row * n + c] = __double2half(ar[c] * inv);
  if (lane == 0) sc[row] = (float)m;
}

// z = Ainv r from the row-scaled FP16 copy: 16-byte loads of eight entries,
// FP32 sums, one warp per row (n a multiple of 8)
__global__ void k_dense_solve_h(int n, const __half *__restrict__ Ah, const float *__restrict__ sc,
                                const float *__restrict__ r, float *__restrict__ z, const int *stop) {
  PBG_PDL_ENTRY();
  if (stop && *stop) return;
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= n) return;
  const uint4 *ar = reinterpret_cast<const uint4 *>(Ah + (long long)row * n);
  float acc = 0.0f;
  for (int c8 = lane; c8 < n / 8; c8 += 32) {
    const uint4 u = ar[c8];
    const __half2 *h = reinterpret_cast<const __half2 *>(&u);
    const float4 r0 = *reinterpret_cast<const float4 *>(r + c8 * 8);
    const float4 r1 = *reinterpret_cast<const float4 *>(r + c8 * 8 + 4);
    const float2 a0 = __half22float2(h[0]), a1 = __half22float2(h[1]);
    const float2 a2 = __half22float2(h[2]), a3 = __half22float2(h[3]);
    acc += a0.x * r0.x + a0.y * r0.y + a1.x * r0.z + a1.y * r0.w;
    acc += a2.x * r1.x + a2.y * r1.y + a3.x * r1.z + a3.y * r1.w;
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  if (lane == 0) z[row] = acc * sc[row];
}

// Large coarsest levels in the mixed path apply the FP16 copy (half the
// bytes of the FP32 one) unless PBG_DENSE_HALF=0.
static bool dense_half_enabled() {
  static const bool on = [] {
    const char *e = getenv("PBG_DENSE_HALF");
    return !(e && atoi(e) == 0);
  }();
  return on;
}
constexpr int kDenseHalfMin = 2048;  // coarsest cells from which the FP16 copy is used

__global__ void k_to_float(long long N, const double *__restrict__ a, float *__restrict__ o) {
  GRID_LOOP(p, N) o[p] = (float)a[p];
}

// z = Ainv r on the coarsest level (the FP32 inverse for T = float)
template <typename T>
void Engine::dense_solve(const T *r, T *z, const int *stop, cudaStream_t s) {
  using AT = typename std::conditional<sizeof(T) == 4, float, double>::type;
  const int blocks = (int)(((long long)ncoarse * 32 + kThreads - 1) / kThreads);
  if constexpr (sizeof(T) == 4) {
    if (Ainv16.n) {
      launch_pdl(k_dense_solve_h, blocks, kThreads, s, ncoarse, (const __half *)Ainv16.p,
                 (const float *)Ainv16s.p, (const float *)r, (float *)z, stop);
      return;
    }
  }
  launch_pdl(k_dense_solve<T, AT>, blocks, kThreads, s, ncoarse, (const AT *)ainv<T>(), r, z, stop);
}

void Engine::build(const EMat<double> &A0_, cudaStream_t s, bool mixed) {
  w64.drop_graph();
  w32.drop_graph();
  w64.L.clear();
  w32.L.clear();
  L.clear();
  A0 = A0_;
  pad = RowPad();
  const bool padded = A0.ncell() >= kPadMin && A0.ncell() <= kPadMax;
  // rows along j only where the 16-byte kernels can run on them
  pad.two_d = padded && A0.nz == 1 && padded_row(A0.ny) % kRowVec == 0;
  pad.F = pad.two_d ? A0.ny : A0.nz;
  pad.FP = padded ? padded_row(pad.F) : pad.F;
  L.emplace_back();
  {
    ELevel &l0 = L[0];
    l0.grid = {A0.nx, A0.ny, A0.nz};
    l0.nx = A0.nx; l0.ny = pad.two_d ? 1 : A0.ny; l0.nz = pad.FP;
    l0.d64.alloc(l0.ncell());
    if (pad.any()) {
      for (DBuf<double> *a : {&pc, &pw, &ps, &pb})
        if (a->n != (size_t)l0.ncell()) a->alloc(l0.ncell());
      l0.m64 = make_emat<double>(l0.nx, l0.ny, l0.nz, pc.p, pw.p, ps.p, pb.p, l0.d64.p);
    } else {
      for (DBuf<double> *a : {&pc, &pw, &ps, &pb}) a->release();
      l0.m64 = make_emat<double>(A0.nx, A0.ny, A0.nz, A0.c, A0.w, A0.s, A0.b, l0.d64.p);
    }
  }
  auto dense = [this] {
    if (!opt.coarse_auto) return (long long)opt.coarse_max;
    return (long long)std::max(opt.coarse_max, L.size() <= 2 ? kCoarseAutoTop : kCoarseAuto);
  };
  // Cells of the grid count, not pad cells: padding adds no level.
  auto half = [](int n) { return (n + 1) / 2; };
  while (L.back().grid.ncell() > dense()) {
    const ELevel &f = L.back();
    ELevel c;
    c.grid = {half(f.grid.nx), half(f.grid.ny), half(f.grid.nz)};
    c.nx = half(f.nx);
    c.ny = half(f.ny);
    c.nz = half(f.nz);
    if (padded && c.ncell() >= kPadMin) c.nz = padded_row(c.nz);   // rows of whole vectors here too
    long long n = c.ncell();
    c.c64.alloc(n); c.w64.alloc(n); c.s64.alloc(n); c.b64.alloc(n); c.d64.alloc(n);
    c.m64 = make_emat<double>(c.nx, c.ny, c.nz, c.c64.p, c.w64.p, c.s64.p, c.b64.p, c.d64.p);
    L.push_back(std::move(c));
  }
  ncoarse = (int)L.back().ncell();
  // one allocation for the inverse and what it is formed in: each of a
  // megabyte or more costs about 0.4 ms of a first solve
  const size_t nn = (size_t)ncoarse * ncoarse;
  dense_mem.fit(2 * nn + (mixed ? (nn + 1) / 2 : 0));
  Ainv = dense_mem.p;
  Dtmp = Ainv + nn;
  Ainv32 = mixed ? reinterpret_cast<float *>(Dtmp + nn) : nullptr;
  Ainv16.release();
  Ainv16s.release();
  if (mixed && dense_half_enabled() && ncoarse >= kDenseHalfMin && ncoarse % 8 == 0) {
    Ainv16.alloc((size_t)ncoarse * ncoarse);
    Ainv16s.alloc((size_t)ncoarse);
  }
  have32 = false;
  if (mixed) {
    for (auto &lv : L) {
      long long m = lv.ncell();
      lv.c32.alloc(m); lv.w32.alloc(m); lv.s32.alloc(m); lv.b32.alloc(m); lv.d32.alloc(m);
      lv.m32 = make_emat<float>(lv.nx, lv.ny, lv.nz, lv.c32.p, lv.w32.p, lv.s32.p, lv.b32.p, lv.d32.p);
    }
    have32 = true;
  }
  if (!hsc) PBG_CUDA(cudaMallocHost((void **)&hsc, 64 * sizeof(double)));
  if (dsc.n < 8) dsc.alloc(8);
  compute(s);
  PBG_CUDA(cudaStreamSynchronize(s));
}

// Numeric set-up on the allocated hierarchy, all on the device: inverse
// diagonals, Galerkin coarse operators, FP32 copies and the dense inverse of
// the coarsest level. Used by build() and again after the fine matrix
// changed in place: buffers, and so the captured iteration graphs, stay
// valid. Enqueued on s, no host synchronisation.
void Engine::compute(cudaStream_t s) {
  auto out = [&](ELevel &lv) {
    LevelOut o{const_cast<double *>(lv.m64.c),
               const_cast<double *>(lv.m64.w), const_cast<double *>(lv.m64.s),
               const_cast<double *>(lv.m64.b), lv.d64.p,
               nullptr, nullptr, nullptr, nullptr, nullptr};
    if (have32) { o.c32 = lv.c32.p; o.w32 = lv.w32.p; o.s32 = lv.s32.p; o.b32 = lv.b32.p; o.d32 = lv.d32.p; }
    return o;
  };
  if (pad.any()) {
    const uint32_t rows = (uint32_t)(L[0].ncell() / pad.FP);
    k_pad_matrix<<<grid_for(L[0].ncell()), kThreads, 0, s>>>(A0, pad, rows, FastDiv((uint32_t)pad.FP), pc.p, pw.p,
                                                             ps.p, pb.p); note_launch();
  }
  k_level_finish<<<grid_for(L[0].ncell()), kThreads, 0, s>>>(L[0].m64, out(L[0])); note_launch();
  for (size_t l = 1; l < L.size(); ++l) {
    ELevel &c = L[l];
    k_galerkin<<<grid_for(c.ncell()), kThreads, 0, s>>>(L[l - 1].m64, Geo(c.nx, c.ny, c.nz), out(c));
    k_level_finish<<<grid_for(c.ncell()), kThreads, 0, s>>>(c.m64, out(c));
    note_launch(); note_launch();
  }
  // dense inverse of the coarsest operator: blocked Gauss-Jordan, out of place
  const int n = ncoarse;
  const size_t nn = (size_t)n * n;
  double *src = Dtmp, *dst = Ainv;
  if ((n + kGjB - 1) / kGjB % 2 == 0) std::swap(src, dst);   // the last step writes Ainv
  PBG_CUDA(cudaMemsetAsync(src, 0, nn * sizeof(double), s));
  k_dense_fill<<<grid_for(n), kThreads, 0, s>>>(L.back().m64, src); note_launch();
  k_dense_dmax<<<1, 1024, 0, s>>>(n, src, dsc.p + 7); note_launch();
  const int gjr = (n + kGjRows - 1) / kGjRows, gjc = (n + kGjCols - 1) / kGjCols;
  const dim3 tiles(gjr, std::min(gjc, std::max(1, kGjGrid / gjr)));
  for (int k0 = 0; k0 < n; k0 += kGjB) {
    k_gj_block<<<tiles, 256, 0, s>>>(n, k0, src, dst, dsc.p + 7, 1e-10); note_launch();
    std::swap(src, dst);
  }
  if (have32) {
    k_to_float<<<grid_for((long long)nn), kThreads, 0, s>>>((long long)nn, Ainv, Ainv32); note_launch();
    if (Ainv16.n) {
      const int blocks = (int)(((long long)ncoarse * 32 + kThreads - 1) / kThreads);
      k_to_half_rows<<<blocks, kThreads, 0, s>>>(ncoarse, Ainv, Ainv16.p, Ainv16s.p); note_launch();
    }
  }
  PBG_CUDA(cudaGetLastError());
}

// Numeric refresh for a changed fine matrix of the same shape at the same
// addresses; false if the hierarchy has to be built anew.
bool Engine::refresh(const EMat<double> &A, bool mixed, cudaStream_t s) {
  if (L.empty() || (mixed && !have32) || A0.nx != A.nx || A0.ny != A.ny || A0.nz != A.nz ||
      A0.c != A.c || A0.w != A.w || A0.s != A.s || A0.b != A.b)
    return false;
  compute(s);
  return true;
}

// Preconditioner M r -> z on level l. kc: the K-cycle's second application,
// whose right-hand side r1 = b - a1 q1 is formed (and stored) by k_jac2.
template <typename T>
void Engine::precond(int l, const T *r, T *z, bool dots, const T *u, double *out2, EWork<T> &w,
                     RedPool &red, const int *stop, cudaStream_t s, bool kc) {
  const int last = (int)L.size() - 1;
  const CycleW<T> om{(T)opt.omega_a, (T)opt.omega_b, (T)opt.over};
  auto &v = w.L[l];
  if (l == last) {
    dense_solve<T>(r, z, stop, s);
    if (dots) {  // a level-0 problem small enough to be the coarsest
      EMat<T> A = mat<T>(l);
      PBG_CUDA(cudaMemcpyAsync(v.xa.p, z, sizeof(T) * A.ncell(), cudaMemcpyDeviceToDevice, s));
      // omega = 0 keeps z and computes the dot products
      launch_pdl(k_jac_dots<T>, grid_for(A.ncell()), kThreads, s, A, r, (const T *)v.xa.p, z, T(0), u, out2,
                 red.slot_part(0), red.slot_count(0), stop);
    }
    return;
  }
  EMat<T> A = mat<T>(l);
  const int g = grid_for(A.ncell());
  const ELevel &H = L[l + 1];
  auto &vh = w.L[l + 1];
  const T *rr = kc ? v.r1.p : r;
  const bool vec = A.nz % VecTraits<T>::V == 0;
  const int gv = grid_for(A.ncell() / VecTraits<T>::V, kThreads, kVecBlocks);
  const KScal *ksl = kc ? w.ks.p + l : nullptr;
  const int gw = grid_for(A.ncell() / VecTraits<T>::V, kThreads, kVecWideBlocks<T>);
  launch_pdl(vec ? kv_jac2<T> : k_jac2<T>, vec ? gw : g, kThreads, s, A, r, (const T *)v.b.p,
             (const T *)v.q1.p, ksl, v.r1.p, v.xb.p, om, stop);
  const long long rthreads = H.ncell() >= kRestrictSerialMin ? H.ncell() : H.ncell() * 8;
  launch_pdl(k_resid_restrict<T>, grid_for(rthreads), kThreads, s, A, rr, (const T *)v.xb.p,
             Geo(H.nx, H.ny, H.nz), vh.b.p, stop);
  const T *eH, *z2H = nullptr;
  const KScal *ksH = nullptr;
  if (l + 1 == last) {
    dense_solve<T>(vh.b.p, vh.x.p, stop, s);
    eH = vh.x.p;
  } else {
    if (l + 1 <= opt.kc_max) {
      kcycle<T>(l + 1, w, red, stop, s);
      eH = vh.z1.p; z2H = vh.z2.p; ksH = w.ks.p + l + 1;
    } else {  // one visit: e = M b on level l+1
      precond<T>(l + 1, vh.b.p, vh.z1.p, false, nullptr, nullptr, w, red, stop, s, false);
      eH = vh.z1.p;
    }
  }
  launch_pdl(vec ? kv_prolong_jac<T> : k_prolong_jac<T>, vec ? gv : g, kThreads, s, A, rr,
             (const T *)v.xb.p, H.ny, H.nz, eH, z2H, ksH, v.xa.p, om, stop);
  if (dots && vec && l == 0) {
    // u is the q of the previous FCG iteration, picked by parity on the device
    launch_pdl(kv_jac<T, true>, gv, kThreads, s, A, rr, (const T *)v.xa.p, z, om.a, (const T *)w.q0.p,
               (const T *)w.q0b.p, (const FcgScal *)w.fs.p, out2, red.slot_part(0), red.slot_count(0), stop);
  } else if (dots) {
    launch_pdl(k_jac_dots<T>, g, kThreads, s, A, rr, (const T *)v.xa.p, z, om.a, u, out2, red.slot_part(0),
               red.slot_count(0), stop);
  } else if (vec) {
    launch_pdl(kv_jac<T, false>, gv, kThreads, s, A, rr, (const T *)v.xa.p, z, om.a, (const T *)nullptr,
               (const T *)nullptr, (const FcgScal *)nullptr, (double *)nullptr, (double *)nullptr,
               (unsigned *)nullptr, stop);
  } else {
    launch_pdl(k_jac<T>, g, kThreads, s, A, rr, (const T *)v.xa.p, z, om.a, stop);
  }
}

template <typename T>
void Engine::kcycle(int l, EWork<T> &w, RedPool &red, const int *stop, cudaStream_t s) {
  EMat<T> A = mat<T>(l);
  const int g = grid_for(A.ncell());
  auto &v = w.L[l];
  KScal *ks = w.ks.p + l;
  precond<T>(l, v.b.p, v.z1.p, false, nullptr, nullptr, w, red, stop, s, false);
  launch_pdl(k_kc_q1<T>, g, kThreads, s, A, (const T *)v.z1.p, (const T *)v.b.p, v.q1.p, ks,
             red.slot_part(0), red.slot_count(0), stop);
  precond<T>(l, nullptr, v.z2.p, false, nullptr, nullptr, w, red, stop, s, true);
  launch_pdl(k_kc_q2<T>, g, kThreads, s, A, (const T *)v.z2.p, (const T *)v.q1.p, (const T *)v.r1.p, v.v.p,
             ks, red.slot_part(0), red.slot_count(0), stop);
}

// Flexible CG on level 0 for A e = b (e starts at zero); returns iterations.
// One iteration (the preconditioner's K-cycle over all levels plus the two
// FCG kernels) is captured once into a CUDA graph and replayed; every kernel
// in it returns at once when the device-side done flag is set.
template <typename T>
int Engine::fcg(EWork<T> &w, const T *b, double tol, int maxit, RedPool &red, cudaStream_t s,
                double *hist, FcgScal *hfs) {
  EMat<T> A = mat<T>(0);
  const long long N = A.ncell();
  const int g = grid_for(N);
  FcgScal *fs = w.fs.p;
  // one FCG iteration: the preconditioner's K-cycle over all levels plus
  // the two FCG kernels; every kernel returns at once when *stop is set
  // (stop == nullptr: no check)
  auto iteration = [&](const int *stop) {
    precond<T>(0, w.r0.p, w.z0.p, true, w.q0.p, &fs->zr, w, red, stop, s, false);
    if (A.nz % VecTraits<T>::V == 0 && (int)L.size() > 1) {
      const int gv = grid_for(N / VecTraits<T>::V, kThreads, kVecBlocks);
      const int gw = grid_for(N / VecTraits<T>::V, kThreads, kVecWideBlocks<T>);
      launch_pdl(kv_fcg_pq<T>, gw, kThreads, s, A, (const T *)w.z0.p, w.pA.p, w.pB.p, w.q0.p, w.q0b.p, fs,
                 red.slot_part(0), red.slot_count(0));
      launch_pdl(kv_fcg_xr<T>, gv, kThreads, s, N, w.x0.p, w.r0.p, (const T *)w.pA.p, (const T *)w.pB.p,
                 (const T *)w.q0.p, (const T *)w.q0b.p, fs, red.slot_part(0), red.slot_count(0));
    } else {
      launch_pdl(k_fcg_pq<T>, g, kThreads, s, A, (const T *)w.z0.p, w.pA.p, w.pB.p, w.q0.p, fs,
                 red.slot_part(0), red.slot_count(0));
      launch_pdl(k_fcg_xr<T>, g, kThreads, s, N, w.x0.p, w.r0.p, (const T *)w.pA.p, (const T *)w.pB.p,
                 (const T *)w.q0.p, fs, red.slot_part(0), red.slot_count(0));
    }
  };
  // captured once: the loop where it is used, else the iteration alone
  if (!w.iter_graph && !w.loop_graph) {
    const unsigned long long before = g_launch_count;
    auto counted = [&] {
      w.iter_nodes = (size_t)(g_launch_count - before);
      __atomic_sub_fetch(&g_launch_count, (unsigned long long)w.iter_nodes, __ATOMIC_RELAXED);
    };
    if (!graph_loop_enabled()) {
      cudaGraph_t graph = nullptr;
      PBG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
      try {
        iteration(&fs->done);
      } catch (...) {
        cudaStreamEndCapture(s, &graph);  // leave the stream usable
        if (graph) cudaGraphDestroy(graph);
        throw;
      }
      PBG_CUDA(cudaStreamEndCapture(s, &graph));
      counted();
      PBG_CUDA(cudaGraphInstantiate(&w.iter_graph, graph, 0));
      cudaGraphDestroy(graph);
    } else {
      // the same iteration as the body of a WHILE node: a gate kernel sets
      // its condition before the first pass, the last kernel of the body
      // after each pass
      cudaGraph_t lg = nullptr;
      PBG_CUDA(cudaGraphCreate(&lg, 0));
      try {
        cudaGraphConditionalHandle h;
        PBG_CUDA(cudaGraphConditionalHandleCreate(&h, lg, 0, cudaGraphCondAssignDefault));
        cudaKernelNodeParams kp = {};
        const FcgScal *cfs = fs;
        void *kargs[] = {(void *)&h, (void *)&cfs};
        kp.func = (void *)k_fcg_gate;
        kp.gridDim = dim3(1);
        kp.blockDim = dim3(32);
        kp.sharedMemBytes = 0;
        kp.kernelParams = kargs;
        kp.extra = nullptr;
        cudaGraphNode_t gate;
        PBG_CUDA(cudaGraphAddKernelNode(&gate, lg, nullptr, 0, &kp));
        cudaGraphNodeParams np = {};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = h;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        cudaGraphNode_t node;
        PBG_CUDA(cudaGraphAddNode(&node, lg, &gate, 1, &np));
        cudaGraph_t body = np.conditional.phGraph_out[0];
        PBG_CUDA(cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        try {
          iteration(nullptr);
          k_fcg_continue<<<1, 32, 0, s>>>(h, fs);
        } catch (...) {
          cudaStreamEndCapture(s, &body);
          throw;
        }
        PBG_CUDA(cudaStreamEndCapture(s, &body));
        counted();
        PBG_CUDA(cudaGraphInstantiate(&w.loop_graph, lg, 0));
      } catch (...) {
        cudaGraphDestroy(lg);
        throw;
      }
      cudaGraphDestroy(lg);
    }
  }
  PBG_CUDA(cudaMemsetAsync(w.q0.p, 0, sizeof(T) * N, s));
  PBG_CUDA(cudaMemsetAsync(w.q0b.p, 0, sizeof(T) * N, s));
  k_fcg_init<T><<<g, kThreads, 0, s>>>(N, b, w.x0.p, w.r0.p, fs, tol, maxit, hist,
                                       red.slot_part(0), red.slot_count(0)); note_launch();
  PBG_CUDA(cudaGetLastError());
  if (w.loop_graph) {
    PBG_CUDA(cudaGraphLaunch(w.loop_graph, s));
    PBG_CUDA(cudaMemcpyAsync(hfs, fs, sizeof(FcgScal), cudaMemcpyDeviceToHost, s));
    PBG_CUDA(cudaStreamSynchronize(s));
    __atomic_add_fetch(&g_launch_count, (unsigned long long)hfs->loops * (w.iter_nodes + 1) + 1, __ATOMIC_RELAXED);
    return hfs->iter;
  }
  int enq = 0, chunk = 4;
  for (;;) {
    PBG_CUDA(cudaMemcpyAsync(hfs, fs, sizeof(FcgScal), cudaMemcpyDeviceToHost, s));
    PBG_CUDA(cudaStreamSynchronize(s));
    if (hfs->done || enq >= maxit) break;
    int cnt = chunk;
    if (enq + cnt > maxit) cnt = maxit - enq;
    for (int c = 0; c < cnt; ++c) PBG_CUDA(cudaGraphLaunch(w.iter_graph, s));
    __atomic_add_fetch(&g_launch_count, (unsigned long long)(cnt * w.iter_nodes), __ATOMIC_RELAXED);
    enq += cnt;
    if (chunk < 16) chunk *= 2;
  }
  return hfs->iter;
}

// Symmetric approximation of a seven-array operator in the engine's
// storage: each coupling the mean of the two cells' own values (w of a cell
// and e of its west neighbour, and so on), c unchanged; a coupling that only
// one side keeps drops out. That one-sided case is a cell inside a body
// (c = 1e-12 c0, its couplings zeroed) next to a fluid cell off the cut
// list: half the coupling against that tiny diagonal would make the
// approximation indefinite, while in the matrix itself the inside cell's
// value is decoupled. On the reference's cut sphere the refinement around
// it reduces the residual by 1e-2 to 3e-2 per sweep past the first; the
// smaller of the two sides instead (always diagonally dominant) gave 2e-2
// to 4e-2 there but lost the upwind part of a convected matrix, where the
// mean keeps it as a skew term.
__device__ __forceinline__ double sym_coupling(double x, double y) {
  return (x != 0.0 && y != 0.0) ? 0.5 * (x + y) : 0.0;
}

__global__ void k_symmetrize(MatView<double> A, Geo G, double *__restrict__ C, double *__restrict__ W,
                             double *__restrict__ S, double *__restrict__ B) {
  const uint32_t SI = G.nynz, SJ = (uint32_t)A.nz;
  GRID_LOOP(p, G.n) {
    const Pos q = G.pos(p);
    const Nb<double> a = coeffs(A, p, q);
    C[p] = A.c[p];
    W[p] = q.i > 0 ? sym_coupling(a.w, A.e[p - SI]) : 0.0;
    S[p] = q.j > 0 ? sym_coupling(a.s, A.n[p - SJ]) : 0.0;
    B[p] = q.k > 0 ? sym_coupling(a.b, A.t[p - 1]) : 0.0;
  }
}

void symmetrize(const MatView<double> &A, double *c, double *w, double *s, double *b, cudaStream_t st) {
  k_symmetrize<<<grid_for(A.ncell()), kThreads, 0, st>>>(A, Geo(A.nx, A.ny, A.nz), c, w, s, b);
  note_launch();
  PBG_CUDA(cudaGetLastError());
}

// r = b - A x with the operator the solve is for (the symmetric level 0,
// or the seven-array one whose symmetric part the hierarchy holds), its
// rounding into rT, and |r|^2, |b|^2 into dsc[0..1].
template <typename T>
void Engine::true_resid(const double *x, const double *b, T *rT, RedPool &red, cudaStream_t s) {
  const EMat<double> A = A0;
  const int g = grid_for(A.ncell());
  if (nonsym)
    k_true_resid_ns<T><<<g, kThreads, 0, s>>>(top, A.g, x, b, rT, pad, dsc.p, red.slot_part(0),
                                              red.slot_count(0));
  else
    k_true_resid<T><<<g, kThreads, 0, s>>>(A, x, b, rT, pad, dsc.p, red.slot_part(0), red.slot_count(0));
  note_launch();
}

// A non-symmetric operator is solved by refinement around its symmetric
// part, which converges only while the asymmetry is mild (a cut body's face
// fractions); with a strong one (convection) a sweep can raise the
// residual. The iterate before each correction is kept, and a sweep that
// does not reduce the residual is undone and ends the solve (ST_DIVERGED).
void Engine::keep_iterate(const double *x, long long N, cudaStream_t s) {
  if (!nonsym) return;
  if (xtmp.n < (size_t)N) xtmp.alloc(N);
  PBG_CUDA(cudaMemcpyAsync(xtmp.p, x, N * sizeof(double), cudaMemcpyDeviceToDevice, s));
}

void Engine::restore_iterate(double *x, long long N, cudaStream_t s) {
  PBG_CUDA(cudaMemcpyAsync(x, xtmp.p, N * sizeof(double), cudaMemcpyDeviceToDevice, s));
  PBG_CUDA(cudaStreamSynchronize(s));
}

EngineResult Engine::solve_fp64(double *x, const double *b, double tol, int maxit, RedPool &red,
                                cudaStream_t s, double *hist) {
  w64.ensure(L);
  const EMat<double> A = A0;
  const long long N = A.ncell();
  const int g = grid_for(N);
  FcgScal *hfs = (FcgScal *)hsc;
  double *rhs = w64.L[0].b.p;
  EngineResult res{ST_RUNNING, 0, 0, 0, 0.0};
  true_resid<double>(x, b, rhs, red, s);
  PBG_CUDA(cudaMemcpyAsync(hsc + 32, dsc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
  PBG_CUDA(cudaStreamSynchronize(s));
  double rr = hsc[32], bb = hsc[33];
  if (!(bb > 0.0)) { res.status = ST_INITIAL; res.converged = 1; return res; }
  double rel = std::sqrt(rr / bb);
  // a non-symmetric operator converges by the refinement around its
  // symmetric part: more sweeps
  const int sweeps = nonsym ? 16 : 4;
  for (int sweep = 0; sweep < sweeps && rel > tol; ++sweep) {
    double itol = std::fmin(0.9 * tol / rel, 0.5);
    int its = fcg<double>(w64, rhs, itol, maxit - res.iterations, red, s, hist, hfs);
    res.iterations += its;
    res.sweeps++;
    keep_iterate(x, N, s);
    k_add_corr<double><<<g, kThreads, 0, s>>>(A.g, x, w64.x0.p, pad); note_launch();
    true_resid<double>(x, b, rhs, red, s);
    PBG_CUDA(cudaMemcpyAsync(hsc + 32, dsc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
    PBG_CUDA(cudaStreamSynchronize(s));
    const double nrel = std::sqrt(hsc[32] / bb);
    if (nonsym && !(nrel < rel)) { restore_iterate(x, N, s); res.status = ST_DIVERGED; break; }
    rel = nrel;
    if (hfs->status == ST_NAN || hfs->status == ST_BREAKDOWN) { res.status = hfs->status; break; }
    if (res.iterations >= maxit) break;
  }
  res.relres = rel;
  if (rel <= tol) { res.converged = 1; res.status = ST_CONVERGED; }
  else if (res.status == ST_RUNNING) res.status = (rel == rel) ? ST_MAXITER : ST_NAN;
  return res;
}

EngineResult Engine::solve_mixed(double *x, const double *b, double tol, double inner_tol,
                                 int max_sweeps, int inner_maxit, RedPool &red, cudaStream_t s,
                                 double *hist) {
  w32.ensure(L);
  const EMat<double> A = A0;
  const long long N = A.ncell();
  const int g = grid_for(N);
  FcgScal *hfs = (FcgScal *)hsc;
  float *rhs = w32.L[0].b.p;
  EngineResult res{ST_RUNNING, 0, 0, 0, 0.0};
  true_resid<float>(x, b, rhs, red, s);
  PBG_CUDA(cudaMemcpyAsync(hsc + 32, dsc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
  PBG_CUDA(cudaStreamSynchronize(s));
  double rr = hsc[32], bb = hsc[33];
  if (!(bb > 0.0)) { res.status = ST_INITIAL; res.converged = 1; return res; }
  double rel = std::sqrt(rr / bb);
  for (int sweep = 0; sweep < max_sweeps && rel > tol; ++sweep) {
    // solve no further than the outer target needs in the last sweep
    double itol = std::fmax(inner_tol, 0.9 * tol / rel);
    // history slots this sweep may fill: it < kHistMax in k_fcg_xr, so the
    // offset pointer is passed only while offset + kHistMax stays in bounds
    double *h = (hist && res.iterations == 0) ? hist : nullptr;
    int its = fcg<float>(w32, rhs, itol, inner_maxit, red, s, h, hfs);
    res.iterations += its;
    res.sweeps++;
    keep_iterate(x, N, s);
    k_add_corr<float><<<g, kThreads, 0, s>>>(A.g, x, w32.x0.p, pad); note_launch();
    true_resid<float>(x, b, rhs, red, s);
    PBG_CUDA(cudaMemcpyAsync(hsc + 32, dsc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
    PBG_CUDA(cudaStreamSynchronize(s));
    double nrel = std::sqrt(hsc[32] / bb);
    if (nonsym && !(nrel < rel)) { restore_iterate(x, N, s); res.status = ST_DIVERGED; break; }
    if (!(nrel == nrel)) { rel = nrel; res.status = ST_NAN; break; }
    if (hfs->status == ST_BREAKDOWN && nrel >= rel) { rel = nrel; res.status = ST_BREAKDOWN; break; }
    rel = nrel;
  }
  res.relres = rel;
  if (rel <= tol) { res.converged = 1; res.status = ST_CONVERGED; }
  else if (res.status == ST_RUNNING) res.status = ST_MAXITER;
  return res;
}

// Times the fine-level smoothing sweep the solver launches: the vectorised
// kv_jac when the rows allow it, else the scalar k_jac.
template <typename T>
static double time_sweeps(const EMat<T> &A, const T *r, T *xa, T *xb, T om, int reps, cudaStream_t s) {
  cudaEvent_t e0, e1;
  PBG_CUDA(cudaEventCreate(&e0));
  PBG_CUDA(cudaEventCreate(&e1));
  const bool vec = A.nz % VecTraits<T>::V == 0;
  const int g = grid_for(A.ncell());
  const int gv = grid_for(A.ncell() / VecTraits<T>::V, kThreads, kVecBlocks);
  auto sweep = [&](const T *xi, T *xo) {
    if (vec)
      kv_jac<T, false><<<gv, kThreads, 0, s>>>(A, r, xi, xo, om, nullptr, nullptr, nullptr, nullptr,
                                               nullptr, nullptr, nullptr);
    else
      k_jac<T><<<g, kThreads, 0, s>>>(A, r, xi, xo, om, nullptr);
    note_launch();
  };
  sweep(xa, xb);
  PBG_CUDA(cudaEventRecord(e0, s));
  for (int q = 0; q < reps; ++q) sweep((q & 1) ? xb : xa, (q & 1) ? xa : xb);
  PBG_CUDA(cudaEventRecord(e1, s));
  PBG_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  PBG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return (double)ms / reps;
}

double Engine::bench_sweep(int precision, int reps, cudaStream_t s) {
  if (precision == 0) {
    w64.ensure(L);
    PBG_CUDA(cudaMemsetAsync(w64.r0.p, 0, sizeof(double) * L[0].ncell(), s));
    PBG_CUDA(cudaMemsetAsync(w64.L[0].xa.p, 0, sizeof(double) * L[0].ncell(), s));
    return time_sweeps<double>(L[0].m64, w64.r0.p, w64.L[0].xa.p, w64.L[0].xb.p, 0.8, reps, s);
  }
  w32.ensure(L);
  PBG_CUDA(cudaMemsetAsync(w32.r0.p, 0, sizeof(float) * L[0].ncell(), s));
  PBG_CUDA(cudaMemsetAsync(w32.L[0].xa.p, 0, sizeof(float) * L[0].ncell(), s));
  return time_sweeps<float>(L[0].m32, w32.r0.p, w32.L[0].xa.p, w32.L[0].xb.p, 0.8f, reps, s);
}

}  // namespace pbg
