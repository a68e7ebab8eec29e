// Kernels of the lexicographic sweeps (schedule and storage: pbg_sweeps.cuh).
#pragma once

#include "pbg_sweeps.cuh"

namespace pbg {

// a / c with c's stored reciprocal y: KnownDiv with its range checks on the
// exponents, beside the dependent operations instead of before them. A zero
// dividend comes out right for +0 only; everything else outside the range,
// and a NaN y, takes the division itself.
__device__ __forceinline__ double sweep_div(double a, double c, double y) {
  const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
  const unsigned ey = ((unsigned)__double2hiint(y) >> 20) & 0x7ffu;
  const bool in = ea - (1023u - 899u) < 1799u || __double_as_longlong(a) == 0;   // 2^-899 <= |a| < 2^900
  const double q0 = __dmul_rn(a, y);
  double q = __fma_rn(__fma_rn(-q0, c, a), y, q0);
  if (!in || ey == 0x7ffu) q = __ddiv_rn(a, c);
  return q;
}

__device__ __forceinline__ double msub(double s, double a, double b) { return __dsub_rn(s, __dmul_rn(a, b)); }

// The tile of this block, taken by ticket; row-major order is a topological
// order of the tiles' dependences (the tiles before it along i and along j).
__device__ __forceinline__ int sweep_ticket(const SweepSync &y) {
  __shared__ int tile;
  if (threadIdx.x == 0) tile = (int)atomicAdd(&y.ticket[0], 1u);
  __syncthreads();
  return tile;
}
__device__ __forceinline__ void sweep_finish(const SweepSync &y, int tiles) {
  if (threadIdx.x != 0) return;
  if (atomicAdd(&y.ticket[1], 1u) == (unsigned)tiles - 1) { y.ticket[0] = 0; y.ticket[1] = 0; }
}

// Waits until word p carries this launch's epoch and returns it. A poll that
// runs out (or one that did elsewhere) sets *stuck and gives up with zero, so
// that every block ends; the host reports the failure.
__device__ __noinline__ TagWord sweep_poll(const TagWord *p, const SweepSync &y, bool &dead) {
  TagWord a = {0ull, 0ull};
  for (int m = 1; !dead; ++m) {
    a = word_ld(p);
    if (a.tag == y.epoch) break;
    if (m >= kSweepPoll) { atomicExch(y.stuck, 1); dead = true; }
    else if ((m & 1023) == 0 && *(volatile int *)y.stuck) dead = true;
    a.v = 0ull;
  }
  return a;
}

// 8 bytes to shared memory, completion by groups: the loads of later steps
// stay in flight while an earlier step's are waited for
__device__ __forceinline__ void sweep_copy(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
               :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Position of a column in the march. In a backward sweep i, j and k run
// down: li, lj, kk and the tile indices count in march direction.
template <bool BWD>
struct SweepPos {
  int I, J, li, lj, i, j;
  bool col, hasW, hasS;   // the column, and those before it along i and along j, exist
  __device__ __forceinline__ SweepPos(const SweepGeo &g, int tile, int li_, int lj_) : li(li_), lj(lj_) {
    I = tile / g.tj; J = tile - I * g.tj;
    const int mi = I * kSweepTile + li, mj = J * kSweepTile + lj;
    i = BWD ? g.ti * kSweepTile - 1 - mi : mi;
    j = BWD ? g.tj * kSweepTile - 1 - mj : mj;
    col = i < g.nx && j < g.ny;
    hasW = col && (BWD ? i + 1 < g.nx : i > 0);
    hasS = col && (BWD ? j + 1 < g.ny : j > 0);
  }
  __device__ __forceinline__ int at(const SweepGeo &g, int kk) const { return BWD ? g.nz - 1 - kk : kk; }
};

// The march of one tile. Warps 0 and 1 hold a column a thread and do nothing
// but the dependent arithmetic of a step (Body::step). Warp 2 brings the
// columns beside the tile from the exchange into the halo of the shared
// ring, a block of kSweepAhead steps before they are read; warp 3 publishes
// the tile's last columns, one step after they are formed; warps 4 and 5
// copy the operands of later steps to shared memory (asynchronously: loads
// into registers would wait for each other, a warp has few load counters)
// and store the results one step after they are formed. NV values a cell
// travel; a column beside a cell is read at the cell's kk + LOOK.
template <int NV, int A, int LOOK, bool BWD, class Body, class... Arg>
__device__ __forceinline__ void sweep_march(const SweepGeo &g, const SweepSync &y, const Arg &...arg) {
  constexpr int P = kSweepAhead, E = kSweepTile + 1, SLOT = NV * E * E, NP = Body::planes;
  __shared__ double ring[2 * P][SLOT];   // values formed at a step; halo: values read at the next
  __shared__ double stage[P][NP][kSweepCols];
  const int tile = sweep_ticket(y);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nz = g.nz;
  const int T = (nz + 2 * A * (kSweepTile - 1) + LOOK + P - 1) / P * P;
  // every step: all but warp 2; a block of steps: warp 2 and the arithmetic warps
  auto step_barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(kSweepThreads - 32) : "memory"); };
  auto block_barrier = [] { asm volatile("bar.sync 2, %0;" ::"n"(kSweepCols + 32) : "memory"); };
  // lanes 0-7 of warps 2 and 3: the columns along i's edge, 8-15: along j's
  const bool along_i = lane < kSweepTile, used = lane < 2 * kSweepTile;
  const int m = lane % kSweepTile, last = kSweepTile - 1;
  if (warp == 2) {
    const SweepPos<BWD> q(g, tile, along_i ? 0 : m, along_i ? m : 0);
    const bool on = used && (along_i ? q.hasW : q.hasS);
    const TagWord *p = along_i ? y.words + ((size_t)(q.I - 1) * g.ny + q.j) * nz
                                 : y.words + g.words_i() + ((size_t)(q.J - 1) * g.nx + q.i) * nz;
    const int at = along_i ? m + 1 : (m + 1) * E;
    int ke = -A * m;   // the beside column's k of the block's first read
    bool dead = false;
    for (int t0 = 0; t0 < T; t0 += P, ke += P) {
      // halo for the reads of steps t0 .. t0 + P - 1, in the slots before them
      const int slot0 = (t0 + 2 * P - 1) % (2 * P);
      TagWord w[P][NV];
      auto fetch = [&] {
        bool ok = true;
#pragma unroll
        for (int u = 0; u < P; ++u)
#pragma unroll
          for (int v = 0; v < NV; ++v)
            if (on && (unsigned)(ke + u) < (unsigned)nz) w[u][v] = word_ld(p + ke + u + v * g.words());
#pragma unroll
        for (int u = 0; u < P; ++u)
#pragma unroll
          for (int v = 0; v < NV; ++v)
            if (on && (unsigned)(ke + u) < (unsigned)nz && w[u][v].tag != y.epoch) ok = false;
        return ok;
      };
      if (!fetch()) {   // caught up with the neighbour: wait for the block's last word first
        sweep_poll(p + min(ke + P, nz) - 1 + (NV - 1) * g.words(), y, dead);
        fetch();
      }
#pragma unroll
      for (int u = 0; u < P; ++u)
#pragma unroll
        for (int v = 0; v < NV; ++v)
          if (on && (unsigned)(ke + u) < (unsigned)nz) {
            if (w[u][v].tag != y.epoch) w[u][v] = sweep_poll(p + ke + u + v * g.words(), y, dead);
            ring[(slot0 + u) % (2 * P)][v * E * E + at] = __longlong_as_double((long long)w[u][v].v);
          }
      block_barrier();
    }
  } else if (warp == 3) {
    const SweepPos<BWD> q(g, tile, along_i ? last : m, along_i ? m : last);
    const int start = -A * (last + m) - LOOK;
    const bool on = used && q.col && (along_i ? q.I + 1 < g.ti : q.J + 1 < g.tj);
    const int at = (q.li + 1) * E + q.lj + 1;
    TagWord *p = (along_i ? y.words + ((size_t)q.I * g.ny + q.j) * nz
                            : y.words + g.words_i() + ((size_t)q.J * g.nx + q.i) * nz) + start;
    step_barrier();
    for (int t0 = 0, h = 0; t0 < T; t0 += P, h = P - h) {
#pragma unroll
      for (int u = 0; u < P; ++u) {
        step_barrier();
        if (on && (unsigned)(start + t0 + u) < (unsigned)nz)
#pragma unroll
          for (int v = 0; v < NV; ++v) word_st(p + u + v * g.words(), ring[h + u][v * E * E + at], y.epoch);
      }
      p += P;
    }
  } else {
    const int col = threadIdx.x % kSweepCols;
    const SweepPos<BWD> q(g, tile, col / kSweepTile, col % kSweepTile);
    const int start = -A * (q.li + q.lj) - LOOK, at = (q.li + 1) * E + q.lj + 1;
    double *cur = &ring[0][at], *oth = &ring[P][at];   // this block's slots and the other half
    Body b(g, q, start, arg...);
    if (warp < 2) {
      const double *mine = &stage[0][0][col];
      step_barrier();
      for (int kk = start, t0 = 0; t0 < T; t0 += P, kk += P) {
        block_barrier();
#pragma unroll
        for (int u = 0; u < P; ++u) {
          const double *prev = u > 0 ? cur + (u - 1) * SLOT : oth + (P - 1) * SLOT;
          double w[NV], s[NV], o[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) { w[v] = prev[v * E * E - E]; s[v] = prev[v * E * E - 1]; }
          b.fetch(mine + u * (NP * kSweepCols));
          b.before(w, s);
          if (q.col && (unsigned)(kk + u) < (unsigned)nz) {
            b.step(u, kk + u, w, s, o);
#pragma unroll
            for (int v = 0; v < NV; ++v) cur[u * SLOT + v * E * E] = o[v];
          }
          b.after(w, s);
          step_barrier();
        }
        b.next();
        double *tmp = cur; cur = oth; oth = tmp;
      }
    } else {
      double *mine = &stage[0][0][col];
      auto load = [&](int u, int kk) {
        if (q.col && (unsigned)kk < (unsigned)nz) b.load(u, kk, mine + u % P * (NP * kSweepCols));
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      auto store = [&](int u, int kk, const double *slot) {
        if (q.col && (unsigned)kk < (unsigned)nz) b.store(u, slot[0]);
      };
#pragma unroll
      for (int u = 0; u < P - 1; ++u) load(u, start + u);
      asm volatile("cp.async.wait_group %0;" ::"n"(P - 2) : "memory");
      step_barrier();
      for (int kk = start, t0 = 0; t0 < T; t0 += P, kk += P) {
#pragma unroll
        for (int u = 0; u < P; ++u) {
          // the step after the last loaded one, into the slot of the step before this one
          load(u + P - 1, kk + u + P - 1);
          store(u - 1, kk + u - 1, u > 0 ? cur + (u - 1) * SLOT : oth + (P - 1) * SLOT);
          asm volatile("cp.async.wait_group %0;" ::"n"(P - 2) : "memory");
          step_barrier();
        }
        b.next();
        double *tmp = cur; cur = oth; oth = tmp;
      }
      store(-1, start + T - 1, oth + (P - 1) * SLOT);
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  }
  sweep_finish(y, g.tiles());
}

// Distance G of two operands in march order: a constant where tiles have all
// their columns (0.98-0.99 of the time of the variable one: the memory warps
// form fewer addresses), else the grid's.
template <bool FULL> struct MarchStride {
  static constexpr int G = kSweepCols;
  __device__ __forceinline__ explicit MarchStride(const SweepGeo &) {}
};
template <> struct MarchStride<false> {
  const int G;
  __device__ __forceinline__ explicit MarchStride(const SweepGeo &g) : G(g.cols) {}
};

// Body of a triangular sweep of z = M^-1 r: forward z = (r - lower terms) / c
// from r (natural order) into the factor's z plane, backward
// z = (that - upper terms) / c into z (natural order)
// (preconditioner_solve.cpp:14-110). Terms with a neighbour outside the
// domain are skipped (the reference multiplies them by its zero halo).
template <int KIND, bool BWD, bool FULL>
struct IcBody : MarchStride<FULL> {
  using MarchStride<FULL>::G;
  static constexpr int P = kSweepAhead, NP = ic_planes(KIND), C = kSweepCols, planes = NP;
  static constexpr int D = BWD ? -1 : 1;   // a step in natural order
  // coefficient rows: the cell's own (forward), or those of the neighbour
  // whose lower entry is this cell's upper one (backward)
  const double *lO, *lW, *lS, *lr;
  double *zO, *lz;
  int nz;
  bool hasW, hasS;
  double cw, ctw, cs, cts, cb, cc, cy, cr;
  double zB, zW0, zS0;
  __device__ __forceinline__ IcBody(const SweepGeo &g, const SweepPos<BWD> &q, int start, double *M, const double *r,
                                    double *z)
      : MarchStride<FULL>(g), nz(g.nz), hasW(q.hasW), hasS(q.hasS), zB(0.0), zW0(0.0), zS0(0.0) {
    const long long row = (long long)q.at(g, start) * (NP * G);
    const long long nat = ((long long)q.i * g.ny + q.j) * nz + q.at(g, start);
    lO = zO = M + ((long long)(q.col ? g.off(q.i, q.j, NP) : 0) + row);
    lW = BWD && hasW ? M + ((long long)g.off(q.i + 1, q.j, NP) + row) : lO;
    lS = BWD && hasS ? M + ((long long)g.off(q.i, q.j + 1, NP) + row) : lO;
    lr = r + nat;
    lz = z + nat;
  }
  __device__ __forceinline__ int march_step() const { return D * NP * G; }
  __device__ __forceinline__ void load(int u, int kk, double *d) {
    const int S = march_step(), o = u * S;
    sweep_copy(d + kIcC * C, lO + o + kIcC * G);
    sweep_copy(d + kIcY * C, lO + o + kIcY * G);
    sweep_copy(d + kIcZ * C, BWD ? lO + o + kIcZ * G : lr + u);
    if (!BWD || hasW) sweep_copy(d + kIcW * C, lW + o + kIcW * G);
    if (!BWD || hasS) sweep_copy(d + kIcS * C, lS + o + kIcS * G);
    if (!BWD || kk > 0) sweep_copy(d + kIcB * C, lO + o + kIcB * G - (BWD ? S : 0));
    if constexpr (KIND == 2) {
      if (!BWD || (hasW && kk + 1 < nz)) sweep_copy(d + kIcTw * C, lW + o + kIcTw * G + (BWD ? S : 0));
      if (!BWD || (hasS && kk + 1 < nz)) sweep_copy(d + kIcTs * C, lS + o + kIcTs * G + (BWD ? S : 0));
    }
  }
  __device__ __forceinline__ void fetch(const double *d) {
    cc = d[kIcC * C]; cy = d[kIcY * C]; cr = d[kIcZ * C];
    cw = d[kIcW * C]; cs = d[kIcS * C]; cb = d[kIcB * C];
    if constexpr (KIND == 2) { ctw = d[kIcTw * C]; cts = d[kIcTs * C]; }
  }
  __device__ __forceinline__ void next() {
    const int S = march_step();
    lO += P * S; lW += P * S; lS += P * S; lr += P * D; zO += P * S; lz += P * D;
  }
  __device__ __forceinline__ void store(int u, double z) {
    if (BWD) lz[u * D] = z;
    else zO[u * march_step() + kIcZ * G] = z;
  }
  __device__ __forceinline__ void before(const double *w, const double *s) {
    if constexpr (KIND == 1) { zW0 = w[0]; zS0 = s[0]; }
  }
  __device__ __forceinline__ void after(const double *w, const double *s) {
    if constexpr (KIND == 2) { zW0 = w[0]; zS0 = s[0]; }
  }
  __device__ __forceinline__ void step(int u, int kk, const double *w, const double *s, double *o) {
    double sum = cr;
    if (hasW) sum = msub(sum, cw, zW0);
    if (KIND == 2 && hasW && kk + 1 < nz) sum = msub(sum, ctw, w[0]);
    if (hasS) sum = msub(sum, cs, zS0);
    if (KIND == 2 && hasS && kk + 1 < nz) sum = msub(sum, cts, s[0]);
    if (kk > 0) sum = msub(sum, cb, zB);
    zB = sweep_div(sum, cc, cy);
    o[0] = zB;
  }
};

template <int KIND, bool BWD, bool FULL>
__global__ void __launch_bounds__(kSweepThreads) k_ic_sweep(SweepGeo g, double *M, const double *__restrict__ r,
                                                            double *__restrict__ z, SweepSync y,
                                                            const KrylovState *st) {
  if (st->done) return;
  sweep_march<1, sweep_a(KIND), KIND == 2 ? 1 : 0, BWD, IcBody<KIND, BWD, FULL>>(g, y, M, r, z);
}

// IncompleteCholesky0/2::form (preconditioner_form.cpp:16-98) in march
// order. The reference pushes each entry of the factor from the cell that
// completes it; here a cell forms its own entries from the same operands:
// with p the cell before it along i, j or k (for tw and ts at k + 1),
//   w = -A.w / c_p,  s = -A.s / c_p,  tw = -w b_p / c_p,  ts = -s b_p / c_p,
//   b = -A.b / c_p (IC0) or (-A.b - w tw_p - s ts_p) / c_p (IC2),
//   c = sqrt(A.c - w^2 - tw^2 - s^2 - ts^2 - b^2),
// so only c and b travel between columns. Entries whose p lies outside the
// domain are zero.
template <int KIND, bool FULL>
struct IcFormBody : MarchStride<FULL> {
  using MarchStride<FULL>::G;
  static constexpr int P = kSweepAhead, NP = ic_planes(KIND), C = kSweepCols, planes = 4;
  const double *ac, *aw, *as, *ab;
  double *o_;
  int nz;
  bool hasW, hasS;
  double rc, rw, rs, rb;
  double cB, twB, tsB, cW0, cS0;
  __device__ __forceinline__ IcFormBody(const SweepGeo &g, const SweepPos<false> &q, int start,
                                        const MatView<double> &A, double *M)
      : MarchStride<FULL>(g), nz(g.nz), hasW(q.hasW), hasS(q.hasS), cB(0.0), twB(0.0), tsB(0.0), cW0(0.0), cS0(0.0) {
    const long long nat = ((long long)q.i * g.ny + q.j) * nz + start;
    ac = A.c + nat; aw = A.w + nat; as = A.s + nat; ab = A.b + nat;
    o_ = M + ((long long)(q.col ? g.off(q.i, q.j, NP) : 0) + (long long)start * (NP * G));
  }
  __device__ __forceinline__ void load(int u, int, double *d) {
    sweep_copy(d, ac + u); sweep_copy(d + C, aw + u); sweep_copy(d + 2 * C, as + u); sweep_copy(d + 3 * C, ab + u);
  }
  __device__ __forceinline__ void fetch(const double *d) { rc = d[0]; rw = d[C]; rs = d[2 * C]; rb = d[3 * C]; }
  __device__ __forceinline__ void next() { ac += P; aw += P; as += P; ab += P; o_ += P * NP * G; }
  __device__ __forceinline__ void store(int, double) {}   // the arithmetic warps hold the factor
  __device__ __forceinline__ void before(const double *w, const double *s) {
    if constexpr (KIND == 1) { cW0 = w[0]; cS0 = s[0]; }
  }
  __device__ __forceinline__ void after(const double *w, const double *s) {
    if constexpr (KIND == 2) { cW0 = w[0]; cS0 = s[0]; }
  }
  // w, s: c and b of the columns beside at kk + LOOK
  __device__ __forceinline__ void step(int u, int kk, const double *wv, const double *sv, double *out) {
    const double w = hasW ? __ddiv_rn(-rw, cW0) : 0.0;
    const double s = hasS ? __ddiv_rn(-rs, cS0) : 0.0;
    double tw = 0.0, ts = 0.0, b = 0.0;
    if constexpr (KIND == 2) {
      if (hasW && kk + 1 < nz) tw = __ddiv_rn(__dmul_rn(-w, wv[1]), wv[0]);
      if (hasS && kk + 1 < nz) ts = __ddiv_rn(__dmul_rn(-s, sv[1]), sv[0]);
    }
    if (kk > 0) {
      double n = -rb;
      if (KIND == 2) n = msub(msub(n, w, twB), s, tsB);
      b = __ddiv_rn(n, cB);
    }
    double c = msub(rc, w, w);
    if (KIND == 2) c = msub(c, tw, tw);
    c = msub(c, s, s);
    if (KIND == 2) c = msub(c, ts, ts);
    c = __dsqrt_rn(msub(c, b, b));
    out[0] = c;
    if constexpr (KIND == 2) out[1] = b;
    double *o = o_ + u * (NP * G);
    o[kIcC * G] = c;
    o[kIcY * G] = KnownDiv(c).recip();
    o[kIcW * G] = w; o[kIcS * G] = s; o[kIcB * G] = b;
    if constexpr (KIND == 2) { o[kIcTw * G] = tw; o[kIcTs * G] = ts; }
    cB = c; twB = tw; tsB = ts;
  }
};

template <int KIND, bool FULL>
__global__ void __launch_bounds__(kSweepThreads) k_ic_factor(SweepGeo g, MatView<double> A, double *M, SweepSync y) {
  sweep_march<KIND == 2 ? 2 : 1, sweep_a(KIND), KIND == 2 ? 1 : 0, false, IcFormBody<KIND, FULL>>(g, y, A, M);
}

__global__ void k_gs_pack(SweepGeo g, MatView<double> A, const double *__restrict__ ci,
                          const double *__restrict__ b, const double *__restrict__ x, double *o) {
  const size_t n = g.all_rows() * g.cols;
  for (size_t m = blockIdx.x * (size_t)blockDim.x + threadIdx.x; m < n; m += (size_t)gridDim.x * blockDim.x) {
    const size_t row = m / g.cols;
    const int c = (int)(m - row * g.cols);
    const int tile = (int)(row / g.rows), li = c / g.wj, lj = c - li * g.wj;
    const int k = (int)(row - (size_t)tile * g.rows) - g.skew * (li + lj);
    const int i = tile / g.tj * kSweepTile + li, j = tile % g.tj * kSweepTile + lj;
    if (i >= g.nx || j >= g.ny || k < 0 || k >= g.nz) continue;
    const long long p = ((long long)i * g.ny + j) * g.nz + k;
    const Nb<double> a = coeffs(A, p, Pos{i, j, k});
    double *w = o + row * (kGsPlanes * g.cols) + c;
    const double v[kGsPlanes] = {b[p], ci[p], a.w, a.e, a.s, a.n, a.b, a.t, x[p]};
#pragma unroll
    for (int f = 0; f < kGsPlanes; ++f) w[f * g.cols] = v[f];
  }
}

// One Gauss-Seidel sweep: x = ci (b + w xw + e xe + s xs + n xn + b xb +
// t xt) summed left to right (gaussseidel.cpp:50-60), new values before the
// cell, old ones after it, into the march-order x and the natural one. The
// old values are loaded before their cells' new ones are formed: those wait,
// directly or through the exchange, for this cell's own result. A neighbour
// outside the domain counts as zero.
template <bool FULL>
struct GsBody : MarchStride<FULL> {
  using MarchStride<FULL>::G;
  static constexpr int P = kSweepAhead, C = kSweepCols, planes = kGsPlanes + 2;
  const double *lO, *lE, *lN;
  double *xO, *lx;
  int nz;
  bool hasW, hasS, hasE, hasN;
  double rb, rci, rw, re, rs, rn, rbt, rt, xe, xn, xt;
  double xB;
  __device__ __forceinline__ GsBody(const SweepGeo &g, const SweepPos<false> &q, int start, double *M, double *x)
      : MarchStride<FULL>(g), nz(g.nz), hasW(q.hasW), hasS(q.hasS), hasE(q.col && q.i + 1 < g.nx),
        hasN(q.col && q.j + 1 < g.ny), xB(0.0) {
    const long long row = (long long)start * march_step();
    lO = M + ((long long)(q.col ? g.off(q.i, q.j, kGsPlanes) : 0) + row);
    lE = hasE ? M + ((long long)g.off(q.i + 1, q.j, kGsPlanes) + row) : lO;
    lN = hasN ? M + ((long long)g.off(q.i, q.j + 1, kGsPlanes) + row) : lO;
    xO = const_cast<double *>(lO) + kGsX * G;
    lx = x + (((long long)q.i * g.ny + q.j) * nz + start);
  }
  __device__ __forceinline__ int march_step() const { return kGsPlanes * G; }
  // planes of a stage: the cell's eight operands, then the old x at i + 1, j + 1 and k + 1
  __device__ __forceinline__ void load(int u, int kk, double *d) {
    const int S = march_step();
    const double *l = lO + u * S;
#pragma unroll
    for (int f = 0; f < kGsX; ++f) sweep_copy(d + f * C, l + f * G);
    if (hasE) sweep_copy(d + kGsX * C, lE + u * S + kGsX * G);
    if (hasN) sweep_copy(d + (kGsX + 1) * C, lN + u * S + kGsX * G);
    if (kk + 1 < nz) sweep_copy(d + (kGsX + 2) * C, l + kGsX * G + S);
  }
  __device__ __forceinline__ void fetch(const double *d) {
    rb = d[kGsB * C]; rci = d[kGsCi * C];
    rw = d[kGsW * C]; re = d[kGsE * C]; rs = d[kGsS * C]; rn = d[kGsN * C]; rbt = d[kGsBt * C]; rt = d[kGsT * C];
    xe = d[kGsX * C]; xn = d[(kGsX + 1) * C]; xt = d[(kGsX + 2) * C];
  }
  __device__ __forceinline__ void next() {
    const int S = march_step();
    lO += P * S; lE += P * S; lN += P * S; xO += P * S; lx += P;
  }
  __device__ __forceinline__ void store(int u, double v) { xO[u * march_step()] = v; lx[u] = v; }
  __device__ __forceinline__ void before(const double *, const double *) {}
  __device__ __forceinline__ void after(const double *, const double *) {}
  __device__ __forceinline__ void step(int u, int kk, const double *w, const double *s, double *o) {
    double v = rb;
    v = __dadd_rn(v, __dmul_rn(rw, hasW ? w[0] : 0.0));
    v = __dadd_rn(v, __dmul_rn(re, hasE ? xe : 0.0));
    v = __dadd_rn(v, __dmul_rn(rs, hasS ? s[0] : 0.0));
    v = __dadd_rn(v, __dmul_rn(rn, hasN ? xn : 0.0));
    v = __dadd_rn(v, __dmul_rn(rbt, xB));
    v = __dadd_rn(v, __dmul_rn(rt, kk + 1 < nz ? xt : 0.0));
    xB = __dmul_rn(rci, v);
    o[0] = xB;
  }
};

template <bool FULL>
__global__ void __launch_bounds__(kSweepThreads) k_gs_sweep(SweepGeo g, double *M, double *__restrict__ x, SweepSync y,
                                                            const KrylovState *st) {
  if (st->done) return;
  sweep_march<1, 1, 0, false, GsBody<FULL>>(g, y, M, x);
}

}  // namespace pbg
