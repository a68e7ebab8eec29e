// Kernels of the lexicographic sweeps (schedule and storage: pbg_sweeps.cuh).
#pragma once

#include "pbg_sweeps.cuh"

namespace pbg {

__device__ __forceinline__ SweepWord sweep_ld(const SweepWord *p) {
  SweepWord w;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(w.v), "=l"(w.epoch) : "l"(p) : "memory");
  return w;
}
__device__ __forceinline__ void sweep_st(SweepWord *p, double v, unsigned long long epoch) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}"
               :: "l"(p), "l"((unsigned long long)__double_as_longlong(v)), "l"(epoch) : "memory");
}

// a / c with c's stored reciprocal (KnownDiv with its range check kept in y)
__device__ __forceinline__ double sweep_div(double a, double c, double y) {
  const double m = fabs(a);
  if (m > 0x1p-900 && m < 0x1p900 && y == y) {
    const double q0 = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q0, c, a), y, q0);
  }
  if (m == 0.0 && y == y) return __dmul_rn(a, c);
  return __ddiv_rn(a, c);
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

// The word p of this launch's epoch: w as loaded early, polled until valid.
// A poll that runs out (or one that did elsewhere) sets *stuck and goes on
// with zero, so that every block ends; the host reports the failure.
__device__ __forceinline__ double sweep_wait(SweepWord w, const SweepWord *p, const SweepSync &y, bool &dead) {
  if (w.epoch != y.epoch) {
    for (int n = 1; !dead; ++n) {
      w = sweep_ld(p);
      if (w.epoch == y.epoch) break;
      if (n >= kSweepPoll) { atomicExch(y.stuck, 1); dead = true; }
      else if ((n & 1023) == 0 && *(volatile int *)y.stuck) dead = true;
    }
    if (w.epoch != y.epoch) return 0.0;
  }
  return __longlong_as_double((long long)w.v);
}

// Position of a thread in the march. In a backward sweep i, j and k run
// down: li, lj, kk and the tile indices count in march direction.
template <bool BWD>
struct SweepPos {
  int I, J, li, lj, i, j;
  bool col, hasW, hasS;   // the column, and those before it along i and along j, exist
  __device__ __forceinline__ SweepPos(const SweepGeo &g, int tile) {
    I = tile / g.tj; J = tile - I * g.tj;
    li = threadIdx.x / kSweepTile; lj = threadIdx.x % kSweepTile;
    const int mi = I * kSweepTile + li, mj = J * kSweepTile + lj;
    i = BWD ? g.ti * kSweepTile - 1 - mi : mi;
    j = BWD ? g.tj * kSweepTile - 1 - mj : mj;
    col = i < g.nx && j < g.ny;
    hasW = col && (BWD ? i + 1 < g.nx : i > 0);
    hasS = col && (BWD ? j + 1 < g.ny : j > 0);
  }
  __device__ __forceinline__ int at(const SweepGeo &g, int kk) const { return BWD ? g.nz - 1 - kk : kk; }
};

// z = M^-1 r, one of its two triangular sweeps: forward
// z = (r - lower terms) / c from r (natural order) into zm (march order),
// backward z = (zm - upper terms) / c into z (natural order)
// (preconditioner_solve.cpp:14-110). Terms with a neighbour outside the
// domain are skipped (the reference multiplies them by its zero halo).
template <int KIND, bool BWD>
__global__ void __launch_bounds__(kSweepCols) k_ic_sweep(SweepGeo g, IcFactor M, const double *__restrict__ r,
                                                         double *__restrict__ zm, double *__restrict__ z,
                                                         SweepSync y, const KrylovState *st) {
  if (st->done) return;
  constexpr int A = sweep_a(KIND), P = kSweepAhead, LOOK = KIND == 2 ? 1 : 0;
  __shared__ double ring[2][kSweepCols];
  const SweepPos<BWD> q(g, sweep_ticket(y));
  const int me = threadIdx.x, skew = A * (q.li + q.lj) + LOOK, nz = g.nz;
  const long long nat = ((long long)q.i * g.ny + q.j) * nz;
  // coefficient rows: the cell's own (forward), or those of the neighbour
  // whose lower entry is this cell's upper one (backward)
  const size_t oO = q.col ? g.off(q.i, q.j) : 0;
  const size_t oW = BWD && q.hasW ? g.off(q.i + 1, q.j) : oO;
  const size_t oS = BWD && q.hasS ? g.off(q.i, q.j + 1) : oO;
  constexpr int back = BWD ? kSweepCols : 0;
  // columns read from, and published to, the tiles beside this one
  const bool exW = q.hasW && q.li == 0, exS = q.hasS && q.lj == 0;
  const bool putI = q.col && q.li == kSweepTile - 1, putJ = q.col && q.lj == kSweepTile - 1;
  SweepWord *pi = y.words + ((size_t)q.I * g.ny + q.j) * nz;
  SweepWord *pj = y.words + g.words_i() + ((size_t)q.J * g.nx + q.i) * nz;
  const SweepWord *wi = pi - (size_t)g.ny * nz, *wj = pj - (size_t)g.nx * nz;
  double cw[P], ctw[P], cs[P], cts[P], cb[P], cc[P], cy[P], cr[P];
  SweepWord eW[P], eS[P];
  auto load = [&](int u, int t) {
    const int kk = t - skew, ke = kk + LOOK;
    if (q.col && kk >= 0 && kk < nz) {
      const int k = q.at(g, kk);
      const size_t ko = (size_t)k * kSweepCols;
      cc[u] = M.c[oO + ko];
      cy[u] = M.y[oO + ko];
      cr[u] = BWD ? zm[oO + ko] : r[nat + k];
      if (q.hasW) cw[u] = M.w[oW + ko];
      if (q.hasS) cs[u] = M.s[oS + ko];
      if (kk > 0) cb[u] = M.b[oO + ko + back];
      if constexpr (KIND == 2) {
        if (kk + 1 < nz && q.hasW) ctw[u] = M.tw[oW + ko - back];
        if (kk + 1 < nz && q.hasS) cts[u] = M.ts[oS + ko - back];
      }
    }
    if (exW && ke >= 0 && ke < nz) eW[u] = sweep_ld(wi + ke);
    if (exS && ke >= 0 && ke < nz) eS[u] = sweep_ld(wj + ke);
  };
#pragma unroll
  for (int u = 0; u < P; ++u) load(u, u);
  const int T = nz + 2 * A * (kSweepTile - 1) + LOOK;
  double zB = 0.0, zW0 = 0.0, zS0 = 0.0;
  bool dead = false;
  for (int t0 = 0; t0 < T; t0 += P) {
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const int t = t0 + u;
      if (t >= T) break;
      const int kk = t - skew, ke = kk + LOOK;
      double zW1 = 0.0, zS1 = 0.0;   // the columns beside, at kk + LOOK
      if (ke >= 0 && ke < nz) {
        if (exW) zW1 = sweep_wait(eW[u], wi + ke, y, dead);
        else if (q.hasW) zW1 = ring[(t - 1) & 1][me - kSweepTile];
        if (exS) zS1 = sweep_wait(eS[u], wj + ke, y, dead);
        else if (q.hasS) zS1 = ring[(t - 1) & 1][me - 1];
      }
      if constexpr (LOOK == 0) { zW0 = zW1; zS0 = zS1; }
      if (q.col && kk >= 0 && kk < nz) {
        double sum = cr[u];
        if (q.hasW) sum = msub(sum, cw[u], zW0);
        if (KIND == 2 && q.hasW && kk + 1 < nz) sum = msub(sum, ctw[u], zW1);
        if (q.hasS) sum = msub(sum, cs[u], zS0);
        if (KIND == 2 && q.hasS && kk + 1 < nz) sum = msub(sum, cts[u], zS1);
        if (kk > 0) sum = msub(sum, cb[u], zB);
        zB = sweep_div(sum, cc[u], cy[u]);
        ring[t & 1][me] = zB;
        if (putI) sweep_st(pi + kk, zB, y.epoch);
        if (putJ) sweep_st(pj + kk, zB, y.epoch);
        const int k = q.at(g, kk);
        if (BWD) z[nat + k] = zB;
        else zm[oO + (size_t)k * kSweepCols] = zB;
      }
      if constexpr (LOOK == 1) { zW0 = zW1; zS0 = zS1; }
      load(u, t + P);
      __syncthreads();
    }
  }
  sweep_finish(y, g.tiles());
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
template <int KIND>
__global__ void __launch_bounds__(kSweepCols) k_ic_factor(SweepGeo g, MatView<double> A, IcFactor M, SweepSync y) {
  constexpr int W = sweep_a(KIND), P = kSweepAhead, LOOK = KIND == 2 ? 1 : 0;
  __shared__ double rc[2][kSweepCols], rb[2][kSweepCols];
  const SweepPos<false> q(g, sweep_ticket(y));
  const int me = threadIdx.x, skew = W * (q.li + q.lj) + LOOK, nz = g.nz;
  const long long nat = ((long long)q.i * g.ny + q.j) * nz;
  const size_t oO = q.col ? g.off(q.i, q.j) : 0;
  const bool exW = q.hasW && q.li == 0, exS = q.hasS && q.lj == 0;
  const bool putI = q.col && q.li == kSweepTile - 1, putJ = q.col && q.lj == kSweepTile - 1;
  SweepWord *pi = y.words + ((size_t)q.I * g.ny + q.j) * nz;
  SweepWord *pj = y.words + g.words_i() + ((size_t)q.J * g.nx + q.i) * nz;
  const SweepWord *wi = pi - (size_t)g.ny * nz, *wj = pj - (size_t)g.nx * nz;
  const size_t vb = g.words();   // the words of b follow those of c
  double ac[P], aw[P], as[P], ab[P];
  SweepWord eW[P], eWb[P], eS[P], eSb[P];
  auto load = [&](int u, int t) {
    const int kk = t - skew, ke = kk + LOOK;
    if (q.col && kk >= 0 && kk < nz) {
      ac[u] = A.c[nat + kk]; aw[u] = A.w[nat + kk]; as[u] = A.s[nat + kk]; ab[u] = A.b[nat + kk];
    }
    if (exW && ke >= 0 && ke < nz) { eW[u] = sweep_ld(wi + ke); if (KIND == 2) eWb[u] = sweep_ld(wi + vb + ke); }
    if (exS && ke >= 0 && ke < nz) { eS[u] = sweep_ld(wj + ke); if (KIND == 2) eSb[u] = sweep_ld(wj + vb + ke); }
  };
  // c and b of a column beside this one at ke
  auto beside = [&](const SweepWord &wc, const SweepWord &wb, const SweepWord *w, bool ex, int from, int t, int ke,
                    bool &dead, double &c, double &b) {
    if (ex) {
      c = sweep_wait(wc, w + ke, y, dead);
      if (KIND == 2) b = sweep_wait(wb, w + vb + ke, y, dead);
    } else {
      c = rc[(t - 1) & 1][from];
      if (KIND == 2) b = rb[(t - 1) & 1][from];
    }
  };
#pragma unroll
  for (int u = 0; u < P; ++u) load(u, u);
  const int T = nz + 2 * W * (kSweepTile - 1) + LOOK;
  double cB = 0.0, twB = 0.0, tsB = 0.0;   // of the cell before along k
  double cW0 = 0.0, cS0 = 0.0;
  bool dead = false;
  for (int t0 = 0; t0 < T; t0 += P) {
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const int t = t0 + u;
      if (t >= T) break;
      const int kk = t - skew, ke = kk + LOOK;
      double cW1 = 0.0, bW1 = 0.0, cS1 = 0.0, bS1 = 0.0;
      if (ke >= 0 && ke < nz) {
        if (q.hasW) beside(eW[u], eWb[u], wi, exW, me - kSweepTile, t, ke, dead, cW1, bW1);
        if (q.hasS) beside(eS[u], eSb[u], wj, exS, me - 1, t, ke, dead, cS1, bS1);
      }
      if constexpr (LOOK == 0) { cW0 = cW1; cS0 = cS1; }
      if (q.col && kk >= 0 && kk < nz) {
        const double w = q.hasW ? __ddiv_rn(-aw[u], cW0) : 0.0;
        const double s = q.hasS ? __ddiv_rn(-as[u], cS0) : 0.0;
        double tw = 0.0, ts = 0.0, b = 0.0;
        if (KIND == 2 && q.hasW && kk + 1 < nz) tw = __ddiv_rn(__dmul_rn(-w, bW1), cW1);
        if (KIND == 2 && q.hasS && kk + 1 < nz) ts = __ddiv_rn(__dmul_rn(-s, bS1), cS1);
        if (kk > 0) {
          double n = -ab[u];
          if (KIND == 2) n = msub(msub(n, w, twB), s, tsB);
          b = __ddiv_rn(n, cB);
        }
        double c = msub(ac[u], w, w);
        if (KIND == 2) c = msub(c, tw, tw);
        c = msub(c, s, s);
        if (KIND == 2) c = msub(c, ts, ts);
        c = __dsqrt_rn(msub(c, b, b));
        rc[t & 1][me] = c;
        rb[t & 1][me] = b;
        if (putI) { sweep_st(pi + kk, c, y.epoch); if (KIND == 2) sweep_st(pi + vb + kk, b, y.epoch); }
        if (putJ) { sweep_st(pj + kk, c, y.epoch); if (KIND == 2) sweep_st(pj + vb + kk, b, y.epoch); }
        const size_t o = oO + (size_t)kk * kSweepCols;
        M.c[o] = c;
        M.y[o] = KnownDiv(c).recip();
        M.w[o] = w; M.s[o] = s; M.b[o] = b;
        if (KIND == 2) { M.tw[o] = tw; M.ts[o] = ts; }
        cB = c; twB = tw; tsB = ts;
      }
      if constexpr (LOOK == 1) { cW0 = cW1; cS0 = cS1; }
      load(u, t + P);
      __syncthreads();
    }
  }
  sweep_finish(y, g.tiles());
}


__global__ void k_gs_pack(SweepGeo g, MatView<double> A, const double *__restrict__ ci,
                          const double *__restrict__ b, const double *__restrict__ x, GsOps o) {
  const size_t n = g.size();
  for (size_t m = blockIdx.x * (size_t)blockDim.x + threadIdx.x; m < n; m += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(m % kSweepCols);
    const size_t row = m / kSweepCols;
    const int tile = (int)(row / g.rows), li = c / kSweepTile, lj = c % kSweepTile;
    const int k = (int)(row - (size_t)tile * g.rows) - g.skew * (li + lj);
    const int i = tile / g.tj * kSweepTile + li, j = tile % g.tj * kSweepTile + lj;
    if (i >= g.nx || j >= g.ny || k < 0 || k >= g.nz) continue;
    const long long p = ((long long)i * g.ny + j) * g.nz + k;
    const Nb<double> a = coeffs(A, p, Pos{i, j, k});
    o.b[m] = b[p]; o.ci[m] = ci[p]; o.x[m] = x[p];
    o.w[m] = a.w; o.e[m] = a.e; o.s[m] = a.s; o.n[m] = a.n; o.bt[m] = a.b; o.t[m] = a.t;
  }
}

// One Gauss-Seidel sweep: x = ci (b + w xw + e xe + s xs + n xn + b xb +
// t xt) summed left to right (gaussseidel.cpp:50-60), new values before the
// cell, old ones after it, into the march-order x and the natural one. The
// old values are loaded before their cells' new ones are formed: those wait,
// directly or through the exchange, for this cell's own result. A neighbour
// outside the domain counts as zero.
__global__ void __launch_bounds__(kSweepCols) k_gs_sweep(SweepGeo g, GsOps o, double *__restrict__ x, SweepSync y,
                                                         const KrylovState *st) {
  if (st->done) return;
  constexpr int P = kSweepAhead;
  __shared__ double ring[2][kSweepCols];
  const SweepPos<false> q(g, sweep_ticket(y));
  const int me = threadIdx.x, skew = q.li + q.lj, nz = g.nz;
  const long long nat = ((long long)q.i * g.ny + q.j) * nz;
  const size_t oO = q.col ? g.off(q.i, q.j) : 0;
  const bool hasE = q.col && q.i + 1 < g.nx, hasN = q.col && q.j + 1 < g.ny;
  const size_t oE = hasE ? g.off(q.i + 1, q.j) : oO, oN = hasN ? g.off(q.i, q.j + 1) : oO;
  const bool exW = q.hasW && q.li == 0, exS = q.hasS && q.lj == 0;
  const bool putI = q.col && q.li == kSweepTile - 1, putJ = q.col && q.lj == kSweepTile - 1;
  SweepWord *pi = y.words + ((size_t)q.I * g.ny + q.j) * nz;
  SweepWord *pj = y.words + g.words_i() + ((size_t)q.J * g.nx + q.i) * nz;
  const SweepWord *wi = pi - (size_t)g.ny * nz, *wj = pj - (size_t)g.nx * nz;
  double *xs = o.x;
  double rb[P], rci[P], rw[P], re[P], rs[P], rn[P], rbt[P], rt[P], xe[P], xn[P], xt[P];
  SweepWord eW[P], eS[P];
  auto load = [&](int u, int t) {
    const int kk = t - skew;
    if (!q.col || kk < 0 || kk >= nz) return;
    const size_t m = oO + (size_t)kk * kSweepCols;
    rb[u] = o.b[m]; rci[u] = o.ci[m];
    rw[u] = o.w[m]; re[u] = o.e[m]; rs[u] = o.s[m]; rn[u] = o.n[m]; rbt[u] = o.bt[m]; rt[u] = o.t[m];
    xe[u] = hasE ? __ldcg(xs + oE + (size_t)kk * kSweepCols) : 0.0;
    xn[u] = hasN ? __ldcg(xs + oN + (size_t)kk * kSweepCols) : 0.0;
    xt[u] = kk + 1 < nz ? __ldcg(xs + m + kSweepCols) : 0.0;
    if (exW) eW[u] = sweep_ld(wi + kk);
    if (exS) eS[u] = sweep_ld(wj + kk);
  };
#pragma unroll
  for (int u = 0; u < P; ++u) load(u, u);
  const int T = nz + 2 * (kSweepTile - 1);
  double xB = 0.0;
  bool dead = false;
  for (int t0 = 0; t0 < T; t0 += P) {
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const int t = t0 + u;
      if (t >= T) break;
      const int kk = t - skew;
      if (q.col && kk >= 0 && kk < nz) {
        double xW = 0.0, xS = 0.0;
        if (exW) xW = sweep_wait(eW[u], wi + kk, y, dead);
        else if (q.hasW) xW = ring[(t - 1) & 1][me - kSweepTile];
        if (exS) xS = sweep_wait(eS[u], wj + kk, y, dead);
        else if (q.hasS) xS = ring[(t - 1) & 1][me - 1];
        double v = rb[u];
        v = __dadd_rn(v, __dmul_rn(rw[u], xW));
        v = __dadd_rn(v, __dmul_rn(re[u], xe[u]));
        v = __dadd_rn(v, __dmul_rn(rs[u], xS));
        v = __dadd_rn(v, __dmul_rn(rn[u], xn[u]));
        v = __dadd_rn(v, __dmul_rn(rbt[u], xB));
        v = __dadd_rn(v, __dmul_rn(rt[u], xt[u]));
        xB = __dmul_rn(rci[u], v);
        ring[t & 1][me] = xB;
        if (putI) sweep_st(pi + kk, xB, y.epoch);
        if (putJ) sweep_st(pj + kk, xB, y.epoch);
        xs[oO + (size_t)kk * kSweepCols] = xB;
        x[nat + kk] = xB;
      }
      load(u, t + P);
      __syncthreads();
    }
  }
  sweep_finish(y, g.tiles());
}

}  // namespace pbg
