// Exact-order FP64 summation in parallel.
//
// The reference adds a dot product's terms one after another in i,j,k order
// with round-to-nearest after every addition (`for_ijk sum += ...`,
// Src/Field/Scalar/scalar.h:296-326). The reference-parity solvers reproduce
// that sum to the bit. A single thread adding 16.7 M terms takes tens of
// milliseconds per dot product, so the sum is computed like this instead.
//
// Binade argument. Let s be the running sum, 2^e <= |s| < 2^(e+1), and
// u = 2^(e-52) its ulp. While the running sum stays inside that binade every
// partial sum is an integer multiple of u, and
//     fl(s + a) = s + u * rint(a / u)       (round half to even),
// unless a/u is exactly half-way between two integers (a tie, whose
// direction depends on the parity of s/u). So over a stretch of terms that
// keeps the sum in one binade and holds no tie, the sequential sum is s plus
// u times an integer sum, which any order computes exactly.
//
// Per chunk of kThreads terms (one block of the reducing kernel):
//   1. the terms are stored (for the chunks that need a sequential pass);
//   2. an approximate prefix of all earlier terms comes from a decoupled
//      look-back over the chunks' published sums (bounded polling: a block
//      that gives up only loses its hint);
//   3. for the exponent of the approximate sum before its first term, each
//      warp computes K = sum of rint(a/u) over its 32 terms, the minimum and
//      maximum of its running integer prefix, and whether every term was
//      tie-free and finite; the chunk's record composes its warps' records
//      where they share the exponent (32 zero terms fit any);
//   4. the last chunk of each group of kExactGroup chunks to arrive composes
//      the group's records in the same way;
//   5. the last block of the launch walks the groups in order with the exact
//      running sum (one warp per sum): 32 records at a time, a scan of their
//      K gives each record's running sum, and every record up to the first
//      that does not hold the current exponent or does not keep s/u + prefix
//      inside [2^52 + 1, 2^53 - 1] is applied at once, as s += u K. A group
//      that stops the run is entered at its chunks, a chunk at its warps, and
//      the 32 terms of a warp that stops it are added one by one.
// Every step of the walk is either the sequential rounding itself or an
// integer sum proven equal to it, so the result is the sequential sum bit
// for bit whatever the hints were; bad hints only cost time.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "pbg_word.cuh"

namespace pbg {

constexpr int kExactChunkThreads = 256;  // terms per chunk (the reducing block)
constexpr int kExactWarps = kExactChunkThreads / 32;  // warp records per chunk
constexpr int kExactGroup = 64;          // chunks per group record
constexpr int kExactVals = 2;            // sums per reducing kernel at most
constexpr int kExactPoll = 4096;         // look-back polls before a block gives up its hint

// Record of a warp's terms, a chunk or a group at the exponent e.
enum : int { kExactNone, kExactOk, kExactZero };   // kExactZero: every term is zero, fits any sum
struct ExactRec {
  long long K, mn, mx;
  int e, ok;
};

// Header stored kExactHdrBytes before the terms (the `seq` pointer).
struct ExactHdr {
  ExactRec *wrec;      // [kExactVals][cap_chunks][kExactWarps] (32 terms each)
  ExactRec *crec;      // [kExactVals][cap_chunks]
  ExactRec *grec;      // [kExactVals][cap_groups]
  TagWord *sum;        // [kExactVals][cap_chunks] hints: the chunk's sum, tag (gen << 2) | 1,
                       // then the sum of all chunks up to it, tag (gen << 2) | 2
  unsigned *gcount;    // [cap_groups] chunk arrivals per group, zero between uses
  long long cap_chunks, cap_groups;
  unsigned gen;        // launch generation of the hints' tags
  unsigned pad;
};
constexpr size_t kExactHdrBytes = 256;
static_assert(sizeof(ExactHdr) <= kExactHdrBytes, "exact-sum header");

// Doubles of a scratch buffer for terms of ncell cells (header and records
// included); the `seq` pointer handed to the kernels is exact_seq(base).
inline size_t exact_scratch_doubles(long long ncell) {
  const long long ch = (ncell + kExactChunkThreads - 1) / kExactChunkThreads + 1;
  const long long gr = (ch + kExactGroup - 1) / kExactGroup + 1;
  size_t bytes = kExactHdrBytes + sizeof(double) * (size_t)kExactVals * ncell;
  bytes += sizeof(ExactRec) * kExactVals * (size_t)(ch * (kExactWarps + 1) + gr);
  bytes += sizeof(TagWord) * kExactVals * (size_t)ch;
  bytes += sizeof(unsigned) * (size_t)gr + 1024;
  return (bytes + 7) / 8;
}
inline double *exact_seq(double *base) { return base + kExactHdrBytes / 8; }

__device__ __forceinline__ const ExactHdr *exact_hdr(const double *seq) {
  return reinterpret_cast<const ExactHdr *>(reinterpret_cast<const char *>(seq) - kExactHdrBytes);
}

__device__ __forceinline__ unsigned ld_volatile_u32(const unsigned *p) {
  return *reinterpret_cast<const volatile unsigned *>(p);
}

// Record load through L2 (records written by other blocks of the launch).
__device__ __forceinline__ ExactRec exact_load(const ExactRec *s) {
  ExactRec d;
  d.K = __ldcg(&s->K);
  d.mn = __ldcg(&s->mn);
  d.mx = __ldcg(&s->mx);
  d.e = __ldcg(&s->e);
  d.ok = __ldcg(&s->ok);
  return d;
}

constexpr long long kExact53 = 1LL << 53;

// Exponent and integer significand of a normal double, and back: s = S *
// 2^(e-52), 2^52 <= |S| < 2^53.
__device__ __forceinline__ int exact_exp(double s) { return (int)((__double2hiint(s) >> 20) & 0x7ff) - 1023; }
__device__ __forceinline__ long long exact_int(double s) {
  const long long b = __double_as_longlong(s), m = (b & ((1LL << 52) - 1)) | (1LL << 52);
  return b < 0 ? -m : m;
}
__device__ __forceinline__ double exact_double(long long S, int e) {
  const long long m = S < 0 ? -S : S;
  const long long b = (m & ((1LL << 52) - 1)) | ((long long)(e + 1023) << 52);
  return __longlong_as_double(S < 0 ? b | (long long)0x8000000000000000ULL : b);
}
// 2^e, -1022 <= e <= 1023
__device__ __forceinline__ double exact_pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
// the exponents the records cover (s normal, and its unit and 2^53 units too)
__device__ __forceinline__ bool exact_in_range(int e) { return e >= -960 && e <= 960; }

// Composition of the records of a warp's lanes (lane < cnt, in lane order)
// into one, the same in every lane. e: the exponent they must share.
__device__ __forceinline__ ExactRec exact_compose(const ExactRec &r, int cnt, int e) {
  const int lane = threadIdx.x & 31;
  const bool in = lane < cnt, fits = !in || r.ok == kExactZero || (r.ok == kExactOk && r.e == e);
  const long long k = in && r.ok == kExactOk ? r.K : 0;
  long long incl = k;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += y;
  }
  const bool has = in && r.ok == kExactOk;
  long long lo = has ? incl - k + r.mn : kExact53, hi = has ? incl - k + r.mx : -kExact53;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const long long a = __shfl_xor_sync(0xffffffffu, lo, off), b = __shfl_xor_sync(0xffffffffu, hi, off);
    lo = a < lo ? a : lo;
    hi = b > hi ? b : hi;
  }
  ExactRec o;
  o.K = __shfl_sync(0xffffffffu, incl, 31);
  o.mn = lo;
  o.mx = hi;
  o.e = e;
  const bool zero = __all_sync(0xffffffffu, !in || r.ok == kExactZero);
  const bool good = __all_sync(0xffffffffu, fits) && lo > -kExact53 && hi < kExact53 && o.K > -kExact53 && o.K < kExact53;
  o.ok = zero ? kExactZero : (good ? kExactOk : kExactNone);
  return o;
}

// Running sum of the walk, the same in every lane of its warp. While `in`
// holds, s = S * 2^(e-52) with |S| in [2^52, 2^53): the record applications
// keep it there, so s is formed only when terms are added one by one, or at
// the end.
struct ExactWalk {
  double s;
  long long S;
  int e;
  bool in;
};

__device__ __forceinline__ void exact_walk_flush(ExactWalk &w) {
  if (w.in) {
    w.s = exact_double(w.S, w.e);
    w.in = false;
  }
}

// Applies the records of lanes first .. cnt-1 in order up to the first that
// is not provably the sequential result; returns its lane (cnt: all applied).
__device__ __forceinline__ int exact_walk_run(ExactWalk &w, const ExactRec &r, int first, int cnt) {
  const int lane = threadIdx.x & 31;
  if (!w.in && exact_in_range(exact_exp(w.s))) {
    w.S = exact_int(w.s);
    w.e = exact_exp(w.s);
    w.in = true;
  }
  const bool mine = lane >= first && lane < cnt;
  const bool use = mine && r.ok == kExactOk && w.in && r.e == w.e;
  const long long k = use ? r.K : 0;
  long long incl = k;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += y;
  }
  bool fits = mine && r.ok == kExactZero;
  if (use) {
    const long long LO = (1LL << 52) + 1, HI = kExact53 - 1;
    const long long lo = w.S + (incl - k) + r.mn, hi = w.S + (incl - k) + r.mx;
    fits = w.S > 0 ? (lo >= LO && hi <= HI) : (hi <= -LO && lo >= -HI);
  }
  const unsigned bad = __ballot_sync(0xffffffffu, mine && !fits);
  const int stop = bad ? __ffs(bad) - 1 : cnt;
  const long long sum = __shfl_sync(0xffffffffu, incl, stop > 0 ? stop - 1 : 0);
  if (stop > first && w.in) w.S += sum;
  return stop;
}

// The walk of sum q by one warp through the group records, down into a
// group's chunk records, a chunk's warp records and a warp's 32 terms only
// where a record does not apply. Returns the sum (every lane).
static __device__ __noinline__ double exact_walk(const ExactHdr *H, const double *seq, long long n, long long nch,
                                          int q, long long cap, long long capg, double *term) {
  const int lane = threadIdx.x & 31;
  const long long ng = (nch + kExactGroup - 1) / kExactGroup;
  const ExactRec none{0, 0, 0, 0, kExactNone};
  ExactWalk w{0.0, 0, 0, false};
  for (long long gi = 0; gi < ng; gi += 32) {
    const int nb = (int)((ng - gi) < 32 ? (ng - gi) : 32);
    const ExactRec G = lane < nb ? exact_load(&H->grec[q * capg + gi + lane]) : none;
    for (int k = 0; (k = exact_walk_run(w, G, k, nb)) < nb; ++k) {
      const long long c0 = (gi + k) * kExactGroup;
      const int cs = (int)((nch - c0) < kExactGroup ? (nch - c0) : kExactGroup);
      // both halves of the group's chunk records in flight at once
      const ExactRec C0 = lane < cs ? exact_load(&H->crec[q * cap + c0 + lane]) : none;
      const ExactRec C1 = lane + 32 < cs ? exact_load(&H->crec[q * cap + c0 + 32 + lane]) : none;
      for (int h0 = 0; h0 < cs; h0 += 32) {
        const int hb = (cs - h0) < 32 ? (cs - h0) : 32;
        const ExactRec C = h0 == 0 ? C0 : C1;
        for (int m = 0; (m = exact_walk_run(w, C, m, hb)) < hb; ++m) {
          const long long ch = c0 + h0 + m;
          const long long e0 = ch * kExactChunkThreads;
          const int len = (int)((n - e0) < kExactChunkThreads ? (n - e0) : kExactChunkThreads);
          const int nw = (len + 31) / 32;
          const ExactRec W = lane < nw ? exact_load(&H->wrec[(q * cap + ch) * kExactWarps + lane]) : none;
          __syncwarp();
          for (int e = lane; e < len; e += 32) term[e] = __ldcg(&seq[q * n + e0 + e]);
          __syncwarp();
          for (int v = 0; (v = exact_walk_run(w, W, v, nw)) < nw; ++v) {
            exact_walk_flush(w);
            double sv = w.s;   // every lane the same additions
            const int e1 = (32 * v + 32) < len ? (32 * v + 32) : len;
#pragma unroll 8
            for (int e = 32 * v; e < e1; ++e) sv = __dadd_rn(sv, term[e]);
            w.s = sv;
          }
        }
      }
    }
  }
  exact_walk_flush(w);
  return w.s;
}

// The exact-order reduction. Launch shape: one thread per term, blocks of
// kExactChunkThreads, every thread of every block calls it. Returns true in
// thread 0 of the last block to finish, with out[q] the sequential sum of
// the v[q] in thread order.
template <int NV>
__device__ bool exact_reduce(const double (&v)[NV], double *seq, long long n, unsigned *count,
                             double (&out)[NV]) {
  static_assert(NV <= kExactVals, "exact_reduce: too many sums");
  constexpr int NW = kExactChunkThreads / 32;
  const ExactHdr *H = exact_hdr(seq);
  const long long cap = H->cap_chunks, capg = H->cap_groups;
  const unsigned gen = ld_volatile_u32(&H->gen) & 0x3fffffffu;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const long long b = blockIdx.x;
  const long long nch = gridDim.x;
  const long long p = b * kExactChunkThreads + t;

  __shared__ double s_agg[NV][NW];
  __shared__ double s_hint[NV], s_part[NW];
  __shared__ int s_look[2][NW];
  __shared__ ExactRec s_wr[NV][kExactWarps];
  __shared__ bool s_last;
  __shared__ double s_wterm[kExactVals][kExactChunkThreads];
  __shared__ double s_res[kExactVals];

  // 1. the terms
  double a[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    a[q] = p < n ? v[q] : 0.0;
    if (p < n) seq[q * n + p] = v[q];
  }

  // 2. chunk sums and the look-back for the hint
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double x = a[q];
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    if (lane == 0) s_agg[q][wid] = x;
  }
  __syncthreads();
  // 256 chunks before this one at a time, a thread each, back to the first
  // that has published the sum of all up to it
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    TagWord *W = H->sum + q * cap;
    const unsigned long long t1 = ((unsigned long long)gen << 2) | 1u, t2 = t1 + 1;
    double mine = 0.0;
    for (int w = 0; w < NW; ++w) mine += s_agg[q][w];
    if (t == 0 && b > 0) word_st(W + b, mine, t1);
    double pre = 0.0;
    bool okh = true;
    int polls = 0;
    for (long long top = b - 1; top >= 0;) {
      const long long j = top - t;
      const TagWord x = j >= 0 ? word_ld(W + j) : TagWord{0ull, t2};
      const unsigned incl = __ballot_sync(0xffffffffu, x.tag == t2);
      const unsigned none = __ballot_sync(0xffffffffu, x.tag != t1 && x.tag != t2);
      if (lane == 0) {
        s_look[0][wid] = incl ? 32 * wid + __ffs(incl) - 1 : kExactChunkThreads;
        s_look[1][wid] = none ? 32 * wid + __ffs(none) - 1 : kExactChunkThreads;
      }
      __syncthreads();
      int fi = kExactChunkThreads, fn = kExactChunkThreads;
#pragma unroll
      for (int w = 0; w < NW; ++w) { fi = min(fi, s_look[0][w]); fn = min(fn, s_look[1][w]); }
      double y = t <= fi ? __longlong_as_double((long long)x.v) : 0.0;
      if (fn < fi) {   // a chunk between has not published yet
        __syncthreads();
        if (++polls > kExactPoll) { okh = false; break; }
        continue;
      }
      for (int off = 16; off > 0; off >>= 1) y += __shfl_down_sync(0xffffffffu, y, off);
      if (lane == 0) s_part[wid] = y;
      __syncthreads();
      for (int w = 0; w < NW; ++w) pre += s_part[w];
      if (fi < kExactChunkThreads) break;
      top -= kExactChunkThreads;
      __syncthreads();
    }
    if (t == 0) {
      s_hint[q] = okh ? pre : __longlong_as_double(0x7ff8000000000000LL);
      if (okh) word_st(W + b, pre + mine, t2);
    }
    __syncthreads();
  }

  // 3. one record per warp (32 terms) at the exponent of the approximate sum
  // before it, composed by warp q into sum q's chunk record
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double before = s_hint[q];
    for (int w = 0; w < wid; ++w) before += s_agg[q][w];
    const int e = exact_exp(before);   // zero, infinite and NaN hints fall outside the range
    bool good = exact_in_range(e);
    long long k = 0;
    if (good) {
      const double y = a[q] * exact_pow2(52 - e);
      // finite, |y| <= 2^53 and not half-way between two integers
      good = isfinite(y) && fabs(y) <= 9007199254740992.0 && fabs(y - trunc(y)) != 0.5;
      k = good ? __double2ll_rn(y) : 0;
    }
    const bool zero = __all_sync(0xffffffffu, a[q] == 0.0);
    // inclusive prefix over the warp, its total and range
    for (int off = 1; off < 32; off <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, k, off);
      if (lane >= off) k += y;
    }
    long long mn = k, mx = k;
    for (int off = 16; off > 0; off >>= 1) {
      const long long a2 = __shfl_xor_sync(0xffffffffu, mn, off), b2 = __shfl_xor_sync(0xffffffffu, mx, off);
      mn = a2 < mn ? a2 : mn;
      mx = b2 > mx ? b2 : mx;
    }
    good = __all_sync(0xffffffffu, good) && mn > -kExact53 && mx < kExact53;
    if (lane == 31) {
      const ExactRec W{k, mn, mx, e, zero ? kExactZero : (good ? kExactOk : kExactNone)};
      s_wr[q][wid] = W;
      H->wrec[(q * cap + b) * kExactWarps + wid] = W;
    }
  }
  __syncthreads();
  if (wid < NV) {
    const int q = wid;
    const ExactRec W = s_wr[q][lane < kExactWarps ? lane : 0];
    const ExactRec R = exact_compose(W, kExactWarps, s_wr[q][kExactWarps - 1].e);
    if (lane == 0) { H->crec[q * cap + b] = R; __threadfence(); }
  }

  // 4. group records, by the last chunk of the group
  const long long g = b / kExactGroup;
  const long long g0 = g * kExactGroup;
  const int gsize = (int)((nch - g0) < kExactGroup ? (nch - g0) : kExactGroup);
  __syncthreads();
  if (t == 0) {
    __threadfence();
    unsigned prev = atomicAdd(&H->gcount[g], 1u);
    s_last = (prev == (unsigned)gsize - 1);
  }
  __syncthreads();
  if (!s_last) return false;
  if (wid < NV) {
    __threadfence();
    const int q = wid;
    const ExactRec none{0, 0, 0, 0, kExactNone};
    const int c0 = gsize < 32 ? gsize : 32, c1 = gsize - c0;
    const ExactRec A = lane < c0 ? exact_load(&H->crec[q * cap + g0 + lane]) : none;
    const ExactRec B = lane < c1 ? exact_load(&H->crec[q * cap + g0 + 32 + lane]) : none;
    const int E = __shfl_sync(0xffffffffu, c1 > 0 ? B.e : A.e, (c1 > 0 ? c1 : c0) - 1);
    const ExactRec RA = exact_compose(A, c0, E), RB = exact_compose(B, c1, E);
    const ExactRec R = exact_compose(lane == 0 ? RA : RB, c1 > 0 ? 2 : 1, E);
    if (lane == 0) {
      H->grec[q * capg + g] = R;
      if (q == 0) H->gcount[g] = 0u;
      __threadfence();
    }
  }
  __syncthreads();

  // 5. the last block walks the groups; warp q walks sum q
  if (t == 0) {
    __threadfence();
    unsigned prev = atomicAdd(count, 1u);
    s_last = (prev == (unsigned)((nch + kExactGroup - 1) / kExactGroup) - 1);   // the last group's block
  }
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
  if (wid < NV) {
    const double r = exact_walk(H, seq, n, nch, wid, cap, capg, s_wterm[wid]);
    if (lane == 0) s_res[wid] = r;
  }
  __syncthreads();
  if (t != 0) return false;
#pragma unroll
  for (int q = 0; q < NV; ++q) out[q] = s_res[q];
  ExactHdr *Hw = const_cast<ExactHdr *>(H);
  const unsigned nxt = (gen + 1u) & 0x3fffffffu;
  Hw->gen = nxt ? nxt : 1u;  // generation 0 is the zeroed flags' value
  *count = 0u;
  __threadfence();
  return true;
}

}  // namespace pbg
