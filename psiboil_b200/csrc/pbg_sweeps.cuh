// Lexicographic sweeps as one launch: the incomplete Cholesky factor and its
// triangular solves (Prec::ic0 and ic2) and the Gauss-Seidel sweep of the
// reference-parity solvers. (IC3 also reads the column (i-1, j+1), which
// would make neighbouring tiles wait for each other both ways; it keeps one
// launch per plane, k_ic3_* in pbg_ref_kernels.cu.)
//
// The reference runs them cell after cell in i, j, k order. A cell needs the
// results of a few cells before it, all of which lie on an earlier plane
// h = a (i + j) + k (a = 1 or 2), so any schedule that keeps the planes'
// order gives each cell exactly the values of the sequential sweep, and the
// arithmetic per cell is the reference's, in its order (no contraction).
//
// One block owns the 8 x 8 columns of a tile of the (i, j) plane, a thread
// each, and marches along k: at step t thread (li, lj) is at
// k = t - a (li + lj), so the values it needs from the columns beside it
// were formed in the step before and come from shared memory. Values crossing
// a tile's edge go through global memory as 16-byte (value, epoch) words
// written and read whole: a word is valid when it carries the sweep's epoch,
// so no fence and no reset is needed, and a reader that finds an old word
// polls it (bounded). Blocks take their tiles by ticket in an order in which
// every tile's predecessors come first, so a block only ever waits for blocks
// that are already running.
//
// What bounds it: the chain of a (nx + ny - 2) + nz dependent steps, 0.15 us
// each for IC0, 0.20 us for IC2 and 0.12 us for Gauss-Seidel (shared loads, four
// to six dependent FP64 operations of 9 cycles, the division's correction, a
// barrier), and 2.6 to 2.9 us for each tile edge on the way. One launch per plane,
// the form before this, paid 4.5 us a step. Measured (B200): an IC2 sweep at 64^3
// 109 us (1290 before), CG with IC2 64x56x50, 20 iterations, 52.6 -> 5.9 ms;
// Gauss-Seidel 64x72x60, 10 sweeps, 10.9 -> 1.13 ms. All operands that the
// sweeps own are stored in march order (SweepGeo::off), so that a step reads
// contiguous rows at constant offsets from one pointer.
#pragma once

#include "pbg_common.cuh"
#include "pbg_session.h"
#include "pbg_word.cuh"

namespace pbg {

constexpr int kSweepTile = 8;                            // columns of a tile per direction
constexpr int kSweepCols = kSweepTile * kSweepTile;      // columns of a tile, a thread each
constexpr int kSweepThreads = 2 * kSweepCols + 64;       // two warps for the exchange, two for memory
constexpr int kSweepAhead = 6;                           // steps an operand is loaded early
constexpr int kSweepPoll = 1 << 22;                      // polls of one word before giving up
// rows from which the march-order storage is skewed: below it the skew's
// empty rows would outweigh the cells (2-D grids have one row)
constexpr int kSweepSkewMin = 32;

// weight a = b of the schedule: IC0 (kind 1) and Gauss-Seidel read the
// columns beside a cell at its own k, IC2 (kind 2) also at k + 1
__host__ __device__ constexpr int sweep_a(int kind) { return kind == 2 ? 2 : 1; }

// Tiles of a grid and the march-order storage of a cell array.
struct SweepGeo {
  int nx, ny, nz, ti, tj;
  int wj, cols;     // stored columns of a tile: along j, and in all
  int skew;         // of the storage rows (0 on short columns)
  int rows;         // rows of a tile's storage
  __host__ static SweepGeo make(int nx, int ny, int nz, int a) {
    SweepGeo g;
    g.nx = nx; g.ny = ny; g.nz = nz;
    g.ti = (nx + kSweepTile - 1) / kSweepTile;
    g.tj = (ny + kSweepTile - 1) / kSweepTile;
    const int wi = nx < kSweepTile ? nx : kSweepTile;   // a thin grid stores the columns it has
    g.wj = ny < kSweepTile ? ny : kSweepTile;
    g.cols = wi * g.wj;
    g.skew = nz >= kSweepSkewMin ? a : 0;
    g.rows = nz + g.skew * (wi - 1 + g.wj - 1);
    return g;
  }
  __host__ bool full() const { return cols == kSweepCols; }
  __host__ __device__ int tiles() const { return ti * tj; }
  __host__ __device__ size_t all_rows() const { return (size_t)tiles() * rows; }
  // Storage: a row holds `planes` operands of its cells one after the other.
  // Index of operand 0 of cell (i, j, 0); the cell (i, j, k) is k rows
  // further, the next operand cols further.
  __device__ __forceinline__ size_t off(int i, int j, int planes) const {
    const int li = i % kSweepTile, lj = j % kSweepTile;
    const size_t tile = (size_t)(i / kSweepTile) * tj + j / kSweepTile;
    return (tile * rows + skew * (li + lj)) * planes * cols + li * wj + lj;
  }
  // words of one exchanged value: the last columns along i, then along j, of
  // the tiles that have one after them
  __host__ __device__ size_t words_i() const { return (size_t)(ti - 1) * ny * nz; }
  __host__ __device__ size_t words() const { return words_i() + (size_t)(tj - 1) * nx * nz; }
};

// Shared state of the sweeps of one solver's workspace.
struct SweepSync {
  TagWord *words;             // exchange, SweepGeo::words() per value
  unsigned *ticket;             // [0] next tile, [1] finished tiles (both 0 between launches)
  int *stuck;                   // set when a poll ran out
  unsigned long long epoch;     // of this launch, larger than any before it
};

// Operands of a cell in march order. Incomplete Cholesky: the factor's c, the
// rounded 1 / c for the division by it (NaN where KnownDiv's range does not
// hold), w, s, b, the forward sweep's z, and for IC2 tw and ts.
// Gauss-Seidel: right-hand side, ci, the six couplings and x.
enum : int { kIcC, kIcY, kIcW, kIcS, kIcB, kIcZ, kIcTw, kIcTs };
enum : int { kGsB, kGsCi, kGsW, kGsE, kGsS, kGsN, kGsBt, kGsT, kGsX, kGsPlanes };
__host__ __device__ constexpr int ic_planes(int kind) { return kind == 2 ? 8 : 6; }

}  // namespace pbg
