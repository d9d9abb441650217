// warp_segments.cuh -- sums over runs of particles of the same cell.
//
// The particle store is counting-sorted by cell, so neighbouring particles
// mostly lie in the same cell and add to the same int64 fixed-point tallies.
// Integer addition is associative, so sums formed before the atomics leave
// every tally bit-identical to one atomic per particle.  Two ways:
//
// WarpRuns: the lanes of each run of equal keys add their terms with shuffles
// and the run's last lane issues the atomic; for few tallies (the
// deposition's ten).
//
// RunWalk: a warp takes a range of consecutive particles, 32 at a time.  Each
// lane writes the terms of its particle to shared memory, a row per tally;
// then the lanes change roles: a lane owns a row (or two), walks the
// particles in order, and adds to a register until the cell changes, when
// every lane issues its row's one atomic.  For many tallies (the statistics'
// forty: 231 us by shuffles, 93 this way, for 2M electrons; a row's 32 terms
// are 16 loads and 32 additions for all rows at once, and a run goes on from
// one 32 to the next).  The deposition's ten rows leave two thirds of the
// lanes idle in the walk and took 26 us this way, 17.6 by shuffles, for a
// 20 nm FinFET.
#pragma once

#include <cuda_runtime.h>

namespace mcb200 {

constexpr unsigned kNoRun = 0xffffffffu;  // key of a lane without a live particle

// Words of 8 bytes from one row to the next: a pair of terms lies on 16
// bytes, and eight lanes reading pairs of consecutive rows meet all 32 banks.
constexpr int kRunRow = 34;

// kOwn: rows a lane owns (its second one where kOwn is 2).
template <int kOwn>
struct RunWalk {
  unsigned last = kNoRun;   // key of the last chunk's last particle
  unsigned at = 0, cell = 0;  // where the run being summed adds to
  bool open = false;        // there is one; these three are the same in every lane
  int start = 0;            // its first particle
  long long sum[kOwn] = {};

  // The chunk of 32 particles from `base`: this lane's particle has key
  // `mine` and adds to (my_at, my_cell), the terms of row r lie at terms +
  // r * kRunRow.  flush(at, cell, particles, sum) ends a run.  All 32 lanes
  // call this together, after the terms are written.
  template <class Flush>
  __device__ __forceinline__ void chunk(const long long *terms, const int (&row)[kOwn], unsigned mine, unsigned my_at,
                                        unsigned my_cell, int base, Flush &&flush) {
    unsigned before = __shfl_up_sync(0xffffffffu, mine, 1);
    if ((threadIdx.x & 31u) == 0) before = last;
    last = __shfl_sync(0xffffffffu, mine, 31);
    const unsigned heads = __ballot_sync(0xffffffffu, mine != before);
    const unsigned live = __ballot_sync(0xffffffffu, mine != kNoRun);
    __syncwarp();  // the terms are visible
#pragma unroll 1
    for (int p = 0; p < 32; p += 8) {
      longlong2 v[kOwn][4];
#pragma unroll
      for (int w = 0; w < kOwn; ++w)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          v[w][e] = *reinterpret_cast<const longlong2 *>(terms + row[w] * kRunRow + p + 2 * e);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if ((heads >> (p + e)) & 1u) {  // the same in every lane
          end(base + p + e, flush);
          at = __shfl_sync(0xffffffffu, my_at, p + e);
          cell = __shfl_sync(0xffffffffu, my_cell, p + e);
          open = (live >> (p + e)) & 1u;
          start = base + p + e;
        }
#pragma unroll
        for (int w = 0; w < kOwn; ++w) sum[w] += e & 1 ? v[w][e >> 1].y : v[w][e >> 1].x;
      }
    }
    __syncwarp();  // the terms have been read
  }
  // Ends the run before particle p (after the last chunk: one past it).
  template <class Flush>
  __device__ __forceinline__ void end(int p, Flush &&flush) {
    if (open) flush(at, cell, p - start, sum);
#pragma unroll
    for (int w = 0; w < kOwn; ++w) sum[w] = 0;
  }
};

// A chunk's sums by shuffles: each lane keeps its particle's terms.
struct WarpRuns {
  unsigned lane, head;  // this lane, the first lane of its run
  unsigned span;        // longest run in the warp
  bool tail;            // last lane of its run: issues the run's atomics

  // All 32 lanes must call this (and sum) together.
  __device__ __forceinline__ explicit WarpRuns(unsigned key) {
    lane = threadIdx.x & 31u;
    const unsigned prev = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned next = __shfl_down_sync(0xffffffffu, key, 1);
    const bool is_head = lane == 0 || prev != key;
    tail = lane == 31 || next != key;
    const unsigned heads = __ballot_sync(0xffffffffu, is_head);
    head = 31u - __clz(heads & (0xffffffffu >> (31u - lane)));
    span = __reduce_max_sync(0xffffffffu, lane - head + 1u);
  }
  // Inclusive sum over the run up to this lane; the tail lane holds the run's total.
  __device__ __forceinline__ long long sum(long long v) const {
    for (unsigned o = 1; o < span; o <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= head + o) v += u;
    }
    return v;
  }
};

}  // namespace mcb200
