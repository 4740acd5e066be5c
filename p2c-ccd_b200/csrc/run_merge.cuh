// run_merge.cuh — merging eight sorted runs into one: the place of an entry is
// its place in its own run plus the entries before it in the others.
#pragma once

#include "p2c_internal.cuh"

namespace p2c {

constexpr unsigned kMergeRuns = 8;

// Rounds of merging kMergeRuns runs that make one run of up to longest entries
// from runs of tile.
__host__ __device__ inline int merge_rounds(unsigned long long tile, unsigned long long longest) {
  int n = 0;
  for (unsigned long long width = tile; width < longest; width *= kMergeRuns) ++n;
  return n;
}
// Width of the runs that a round merges (rounds from 0; below 2^32 in a round
// that has something to merge).
__device__ __forceinline__ unsigned merge_width(unsigned tile, int round) {
  static_assert(kMergeRuns == 8, "width by shifts of three");
  return tile << (3 * round);
}

// Entries before (key, idx) in the runs, of n[k] <= width entries each (0 for
// the entry's own).  precedes(k, p, key, idx): entry p of run k comes before.
// together (the same in all lanes of the warp): the lanes hold consecutive
// entries of one run, so the first and the last one's places bound everyone's,
// and the warp searches each run for those two, a lane per run and end, before
// every lane searches the few entries between.
template <class Precedes>
__device__ __forceinline__ unsigned entries_before(unsigned width, const unsigned (&n)[kMergeRuns],
                                                   unsigned long long key, unsigned idx, bool together,
                                                   Precedes precedes) {
  unsigned lo[kMergeRuns], hi[kMergeRuns], most = 0u;
  if (together) {
    const int lane = threadIdx.x & 31, src = lane < (int)kMergeRuns ? 0 : 31;
    const unsigned run = (unsigned)lane & (kMergeRuns - 1u), end_idx = __shfl_sync(0xffffffffu, idx, src);
    const unsigned long long end_key = __shfl_sync(0xffffffffu, key, src);
    unsigned len = 0u, at = 0u;
#pragma unroll
    for (unsigned k = 0; k < kMergeRuns; ++k) len = run == k ? n[k] : len;
    for (unsigned step = width; step > 0u; step >>= 1)
      if (at + step <= len && precedes(run, at + step - 1u, end_key, end_idx)) at += step;
#pragma unroll
    for (unsigned k = 0; k < kMergeRuns; ++k) {
      lo[k] = __shfl_sync(0xffffffffu, at, (int)k);
      hi[k] = __shfl_sync(0xffffffffu, at, (int)(kMergeRuns + k));
      most = max(most, hi[k] - lo[k]);
    }
  } else {
#pragma unroll
    for (unsigned k = 0; k < kMergeRuns; ++k) {
      lo[k] = 0u;
      hi[k] = n[k];
      most = max(most, n[k]);
    }
  }
  for (unsigned step = most != 0u ? 1u << (31 - __clz((int)most)) : 0u; step > 0u; step >>= 1) {
#pragma unroll
    for (unsigned k = 0; k < kMergeRuns; ++k)
      if (lo[k] + step <= hi[k] && precedes(k, lo[k] + step - 1u, key, idx)) lo[k] += step;
  }
  unsigned sum = 0u;
#pragma unroll
  for (unsigned k = 0; k < kMergeRuns; ++k) sum += lo[k];
  return sum;
}

}  // namespace p2c
