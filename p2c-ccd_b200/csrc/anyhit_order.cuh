// anyhit_order.cuh — the proposals of every candidate group: its K best
// candidates by (score key, index), and one list of them rank by rank.
//
// Only the K best of a group have a rank that anything reads, so nothing is
// sorted but them.  Six launches over device-side counts:
//   (caller)  group and key per candidate, group sizes; the first candidate
//             of a group gives the group its ordinal
//   range     smallest and largest key of each group larger than K
//   bins      256 or 2048 bins over that range, per group
//   plan      the first bin edge with K candidates below it, room for what
//             lies below it, and how many groups reach each rank
//   gather    keys and indices of the candidates below their group's edge
//   pick      one block per group: narrows the set further while it does not
//             fit shared memory (radix selection on key, then index), orders
//             it there, writes ranks and list entries
//
// Bound by reading 12 bytes a candidate three times.  B200, edge-edge
// candidates with K = 4096: 27 bodies (7.6 M in a buffer of 10.7 M, 54 groups)
// 236 us from candidate to list, against 1690 for the sorts this stands in for
// (64-bit score keys, groups, ranks: 12 radix passes over the buffer); a
// 624k-triangle cloth (2.5 M of 3.5 M, 2 groups) 270 against 632.
// K is at most kPickRanks here: a group's proposals have to fit one block.
// Larger K (no default asks for it) keeps the full sorts.
#pragma once

#include <cub/block/block_scan.cuh>

#include "certify_core.cuh"
#include "certify_engine.cuh"
#include "p2c_internal.cuh"

namespace p2c {

constexpr unsigned kPickRanks = 4096;    // largest K of this path
constexpr unsigned kPickEntries = 8192;  // candidates one block sorts
constexpr int kPickThreads = 1024;
constexpr int kPickDigits = 2048;  // counters of one narrowing round, buckets of the final order
constexpr unsigned kPickBucket = 64;  // longest bucket that is ordered by counting
constexpr int kOrderThreads = 256;
constexpr int kOrderSpan = 4 * kOrderThreads;  // consecutive candidates a block takes at once
constexpr int kOrderBinsMax = 2048;
constexpr unsigned kNoRank = 0xffffffffu;

struct OrderCounters {
  unsigned n_groups;  // groups with candidates (ordinals given out)
  unsigned entries;   // gathered entries
  unsigned plan_blocks;
  unsigned pad;
};

struct OrderSpace {
  const unsigned* grp = nullptr;                // per candidate; >= groups: not a candidate
  const unsigned long long* key = nullptr;      // ascending order of proposals
  unsigned* rank = nullptr;                     // kNoRank unless a proposal (set by the caller)
  unsigned* g_size = nullptr;                   // per group
  unsigned* g_ord = nullptr;                    // per group with candidates: its ordinal
  // by ordinal
  unsigned* o_group = nullptr;
  unsigned long long* o_lo = nullptr;
  unsigned long long* o_hi = nullptr;
  unsigned long long* o_edge = nullptr;  // largest key gathered
  unsigned* o_start = nullptr;
  unsigned* o_fill = nullptr;
  unsigned* hist = nullptr;  // a bin table per ordinal; groups past the last table are gathered whole
  unsigned hist_words = 0;
  int bin_bits = 0;  // set by launch_order, with slots = hist_words >> bin_bits
  unsigned slots = 0;
  unsigned long long* ent_key = nullptr;
  unsigned* ent_idx = nullptr;
  unsigned* list = nullptr;      // proposals, rank by rank
  unsigned* rank_pos = nullptr;  // per family kPickRanks + 1: groups of each size, then list positions
  unsigned long long* n_top = nullptr;  // per family: proposals
  OrderCounters* ctr = nullptr;
  unsigned groups = 0;
  unsigned K = 0;
  int families = 1;
  long long cap = 0;
  long long cap_first = 0;  // candidates of the first family come before this index
};

inline size_t order_ordinals(long long cap, long long groups) {
  return (size_t)std::max(1ll, std::min(cap, groups));
}

// Arrays by ordinal, rank counters and the counter block, carved by take(bytes).
template <class Take>
void carve_order(OrderSpace& o, long long cap, long long groups, int families, Take take) {
  const size_t m = order_ordinals(cap, groups);
  o.g_ord = static_cast<unsigned*>(take((size_t)std::max(groups, 1ll) * 4));
  o.o_group = static_cast<unsigned*>(take(m * 4));
  o.o_lo = static_cast<unsigned long long*>(take(m * 8));
  o.o_hi = static_cast<unsigned long long*>(take(m * 8));
  o.o_edge = static_cast<unsigned long long*>(take(m * 8));
  o.o_start = static_cast<unsigned*>(take(m * 4));
  o.o_fill = static_cast<unsigned*>(take(m * 4));
  o.rank_pos = static_cast<unsigned*>(take((size_t)families * (kPickRanks + 1) * 4));
  o.ctr = static_cast<OrderCounters*>(take(sizeof(OrderCounters)));
  o.families = families;
  o.cap = cap;
  o.groups = (unsigned)groups;
}

// What the ordering expects zeroed, besides g_size (thread i of stride).
__device__ __forceinline__ void order_reset(const OrderSpace& o, long long i, long long stride) {
  for (long long r = i; r < (long long)o.families * (kPickRanks + 1); r += stride) o.rank_pos[r] = 0u;
  if (i == 0) *o.ctr = OrderCounters{};
}

// Counts candidates of one block into their groups: one atomic for the group
// of the block's first candidate, one per warp and group otherwise.  The
// first count of a group hands out its ordinal.
__device__ __forceinline__ void order_count(const OrderSpace& o, unsigned g, unsigned n) {
  if (atomicAdd(o.g_size + g, n) == 0u) {
    const unsigned k = atomicAdd(&o.ctr->n_groups, 1u);
    o.o_group[k] = g;
    o.g_ord[g] = k;
    o.o_lo[k] = ~0ull;
    o.o_hi[k] = 0ull;
    o.o_fill[k] = 0u;
  }
}

// Block-wide counting of a span of candidates; every thread of the block
// calls add() the same number of times and finish() once.
struct SpanCount {
  unsigned main, mine;
  __device__ __forceinline__ SpanCount(unsigned main_group) : main(main_group), mine(0u) {}
  __device__ __forceinline__ void add(const OrderSpace& o, unsigned g) {
    const bool in = g < o.groups;
    if (in && g == main) ++mine;
    const bool other = in && g != main;
    const unsigned m = __match_any_sync(0xffffffffu, other ? g : kNoRank);
    if (other && (threadIdx.x & 31) == __ffs((int)m) - 1) order_count(o, g, (unsigned)__popc(m));
  }
  __device__ __forceinline__ void finish(const OrderSpace& o, unsigned* shared_sum) {  // zeroed before
    const unsigned w = __reduce_add_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && w) atomicAdd(shared_sum, w);
    __syncthreads();
    if (threadIdx.x == 0 && *shared_sum) order_count(o, main, *shared_sum);
  }
};

namespace {

__device__ __forceinline__ unsigned warp_inclusive_sum(unsigned v, int lane) {
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const unsigned up = __shfl_up_sync(0xffffffffu, v, s);
    if (lane >= s) v += up;
  }
  return v;
}

// The consecutive candidates of a block: whole spans, so that a block meets
// few groups and writes what it has gathered on one group only once.
struct BlockRange {
  long long begin, end;
  __device__ __forceinline__ BlockRange(long long n) {
    const long long spans = (n + kOrderSpan - 1) / kOrderSpan, each = (spans + gridDim.x - 1) / gridDim.x;
    begin = min(n, blockIdx.x * each * kOrderSpan);
    end = min(n, begin + each * kOrderSpan);
  }
};

__global__ void __launch_bounds__(kOrderThreads) order_range_kernel(OrderSpace o, const unsigned long long* count) {
  __shared__ unsigned long long lo, hi;
  const long long n = count == nullptr ? o.cap : min((long long)*count, o.cap);
  const long long words = (long long)min(o.slots, o.ctr->n_groups) << o.bin_bits;
  for (long long i = (long long)blockIdx.x * kOrderThreads + threadIdx.x; i < words;
       i += (long long)gridDim.x * kOrderThreads)
    o.hist[i] = 0u;
  const BlockRange r(n);
  unsigned main = o.groups;
  unsigned long long mlo = ~0ull, mhi = 0ull;
  auto flush = [&]() {
    __syncthreads();
    if (threadIdx.x == 0) {
      lo = ~0ull;
      hi = 0ull;
    }
    __syncthreads();
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      mlo = min(mlo, __shfl_xor_sync(0xffffffffu, mlo, s));
      mhi = max(mhi, __shfl_xor_sync(0xffffffffu, mhi, s));
    }
    if ((threadIdx.x & 31) == 0 && mlo <= mhi) {
      atomicMin(&lo, mlo);
      atomicMax(&hi, mhi);
    }
    __syncthreads();
    if (threadIdx.x == 0 && lo <= hi) {
      const unsigned d = o.g_ord[main];
      if (lo < volatile_load(o.o_lo + d)) atomicMin(o.o_lo + d, lo);
      if (hi > volatile_load(o.o_hi + d)) atomicMax(o.o_hi + d, hi);
    }
    mlo = ~0ull;
    mhi = 0ull;
  };
  for (long long base = r.begin; base < r.end; base += kOrderSpan) {
    const unsigned first = o.grp[base];
    if (first != main) {
      if (main < o.groups) flush();
      main = first;
    }
#pragma unroll
    for (int i = 0; i < kOrderSpan / kOrderThreads; ++i) {
      const long long c = base + i * kOrderThreads + threadIdx.x;
      if (c >= r.end) continue;
      const unsigned g = o.grp[c];
      const unsigned long long k = o.key[c];
      if (g >= o.groups || o.g_size[g] <= o.K) continue;
      if (g == main) {
        mlo = min(mlo, k);
        mhi = max(mhi, k);
      } else {
        const unsigned d = o.g_ord[g];
        if (k < volatile_load(o.o_lo + d)) atomicMin(o.o_lo + d, k);
        if (k > volatile_load(o.o_hi + d)) atomicMax(o.o_hi + d, k);
      }
    }
  }
  if (main < o.groups) flush();
}

__device__ __forceinline__ int bin_shift(unsigned long long lo, unsigned long long hi, int bits) {
  return max(0, 64 - __clzll((long long)(hi - lo)) - bits);  // (hi - lo) >> shift < 1 << bits
}

__global__ void __launch_bounds__(kOrderThreads) order_bins_kernel(OrderSpace o, const unsigned long long* count) {
  __shared__ unsigned bins[kOrderBinsMax];
  const int n_bins = 1 << o.bin_bits;
  const long long n = count == nullptr ? o.cap : min((long long)*count, o.cap);
  const BlockRange r(n);
  for (int b = threadIdx.x; b < n_bins; b += kOrderThreads) bins[b] = 0u;
  __syncthreads();
  unsigned main = o.groups, main_ord = kNoRank;  // kNoRank: the group has no bins
  unsigned long long mlo = 0ull;
  int mshift = 0;
  auto flush = [&]() {
    __syncthreads();
    for (int b = threadIdx.x; b < n_bins; b += kOrderThreads) {
      if (bins[b]) atomicAdd(o.hist + ((size_t)main_ord << o.bin_bits) + b, bins[b]);
      bins[b] = 0u;
    }
    __syncthreads();
  };
  for (long long base = r.begin; base < r.end; base += kOrderSpan) {
    const unsigned first = o.grp[base];
    if (first != main) {
      if (main_ord != kNoRank) flush();
      main = first;
      main_ord = kNoRank;
      if (main < o.groups && o.g_size[main] > o.K && o.g_ord[main] < o.slots) {
        main_ord = o.g_ord[main];
        mlo = o.o_lo[main_ord];
        mshift = bin_shift(mlo, o.o_hi[main_ord], o.bin_bits);
      }
    }
#pragma unroll
    for (int i = 0; i < kOrderSpan / kOrderThreads; ++i) {  // whole warps: match below
      const long long c = base + i * kOrderThreads + threadIdx.x;
      const unsigned g = c < r.end ? o.grp[c] : o.groups;
      const unsigned long long k = c < r.end ? o.key[c] : 0ull;
      unsigned slot = kNoRank;
      if (g == main) {
        if (main_ord != kNoRank) atomicAdd(&bins[(k - mlo) >> mshift], 1u);
      } else if (g < o.groups && o.g_size[g] > o.K) {
        const unsigned d = o.g_ord[g];
        if (d < o.slots) {
          const unsigned long long lo = o.o_lo[d];
          slot = (d << o.bin_bits) + (unsigned)((k - lo) >> bin_shift(lo, o.o_hi[d], o.bin_bits));
        }
      }
      if (__any_sync(0xffffffffu, slot != kNoRank)) {
        const unsigned m = __match_any_sync(0xffffffffu, slot);
        if (slot != kNoRank && (threadIdx.x & 31) == __ffs((int)m) - 1) atomicAdd(o.hist + slot, (unsigned)__popc(m));
      }
    }
  }
  if (main_ord != kNoRank) flush();
}

// One warp per group; the last block turns the counts of groups per size into
// the list position of each rank (family after family).
__global__ void __launch_bounds__(kOrderThreads) order_plan_kernel(OrderSpace o, const unsigned* first_group_of_family2) {
  const int lane = threadIdx.x & 31;
  const unsigned n = o.ctr->n_groups;
  const unsigned warps = gridDim.x * (kOrderThreads / 32);
  for (unsigned d = blockIdx.x * (kOrderThreads / 32) + (threadIdx.x >> 5); d < n; d += warps) {
    const unsigned g = o.o_group[d], size = o.g_size[g];
    unsigned kept = size;
    unsigned long long edge = ~0ull;
    if (size > o.K && d < o.slots) {
      const unsigned long long lo = o.o_lo[d], hi = o.o_hi[d];
      const int shift = bin_shift(lo, hi, o.bin_bits);
      // each lane sums consecutive bins, the warp finds the lane that reaches K, then its bins
      const int each = 1 << (o.bin_bits - 5);
      const unsigned* bins = o.hist + ((size_t)d << o.bin_bits);
      unsigned sum = 0u;
#pragma unroll 8
      for (int b = 0; b < each; ++b) sum += bins[lane * each + b];
      const unsigned incl = warp_inclusive_sum(sum, lane);
      const int who = __ffs((int)__ballot_sync(0xffffffffu, incl >= o.K)) - 1;  // the group is larger than K
      unsigned below = __shfl_sync(0xffffffffu, incl - sum, who);
      for (int b0 = who * each; b0 < (who + 1) * each; b0 += 32) {
        const bool in = b0 + lane < (who + 1) * each;
        const unsigned at_incl = warp_inclusive_sum(in ? bins[b0 + lane] : 0u, lane);
        const unsigned m = __ballot_sync(0xffffffffu, below + at_incl >= o.K);
        if (m) {
          const int at = __ffs((int)m) - 1;
          kept = below + __shfl_sync(0xffffffffu, at_incl, at);
          // the bin's last key; the top bin may reach past the largest 64-bit key
          const unsigned long long width = ((unsigned long long)(b0 + at) << shift) | ((1ull << shift) - 1ull);
          edge = width >= hi - lo ? hi : lo + width;
          break;
        }
        below += __shfl_sync(0xffffffffu, at_incl, 31);
      }
    }
    if (lane == 0) {
      o.o_edge[d] = edge;
      o.o_start[d] = atomicAdd(&o.ctr->entries, kept);
      const unsigned f = o.families == 2 && g >= *first_group_of_family2 ? 1u : 0u;
      atomicAdd(o.rank_pos + f * (kPickRanks + 1) + min(size, o.K), 1u);
    }
  }
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&o.ctr->plan_blocks, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // groups with more than r proposals = the groups in front of the list entries of rank r
  constexpr int kEach = (int)kPickRanks / kOrderThreads;
  using Scan = cub::BlockScan<unsigned, kOrderThreads>;
  __shared__ typename Scan::TempStorage tmp;
  for (int f = 0; f < o.families; ++f) {
    unsigned* at = o.rank_pos + f * (kPickRanks + 1);
    unsigned v[kEach], total;
    // reversed: item i of the scan is size kPickRanks - i
#pragma unroll
    for (int i = 0; i < kEach; ++i) v[i] = __ldcg(at + (kPickRanks - (threadIdx.x * kEach + i)));
    Scan(tmp).InclusiveSum(v, v, total);  // v: groups of at least that size
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kEach; ++i) at[kPickRanks - 1 - (threadIdx.x * kEach + i)] = v[i];  // groups past rank r
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kEach; ++i) v[i] = at[threadIdx.x * kEach + i];
    Scan(tmp).ExclusiveSum(v, v, total);
    __syncthreads();
    const unsigned base = f == 0 ? 0u : (unsigned)o.cap_first;
#pragma unroll
    for (int i = 0; i < kEach; ++i) at[threadIdx.x * kEach + i] = base + v[i];
    if (threadIdx.x == 0) o.n_top[f] = total;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kOrderThreads) order_gather_kernel(OrderSpace o, const unsigned long long* count) {
  __shared__ unsigned warp_sum[kOrderThreads / 32], block_at;
  const long long n = count == nullptr ? o.cap : min((long long)*count, o.cap);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (long long base = (long long)blockIdx.x * kOrderSpan; base < n; base += (long long)gridDim.x * kOrderSpan) {
    const unsigned main = o.grp[base];
    const unsigned main_ord = main < o.groups ? o.g_ord[main] : kNoRank;
    const unsigned long long main_edge = main_ord != kNoRank ? o.o_edge[main_ord] : 0ull;
    const unsigned main_start = main_ord != kNoRank ? o.o_start[main_ord] : 0u;
    unsigned keep = 0u;  // bit i: candidate i of this thread is an entry of the main group
    unsigned long long key[kOrderSpan / kOrderThreads];
#pragma unroll
    for (int i = 0; i < kOrderSpan / kOrderThreads; ++i) {
      const long long c = base + i * kOrderThreads + threadIdx.x;
      const unsigned g = c < n ? o.grp[c] : o.groups;
      key[i] = g < o.groups ? o.key[c] : 0ull;
      bool other = false;
      unsigned d = kNoRank;
      if (g < o.groups) {
        if (g == main) {
          keep |= key[i] <= main_edge ? 1u << i : 0u;
        } else {
          d = o.g_ord[g];
          other = key[i] <= o.o_edge[d];
        }
      }
      if (__any_sync(0xffffffffu, other)) {
        const unsigned m = __match_any_sync(0xffffffffu, other ? d : kNoRank);
        unsigned at = 0u;
        const int leader = __ffs((int)m) - 1;
        if (other && lane == leader) at = atomicAdd(o.o_fill + d, (unsigned)__popc(m));
        at = __shfl_sync(0xffffffffu, at, leader);
        if (other) {
          const unsigned e = o.o_start[d] + at + (unsigned)__popc(m & ((1u << lane) - 1u));
          o.ent_key[e] = key[i];
          o.ent_idx[e] = (unsigned)c;
        }
      }
    }
    // the main group's entries: one atomic a block
    const unsigned mine = (unsigned)__popc(keep);
    const unsigned incl = warp_inclusive_sum(mine, lane);
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned sum = 0u;
      for (int k = 0; k < kOrderThreads / 32; ++k) {
        const unsigned x = warp_sum[k];
        warp_sum[k] = sum;
        sum += x;
      }
      block_at = sum ? atomicAdd(o.o_fill + main_ord, sum) : 0u;
    }
    __syncthreads();
    unsigned e = main_start + block_at + warp_sum[w] + incl - mine;
#pragma unroll
    for (int i = 0; i < kOrderSpan / kOrderThreads; ++i)
      if (keep >> i & 1u) {
        o.ent_key[e] = key[i];
        o.ent_idx[e] = (unsigned)(base + i * kOrderThreads + threadIdx.x);
        ++e;
      }
    __syncthreads();
  }
}

struct PickShared {
  unsigned long long key[kPickEntries];
  unsigned idx[kPickEntries];
  unsigned digit[kPickDigits];       // counters, then the end of each bucket
  unsigned short place[kPickEntries];  // entries bucket by bucket
  unsigned warp_sum[kPickThreads / 32];
  unsigned long long lo, hi;
  unsigned n, found, below, longest;
};

// Narrows [lo, lo + 2^bits) of value(e) over the entries in(e) until the
// entries up to its end number at least K and at most kPickEntries, or the
// range is one value.  Returns true in the first case, with the last value in
// `last`; otherwise the value is `lo` and sh.below the entries before it.
template <class In, class Value>
__device__ __forceinline__ bool narrow(PickShared& sh, unsigned m, unsigned K, unsigned long long lo, int bits, In in,
                                       Value value, unsigned long long& last) {
  while (true) {
    const int take = min(bits, 11), shift = bits - take;
    for (int b = threadIdx.x; b < kPickDigits; b += kPickThreads) sh.digit[b] = 0u;
    __syncthreads();
    for (unsigned e = threadIdx.x; e < m; e += kPickThreads) {
      if (!in(e)) continue;
      const unsigned long long v = value(e);
      if (v < lo) continue;
      const unsigned long long r = (v - lo) >> shift;
      if (r < (1ull << take)) atomicAdd(&sh.digit[r], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      unsigned below = sh.below;
      for (int b0 = 0; b0 < (1 << take); b0 += 32) {
        const unsigned c = b0 + (int)threadIdx.x < (1 << take) ? sh.digit[b0 + threadIdx.x] : 0u;
        const unsigned incl = warp_inclusive_sum(c, (int)threadIdx.x);
        const unsigned f = __ballot_sync(0xffffffffu, below + incl >= K);
        if (f) {
          const int at = __ffs((int)f) - 1;
          if ((int)threadIdx.x == at) {
            sh.found = (unsigned)(b0 + at);
            sh.n = below + incl;
            sh.below = below + incl - c;
          }
          break;
        }
        below += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    __syncthreads();
    const unsigned long long at = (unsigned long long)sh.found << shift;
    const bool fits = sh.n <= kPickEntries;
    __syncthreads();
    if (fits) {
      const unsigned long long end = at + ((1ull << shift) - 1ull);
      last = end > ~0ull - lo ? ~0ull : lo + end;
      return true;
    }
    lo += at;
    bits = shift;
    if (bits == 0) {
      last = lo;
      return false;
    }
  }
}

// One block per group (one warp up to 32 entries): the K smallest of its
// entries by (key, index), in order.  Kept entries go to buckets of equal key
// ranges and count the smaller ones of their bucket: 2048 buckets hold two
// entries each where keys differ.  Many ties make long buckets; then a bitonic
// sort orders all of them.  27 bodies: 33 us; the bitonic sort alone, and 256
// bins before it, 303.
__global__ void __launch_bounds__(kPickThreads) order_pick_kernel(OrderSpace o, const unsigned* first_group_of_family2) {
  extern __shared__ __align__(16) unsigned char pick_raw[];
  PickShared& sh = *reinterpret_cast<PickShared*>(pick_raw);
  const unsigned n_groups = o.ctr->n_groups;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned split = o.families == 2 ? *first_group_of_family2 : o.groups;
  for (unsigned d = blockIdx.x * (kPickThreads / 32) + w; d < n_groups; d += gridDim.x * (kPickThreads / 32)) {
    const unsigned m = o.o_fill[d];
    if (m > 32u) continue;
    const unsigned g = o.o_group[d], want = min(o.g_size[g], o.K), at = o.o_start[d] + lane;
    const unsigned long long k = (unsigned)lane < m ? o.ent_key[at] : ~0ull;
    const unsigned c = (unsigned)lane < m ? o.ent_idx[at] : 0xffffffffu;
    unsigned r = 0u;
#pragma unroll
    for (int s = 0; s < 32; ++s) {
      const unsigned long long ok = __shfl_sync(0xffffffffu, k, s);
      const unsigned oc = __shfl_sync(0xffffffffu, c, s);
      r += ok < k || (ok == k && oc < c) ? 1u : 0u;
    }
    if ((unsigned)lane < m && r < want) {
      o.rank[c] = r;
      o.list[atomicAdd(o.rank_pos + (g >= split ? kPickRanks + 1 : 0u) + r, 1u)] = c;
    }
  }
  for (unsigned d = blockIdx.x; d < n_groups; d += gridDim.x) {
    const unsigned g = o.o_group[d], m = o.o_fill[d], start = o.o_start[d];
    if (m <= 32u) continue;
    const unsigned want = min(o.g_size[g], o.K);
    unsigned* pos = o.rank_pos + (g >= split ? kPickRanks + 1 : 0u);
    const unsigned long long* ek = o.ent_key + start;
    const unsigned* ei = o.ent_idx + start;
    unsigned long long key_last = ~0ull, idx_last = 0xffffffffull;  // kept: key < key_last, or equal and idx <= idx_last
    if (m > kPickEntries) {
      if (threadIdx.x == 0) sh.below = 0u;
      const unsigned long long lo = o.o_lo[d], hi = min(o.o_hi[d], o.o_edge[d]);
      const int bits = hi == lo ? 0 : 64 - __clzll((long long)(hi - lo));
      if (!narrow(sh, m, want, lo, bits, [](unsigned) { return true; }, [&](unsigned e) { return ek[e]; }, key_last)) {
        const unsigned long long tie = key_last;
        narrow(sh, m, want, 0ull, 32, [&](unsigned e) { return ek[e] == tie; },
               [&](unsigned e) { return (unsigned long long)ei[e]; }, idx_last);
      }
    }
    if (threadIdx.x == 0) {
      sh.n = 0u;
      sh.longest = 0u;
      sh.lo = ~0ull;
      sh.hi = 0ull;
    }
    for (int b = threadIdx.x; b < kPickDigits; b += kPickThreads) sh.digit[b] = 0u;
    __syncthreads();
    unsigned long long klo = ~0ull, khi = 0ull;
    for (unsigned e0 = 0; e0 < m; e0 += kPickThreads) {
      const unsigned e = e0 + threadIdx.x;
      const unsigned long long k = e < m ? ek[e] : ~0ull;
      const unsigned i = e < m ? ei[e] : 0u;
      const bool keep = e < m && (k < key_last || (k == key_last && i <= idx_last));
      const unsigned mask = __ballot_sync(0xffffffffu, keep);
      unsigned at = 0u;
      if (lane == 0 && mask) at = atomicAdd(&sh.n, (unsigned)__popc(mask));
      at = __shfl_sync(0xffffffffu, at, 0) + (unsigned)__popc(mask & ((1u << lane) - 1u));
      if (keep) {
        sh.key[at] = k;
        sh.idx[at] = i;
        klo = min(klo, k);
        khi = max(khi, k);
      }
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      klo = min(klo, __shfl_xor_sync(0xffffffffu, klo, s));
      khi = max(khi, __shfl_xor_sync(0xffffffffu, khi, s));
    }
    if (lane == 0) {
      atomicMin(&sh.lo, klo);
      atomicMax(&sh.hi, khi);
    }
    __syncthreads();
    const unsigned cnt = sh.n;
    const unsigned long long lo = sh.lo;
    const int shift = bin_shift(lo, sh.hi, 11);
    for (unsigned e = threadIdx.x; e < cnt; e += kPickThreads) atomicAdd(&sh.digit[(sh.key[e] - lo) >> shift], 1u);
    __syncthreads();
    constexpr int kEach = kPickDigits / kPickThreads;
    unsigned c[kEach], sum = 0u, longest = 0u;
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
      c[k] = sh.digit[threadIdx.x * kEach + k];
      sum += c[k];
      longest = max(longest, c[k]);
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    const unsigned incl = warp_inclusive_sum(sum, lane);
    if (lane == 31) sh.warp_sum[w] = incl;
    if (lane == 0) atomicMax(&sh.longest, longest);
    __syncthreads();
    if (sh.longest <= kPickBucket) {
      unsigned at = incl - sum;
      for (int k = 0; k < w; ++k) at += sh.warp_sum[k];
#pragma unroll
      for (int k = 0; k < kEach; ++k) {
        sh.digit[threadIdx.x * kEach + k] = at;
        at += c[k];
      }
      __syncthreads();
      for (unsigned e = threadIdx.x; e < cnt; e += kPickThreads)
        sh.place[atomicAdd(&sh.digit[(sh.key[e] - lo) >> shift], 1u)] = (unsigned short)e;
      __syncthreads();
      for (unsigned p = threadIdx.x; p < cnt; p += kPickThreads) {
        const unsigned e = sh.place[p];
        const unsigned long long k = sh.key[e];
        const unsigned i = sh.idx[e], b = (unsigned)((k - lo) >> shift);
        const unsigned first = b == 0u ? 0u : sh.digit[b - 1], end = sh.digit[b];
        if (first >= want) continue;
        unsigned r = first;
        for (unsigned q = first; q < end; ++q) {
          const unsigned f = sh.place[q];
          const unsigned long long fk = sh.key[f];
          r += fk < k || (fk == k && sh.idx[f] < i) ? 1u : 0u;
        }
        if (r < want) {
          o.rank[i] = r;
          o.list[atomicAdd(pos + r, 1u)] = i;
        }
      }
    } else {
      unsigned size = 2u;
      while (size < cnt) size <<= 1;
      for (unsigned e = cnt + threadIdx.x; e < size; e += kPickThreads) {
        sh.key[e] = ~0ull;
        sh.idx[e] = 0xffffffffu;
      }
      __syncthreads();
      // 32 consecutive compare pairs span 64 entries, so steps of at most 32
      // stay within one warp's entries
      for (unsigned k = 2; k <= size; k <<= 1) {
        for (unsigned j = k >> 1; j > 0; j >>= 1) {
          for (unsigned p = threadIdx.x; p < size / 2; p += kPickThreads) {
            const unsigned a = 2u * p - (p & (j - 1u)), b = a + j;
            const unsigned long long ka = sh.key[a], kb = sh.key[b];
            const unsigned ia = sh.idx[a], ib = sh.idx[b];
            const bool greater = ka > kb || (ka == kb && ia > ib);
            if (greater == ((a & k) == 0u)) {
              sh.key[a] = kb;
              sh.key[b] = ka;
              sh.idx[a] = ib;
              sh.idx[b] = ia;
            }
          }
          if (j > 32u) __syncthreads();
          else __syncwarp();
        }
        __syncthreads();
      }
      for (unsigned r = threadIdx.x; r < want; r += kPickThreads) {
        const unsigned i = sh.idx[r];
        o.rank[i] = r;
        o.list[atomicAdd(pos + r, 1u)] = i;
      }
    }
    __syncthreads();
  }
}

}  // namespace

// Ranks and list of the proposals (K in [1, kPickRanks]).  The caller has
// filled grp, key, rank = kNoRank, and counted the groups by SpanCount, with
// rank_pos and the counters zeroed before.  first_group_of_family2: device
// word, read with two families only.
inline int launch_order(OrderSpace o, const unsigned long long* count, const unsigned* first_group_of_family2,
                        cudaStream_t s) {
  DeviceInfo info;
  if (int rc = current_device_info(&info)) return rc;
  // At most cap / (K + 1) groups are larger than K, so a table of at most K
  // bins fits for each of them; 2048 bins keep what is gathered close to K
  // (256: 75k of 1.9 M candidates of one group for K = 4096, 2048: 13k).
  o.bin_bits = o.K >= 2048u ? 11 : 8;
  o.slots = o.hist_words >> o.bin_bits;
  const long long spans = (o.cap + kOrderSpan - 1) / kOrderSpan;
  const unsigned grid = (unsigned)std::max(1ll, std::min(spans, 8ll * info.sm_count));
  if (o.cap > (long long)o.K) {  // otherwise no group is larger than K
    order_range_kernel<<<grid, kOrderThreads, 0, s>>>(o, count);
    order_bins_kernel<<<grid, kOrderThreads, 0, s>>>(o, count);
  }
  const long long m = (long long)order_ordinals(o.cap, o.groups);
  const unsigned plan = (unsigned)std::max(1ll, std::min((m + 7) / 8, 4ll * info.sm_count));
  order_plan_kernel<<<plan, kOrderThreads, 0, s>>>(o, first_group_of_family2);
  order_gather_kernel<<<grid, kOrderThreads, 0, s>>>(o, count);
  P2C_CUDA(cudaFuncSetAttribute(order_pick_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(PickShared)));
  const unsigned pick = (unsigned)std::max(1ll, std::min<long long>(m, info.sm_count));
  order_pick_kernel<<<pick, kPickThreads, sizeof(PickShared), s>>>(o, first_group_of_family2);
  P2C_CUDA(cudaGetLastError());
  return P2C_OK;
}

}  // namespace p2c
