// pair_rows.cuh — candidate pairs (a, b) in ascending order, for one or two
// lists whose counts are known on the device.
//
// A counting sort by a (count, scan, place) puts the pairs into rows, then
// every row orders its own b: rows of up to 16 pairs count the smaller ones
// pair by pair, rows of up to 1,024 are sorted by one warp each in registers,
// longer ones in tiles of 8,192 by one block each, merged eight at a time by a
// launch per round that returns at once when there is nothing to merge.  Plain
// launches: a cooperative one, which could run all rounds, fails on a stream
// that owns part of the SMs only.
//
// Bound by L2: each pair is read twice and placed once at random (an 8-byte
// write to its row), which stays in the 126 MB L2 for the lists of a step.  A
// radix sort makes five passes over the buffers' capacity, each a read and a
// scattered write.  B200, both families, us: 27 bodies (10.5 M pairs in 14.9 M
// places) 865 -> 473; a 624k-triangle cloth (3.1 M in 4.4 M) 327 -> 90.
#pragma once

#include <cub/device/device_scan.cuh>

#include "p2c_internal.cuh"
#include "run_merge.cuh"

namespace p2c {

constexpr int kRowThreads = 256;
constexpr unsigned kRowCountMax = 16;    // pairs of a row ordered by counting
constexpr unsigned kRowWarpMax = 1024;   // by a warp
constexpr unsigned kRowTile = 8192;      // by a block

struct RowSpan {
  unsigned start, len;
};

struct RowCounters {
  unsigned long long big;  // rows ordered in several tiles (<< 32) and their pairs
  unsigned n_mid, next_mid, n_tiles, longest;
};

// One list of pairs of one scene: packed keys a << shift | b in, a << 32 | b
// out in place, ~0 past the count.  A source tells a list's live entries, the
// row of a key, the bits of b in it, and where the key of a place goes.
struct SceneRows {
  unsigned long long* pairs;
  const unsigned long long* count;
  long long cap;
  int shift;
  __device__ __forceinline__ bool live(long long i) const { return (unsigned long long)i < *count; }
  __device__ __forceinline__ bool load(long long i, unsigned long long& key) const {
    if (!live(i)) return false;
    key = pairs[i];
    return true;
  }
  __device__ __forceinline__ unsigned long long row(unsigned long long key) const { return key >> shift; }
  __device__ __forceinline__ unsigned long long b_mask(unsigned long long) const { return (1ull << shift) - 1ull; }
  __device__ __forceinline__ void pad(long long i) const { pairs[i] = ~0ull; }
  __device__ __forceinline__ void store(unsigned place, unsigned long long key, const unsigned*) const {
    pairs[place] = ((key >> shift) << 32) | (key & b_mask(key));
  }
  __device__ __forceinline__ unsigned long long* input() const { return pairs; }
};

template <class Source>
struct RowList {
  Source src;
  unsigned long long* placed;  // cap
  unsigned* row;               // counts, then starts, then ends of the rows; row[-1] is where the list starts
  long long rows;              // row[rows], of no pair, is where it ends
  RowCounters* ctr;
  RowSpan* mid;
  RowSpan* tiles;
  unsigned* big_at;
  unsigned* big_start;
  int list;
  __device__ __forceinline__ unsigned base() const { return list == 0 ? 0u : row[-1]; }
  __device__ __forceinline__ unsigned n() const { return row[rows] - base(); }
  __device__ __forceinline__ unsigned start(unsigned long long r) const {
    return r == 0ull ? 0u : row[(long long)r - 1] - base();
  }
};

template <class Source>
struct RowLists {
  RowList<Source> l[2];
};

namespace {

// Lanes of a warp that meet in a row add to its counter once: all pairs of a
// primitive that is large against the others share one.
template <class Source>
__global__ void __launch_bounds__(kRowThreads) row_count_kernel(RowLists<Source> L) {
  const RowList<Source>& R = L.l[blockIdx.y];
  const int lane = threadIdx.x & 31;
  for (long long i0 = (long long)blockIdx.x * kRowThreads; i0 < R.src.cap; i0 += (long long)gridDim.x * kRowThreads) {
    const long long i = i0 + threadIdx.x;
    unsigned long long k = 0ull;
    const bool in = i < R.src.cap && R.src.load(i, k);
    const unsigned row = in ? (unsigned)R.src.row(k) : 0xffffffffu;
    const unsigned same = __match_any_sync(0xffffffffu, row);
    if (in && lane == __ffs((int)same) - 1) atomicAdd(R.row + row, (unsigned)__popc(same));
  }
}

template <class Source>
__global__ void __launch_bounds__(kRowThreads) row_place_kernel(RowLists<Source> L) {
  const RowList<Source>& R = L.l[blockIdx.y];
  const unsigned base = R.base();
  const int lane = threadIdx.x & 31;
  for (long long i0 = (long long)blockIdx.x * kRowThreads; i0 < R.src.cap; i0 += (long long)gridDim.x * kRowThreads) {
    const long long i = i0 + threadIdx.x;
    unsigned long long k = 0ull;
    const bool in = i < R.src.cap && R.src.load(i, k);
    const unsigned row = in ? (unsigned)R.src.row(k) : 0xffffffffu;
    const unsigned same = __match_any_sync(0xffffffffu, row);
    const int leader = __ffs((int)same) - 1;
    unsigned at = 0u;
    if (in && lane == leader) at = atomicAdd(R.row + row, (unsigned)__popc(same));
    at = __shfl_sync(0xffffffffu, at, leader) + (unsigned)__popc(same & ((1u << lane) - 1u));
    if (in) R.placed[at - base] = k;
  }
}

// Short rows; longer ones are listed by their first pair.  Entries past a
// list's count are padded.
template <class Source>
__global__ void __launch_bounds__(kRowThreads) row_short_kernel(RowLists<Source> L) {
  const RowList<Source>& R = L.l[blockIdx.y];
  const unsigned n = R.n(), base = R.base();
  const int lane = threadIdx.x & 31;
  for (long long p0 = (long long)blockIdx.x * kRowThreads; p0 < R.src.cap; p0 += (long long)gridDim.x * kRowThreads) {
    const long long pl = p0 + threadIdx.x;
    const unsigned p = (unsigned)pl;
    bool is_mid = false;
    unsigned start = 0u, len = 0u;
    if (pl < n) {
      const unsigned long long k = R.placed[p], r = R.src.row(k);
      const unsigned end = R.row[r] - base;
      start = R.start(r);
      len = end - start;
      if (len <= kRowCountMax) {
        unsigned smaller = 0u;
        for (unsigned j = start; j < end; ++j) smaller += R.placed[j] < k ? 1u : 0u;
        R.src.store(start + smaller, k, R.row);
      } else if (p == start) {
        if (len <= kRowWarpMax) {
          is_mid = true;
        } else {
          const unsigned tiles = (len + kRowTile - 1) / kRowTile;
          const unsigned at = atomicAdd(&R.ctr->n_tiles, tiles);
          for (unsigned t = 0; t < tiles; ++t)
            R.tiles[at + t] = RowSpan{start + t * kRowTile, min(kRowTile, len - t * kRowTile)};
          if (tiles > 1u) {
            const unsigned long long b = atomicAdd(&R.ctr->big, (1ull << 32) | len);
            R.big_start[b >> 32] = start;
            R.big_at[b >> 32] = (unsigned)b;
            atomicMax(&R.ctr->longest, len);
          }
        }
      }
    }
    if (pl < R.src.cap && !R.src.live(pl)) R.src.pad(pl);
    const unsigned m = __ballot_sync(0xffffffffu, is_mid);
    if (m) {
      unsigned at = 0u;
      if (lane == 0) at = atomicAdd(&R.ctr->n_mid, (unsigned)__popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (is_mid) R.mid[at + (unsigned)__popc(m & ((1u << lane) - 1u))] = RowSpan{start, len};
    }
  }
}

// Bitonic sort of a warp's 32 * E words in registers; word e of a lane has
// place lane * E + e.  From runs of E words on, a lane's words all sort the
// same way, so a step is a shuffle and one minimum or maximum by predicate, or
// the latter alone inside a lane (directions worked out word by word made the
// kernel 308 us for 27 bodies, now 155).
template <int E>
__device__ __forceinline__ void row_warp_sort(unsigned (&v)[E], int lane) {
#pragma unroll
  for (int k = 2; k < E; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if ((e & j) != 0) continue;
        const unsigned a = v[e], b = v[e | j];
        v[e] = (e & k) == 0 ? min(a, b) : max(a, b);
        v[e | j] = (e & k) == 0 ? max(a, b) : min(a, b);
      }
    }
  }
#pragma unroll 1
  for (int k = E > 1 ? E : 2; k <= 32 * E; k <<= 1) {
    const bool up = (lane & (k / E)) == 0;
#pragma unroll 1
    for (int j = k >> 1; j >= E; j >>= 1) {
      const bool least = ((lane & (j / E)) == 0) == up;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const unsigned o = __shfl_xor_sync(0xffffffffu, v[e], j / E);
        v[e] = least ? min(v[e], o) : max(v[e], o);
      }
    }
#pragma unroll
    for (int j = E >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if ((e & j) != 0) continue;
        const unsigned a = v[e], b = v[e | j];
        v[e] = up ? min(a, b) : max(a, b);
        v[e | j] = up ? max(a, b) : min(a, b);
      }
    }
  }
}

template <int E, class Source>
__device__ __forceinline__ void row_warp_order(const RowList<Source>& R, RowSpan s, int lane) {
  const unsigned long long first = R.placed[s.start], mask = R.src.b_mask(first);  // b < 2^31: padding sorts last
  unsigned v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const unsigned i = (unsigned)(e * 32 + lane);
    v[e] = i < s.len ? (unsigned)(R.placed[s.start + i] & mask) : 0xffffffffu;
  }
  row_warp_sort<E>(v, lane);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const unsigned i = (unsigned)(lane * E + e);
    if (i < s.len) R.src.store(s.start + i, (first & ~mask) | v[e], R.row);
  }
}

// Rounds that merge the longest row of both lists.
template <class Source>
__device__ __forceinline__ int row_rounds(const RowLists<Source>& L) {
  return merge_rounds(kRowTile, max(L.l[0].ctr->longest, L.l[1].ctr->longest));
}
// Whether a round reads placed (otherwise the places of the same numbers in
// the input).  The last one does: it stores, which may be over the input.
__device__ __forceinline__ bool row_round_placed(int rounds, int round) { return ((rounds - 1 - round) & 1) == 0; }

// Tiles of long rows, a block each; then rows of 17 to 1,024 pairs, a warp each.
// Tiles of one-tile rows go out, those to be merged where the first round reads.
template <class Source>
__global__ void __launch_bounds__(kRowThreads, 4) row_long_kernel(RowLists<Source> L) {
  __shared__ unsigned word[kRowTile];
  const RowList<Source>& R = L.l[blockIdx.y];
  const unsigned n_tiles = R.ctr->n_tiles;
  const int rounds = n_tiles != 0u ? row_rounds(L) : 0;
  unsigned long long* merged = row_round_placed(rounds, 0) ? R.placed : R.src.input();
  for (unsigned t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const RowSpan s = R.tiles[t];
    unsigned size = 2u;
    while (size < s.len) size <<= 1;
    const unsigned long long first = R.placed[s.start], mask = R.src.b_mask(first), r = R.src.row(first);
    for (unsigned e = threadIdx.x; e < size; e += kRowThreads)
      word[e] = e < s.len ? (unsigned)(R.placed[s.start + e] & mask) : 0xffffffffu;
    const unsigned row_len = R.row[r] - R.base() - R.start(r);
    __syncthreads();
    // 32 consecutive compare pairs span 64 words: steps of at most 32 stay within one warp's words
    for (unsigned k = 2; k <= size; k <<= 1) {
      for (unsigned j = k >> 1; j > 0; j >>= 1) {
        for (unsigned p = threadIdx.x; p < size / 2; p += kRowThreads) {
          const unsigned x = 2u * p - (p & (j - 1u)), y = x + j;
          const unsigned wx = word[x], wy = word[y];
          if ((wy < wx) == ((x & k) == 0u)) {
            word[x] = wy;
            word[y] = wx;
          }
        }
        if (j > 32u) __syncthreads();
        else __syncwarp();
      }
      __syncthreads();
    }
    for (unsigned e = threadIdx.x; e < s.len; e += kRowThreads) {
      const unsigned long long key = (first & ~mask) | word[e];
      if (row_len <= kRowTile) R.src.store(s.start + e, key, R.row);
      else merged[s.start + e] = key;
    }
    __syncthreads();
  }
  const unsigned n_mid = R.ctr->n_mid;
  const int lane = threadIdx.x & 31;
  // rows differ by a factor of 60 in length, so warps draw them; the next draw
  // travels while a row is sorted
  unsigned drawn = 0u;
  if (lane == 0) drawn = atomicAdd(&R.ctr->next_mid, 1u);
  while (true) {
    const unsigned t = __shfl_sync(0xffffffffu, drawn, 0);
    if (t >= n_mid) break;
    if (lane == 0) drawn = atomicAdd(&R.ctr->next_mid, 1u);
    const RowSpan s = R.mid[t];
    if (s.len <= 32u) row_warp_order<1>(R, s, lane);
    else if (s.len <= 64u) row_warp_order<2>(R, s, lane);
    else if (s.len <= 128u) row_warp_order<4>(R, s, lane);
    else if (s.len <= 256u) row_warp_order<8>(R, s, lane);
    else if (s.len <= 512u) row_warp_order<16>(R, s, lane);
    else row_warp_order<32>(R, s, lane);
  }
}

// Which big row place v of their sequence belongs to.
template <class Source>
__device__ __forceinline__ unsigned row_big(const RowList<Source>& R, unsigned n_big, unsigned v) {
  unsigned lo = 0u, hi = n_big - 1u;
  while (lo < hi) {
    const unsigned mid = (lo + hi + 1u) >> 1;
    if (R.big_at[mid] <= v) lo = mid;
    else hi = mid - 1u;
  }
  return lo;
}

// One round over the rows of more than one tile (run_merge.cuh).  Bound by the
// latency of the searches and by scattered 8-byte writes, both in L2.  1.4 M
// pairs in rows of up to 145,000, two rounds: 186 us, as much as four pairwise
// rounds in one cooperative launch (176); 266 with every lane searching whole
// runs.
template <class Source>
__global__ void __launch_bounds__(kRowThreads) row_merge_kernel(RowLists<Source> L, int round) {
  pdl_wait();
  pdl_trigger();
  const int rounds = row_rounds(L);
  if (round >= rounds) return;
  const RowList<Source>& R = L.l[blockIdx.y];
  const unsigned long long big = R.ctr->big;
  const unsigned n_big = (unsigned)(big >> 32), total = (unsigned)big;
  const bool last = round == rounds - 1;
  const unsigned long long* from = row_round_placed(rounds, round) ? R.placed : R.src.input();
  unsigned long long* to = row_round_placed(rounds, round) ? R.src.input() : R.placed;
  const unsigned width = merge_width(kRowTile, round);
  for (unsigned long long v0 = (unsigned long long)blockIdx.x * kRowThreads; v0 < total;
       v0 += (unsigned long long)gridDim.x * kRowThreads) {
    const bool live = v0 + threadIdx.x < total;
    const unsigned v = (unsigned)min(v0 + threadIdx.x, (unsigned long long)total - 1ull);
    const unsigned r = row_big(R, n_big, v), at = R.big_at[r];
    const unsigned len = (r + 1u < n_big ? R.big_at[r + 1u] : total) - at, a = v - at;
    const unsigned own = a / width, run0 = own / kMergeRuns * kMergeRuns;
    const unsigned first = R.big_start[r] + run0 * width;  // run0 * width <= a
    const unsigned long long* runs = from + first;
    const unsigned long long key = runs[a - run0 * width];
    unsigned n[kMergeRuns];
#pragma unroll
    for (unsigned k = 0; k < kMergeRuns; ++k) {
      const unsigned long long begin = (unsigned long long)(run0 + k) * width;  // in the row
      n[k] = run0 + k == own || begin >= len ? 0u : (unsigned)min((unsigned long long)width, len - begin);
    }
    const unsigned r0 = __shfl_sync(0xffffffffu, r, 0), own0 = __shfl_sync(0xffffffffu, own, 0);
    const bool together = __all_sync(0xffffffffu, live && r == r0 && own == own0);
    const unsigned place = a - own * width +
                           entries_before(width, n, key, 0u, together, [&](unsigned k, unsigned p, unsigned long long x,
                                                                           unsigned) { return runs[k * width + p] < x; });
    if (!live) continue;
    if (last) R.src.store(first + place, key, R.row);
    else to[first + place] = key;
  }
}

}  // namespace

inline size_t row_scan_bytes(long long rows) {
  size_t bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, bytes, (unsigned*)nullptr, (unsigned*)nullptr, (int)(rows > 0 ? rows : 1));
  return bytes;
}

// Scratch of launch_pair_rows, carved by take(bytes): counters and rows come
// first and have to be zero before the launch (zero_bytes from zero_at).
struct RowScratch {
  RowCounters* ctr;
  unsigned* row;
  size_t zero_bytes;
  unsigned long long* placed[2];
  RowSpan *mid[2], *tiles[2];
  unsigned *big_at[2], *big_start[2];
  void* scan;
  size_t scan_bytes;
};

template <class Take>
RowScratch carve_rows(long long rows, const long long pair_cap[2], Take take) {
  RowScratch s;
  rows += 2;  // the two ends
  s.zero_bytes = 256 + (size_t)rows * 4;
  char* zero = static_cast<char*>(take(s.zero_bytes));
  s.ctr = reinterpret_cast<RowCounters*>(zero);
  s.row = reinterpret_cast<unsigned*>(zero == nullptr ? nullptr : zero + 256);
  for (int k = 0; k < 2; ++k) {
    const size_t cap = (size_t)(pair_cap[k] > 0 ? pair_cap[k] : 1);
    s.placed[k] = static_cast<unsigned long long*>(take(cap * 8));
    s.mid[k] = static_cast<RowSpan*>(take((cap / (kRowCountMax + 1) + 1) * sizeof(RowSpan)));
    s.tiles[k] = static_cast<RowSpan*>(take((cap / kRowWarpMax + 1) * sizeof(RowSpan)));
    s.big_at[k] = static_cast<unsigned*>(take((cap / kRowTile + 1) * 4));
    s.big_start[k] = static_cast<unsigned*>(take((cap / kRowTile + 1) * 4));
  }
  s.scan_bytes = row_scan_bytes(rows);
  s.scan = take(s.scan_bytes);
  return s;
}

// Sorts both lists (one of capacity 0 takes no part).  most_in_row: pairs that
// one row of each list can have.
template <class Source>
int launch_pair_rows(const RowScratch& w, const Source& first, const Source& second, const long long rows[2],
                     const long long most_in_row[2], cudaStream_t s) {
  RowLists<Source> L;
  const Source* src[2] = {&first, &second};
  for (int k = 0; k < 2; ++k)
    L.l[k] = RowList<Source>{*src[k],  w.placed[k], w.row + (k == 0 ? 0 : rows[0] + 1), rows[k], w.ctr + k, w.mid[k],
                             w.tiles[k], w.big_at[k], w.big_start[k], k};
  const long long most = std::max(first.cap, second.cap);
  if (most == 0) return P2C_OK;
  DeviceInfo info;
  if (int rc = current_device_info(&info)) return rc;
  const dim3 blocks((unsigned)std::min<long long>((most + kRowThreads - 1) / kRowThreads, 8ll * info.sm_count), 2);
  P2C_CUDA(cudaMemsetAsync(w.ctr, 0, w.zero_bytes, s));
  row_count_kernel<<<blocks, kRowThreads, 0, s>>>(L);
  size_t bytes = w.scan_bytes;
  P2C_CUDA(cub::DeviceScan::ExclusiveSum(w.scan, bytes, w.row, w.row, (int)(rows[0] + rows[1] + 2), s));
  row_place_kernel<<<blocks, kRowThreads, 0, s>>>(L);
  row_short_kernel<<<blocks, kRowThreads, 0, s>>>(L);
  row_long_kernel<<<dim3((unsigned)info.sm_count * 4u, 2), kRowThreads, 0, s>>>(L);
  const long long longest = std::max(std::min(first.cap, most_in_row[0]), std::min(second.cap, most_in_row[1]));
  for (int round = 0; round < merge_rounds(kRowTile, (unsigned long long)longest); ++round)
    P2C_CUDA(launch_pdl(row_merge_kernel<Source>, dim3((unsigned)info.sm_count * 4u, 2), dim3(kRowThreads), 0, s, L,
                        round));
  P2C_CUDA(cudaGetLastError());
  return P2C_OK;
}

}  // namespace p2c
