// pair_rows.cuh — candidate pairs (a, b) in ascending order, for one or two
// lists whose counts are known on the device.
//
// A counting sort by a (count, scan, place) puts the pairs into rows, then
// every row orders its own b: rows of up to 16 pairs count the smaller ones
// pair by pair, rows of up to 1,024 are sorted by one warp each in registers,
// longer ones in tiles of 8,192 by one block each, merged pairwise by one
// cooperative launch that returns at once when there is nothing to merge.
//
// Bound by L2: each pair is read twice and placed once at random (an 8-byte
// write to its row), which stays in the 126 MB L2 for the lists of a step.  A
// radix sort makes five passes over the buffers' capacity, each a read and a
// scattered write.  B200, both families, us: 27 bodies (10.5 M pairs in 14.9 M
// places) 865 -> 473; a 624k-triangle cloth (3.1 M in 4.4 M) 327 -> 90.
#pragma once

#include <cooperative_groups.h>

#include <cub/device/device_scan.cuh>

#include "p2c_internal.cuh"

namespace p2c {

constexpr int kRowThreads = 256;
constexpr unsigned kRowCountMax = 16;    // pairs of a row ordered by counting
constexpr unsigned kRowWarpMax = 1024;   // by a warp
constexpr unsigned kRowTile = 8192;      // by a block
constexpr int kRowMergeOut = 8;          // places a thread merges at once

struct RowSpan {
  unsigned start, len;
};

struct RowCounters {
  unsigned long long big;  // rows ordered in several tiles (<< 32) and their pairs
  unsigned n_mid, next_mid, n_tiles, longest;
};

// One list: packed keys a << shift | b in, a << 32 | b out, ~0 past the count.
struct RowList {
  unsigned long long* pairs;
  unsigned long long* placed;  // cap
  const unsigned long long* count;
  long long cap;
  int shift;
  unsigned* row;  // counts, then starts, then ends of the rows, from row_base on
  long long rows;
  RowCounters* ctr;
  RowSpan* mid;
  RowSpan* tiles;
  unsigned* big_at;
  unsigned* big_start;
  __device__ __forceinline__ unsigned n() const { return (unsigned)min(*count, (unsigned long long)cap); }
};

struct RowLists {
  RowList l[2];
};

namespace {

__global__ void __launch_bounds__(kRowThreads) row_count_kernel(RowLists L) {
  const RowList& R = L.l[blockIdx.y];
  const unsigned n = R.n();
  for (unsigned i = blockIdx.x * kRowThreads + threadIdx.x; i < n; i += gridDim.x * kRowThreads)
    atomicAdd(R.row + (R.pairs[i] >> R.shift), 1u);
}

// The rows of the second list follow the first's in one scan.
__device__ __forceinline__ unsigned row_base(const RowLists& L, int list) { return list == 0 ? 0u : L.l[0].n(); }

__global__ void __launch_bounds__(kRowThreads) row_place_kernel(RowLists L) {
  const RowList& R = L.l[blockIdx.y];
  const unsigned n = R.n(), base = row_base(L, blockIdx.y);
  for (unsigned i = blockIdx.x * kRowThreads + threadIdx.x; i < n; i += gridDim.x * kRowThreads) {
    const unsigned long long k = R.pairs[i];
    R.placed[atomicAdd(R.row + (k >> R.shift), 1u) - base] = k;
  }
}

__device__ __forceinline__ unsigned long long row_pair(unsigned long long a, unsigned long long b) {
  return (a << 32) | b;
}

// Short rows in place; longer ones are listed by their first pair.
__global__ void __launch_bounds__(kRowThreads) row_short_kernel(RowLists L) {
  const RowList& R = L.l[blockIdx.y];
  const unsigned n = R.n(), base = row_base(L, blockIdx.y);
  const int lane = threadIdx.x & 31;
  for (long long p0 = (long long)blockIdx.x * kRowThreads; p0 < R.cap; p0 += (long long)gridDim.x * kRowThreads) {
    const long long pl = p0 + threadIdx.x;
    const unsigned p = (unsigned)pl;
    bool is_mid = false;
    unsigned start = 0u, len = 0u;
    if (pl < n) {
      const unsigned long long k = R.placed[p], a = k >> R.shift;
      const unsigned end = R.row[a] - base;
      start = a == 0ull ? 0u : R.row[a - 1] - base;
      len = end - start;
      if (len <= kRowCountMax) {
        unsigned smaller = 0u;
        for (unsigned j = start; j < end; ++j) smaller += R.placed[j] < k ? 1u : 0u;
        R.pairs[start + smaller] = row_pair(a, k & ((1ull << R.shift) - 1ull));
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
    } else if (pl < R.cap) {
      R.pairs[pl] = ~0ull;
    }
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

template <int E>
__device__ __forceinline__ void row_warp_order(const RowList& R, RowSpan s, int lane) {
  const unsigned long long mask = (1ull << R.shift) - 1ull;  // b < 2^31: the padding sorts last
  unsigned v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const unsigned i = (unsigned)(e * 32 + lane);
    v[e] = i < s.len ? (unsigned)(R.placed[s.start + i] & mask) : 0xffffffffu;
  }
  const unsigned long long a = R.placed[s.start] >> R.shift;
  row_warp_sort<E>(v, lane);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const unsigned i = (unsigned)(lane * E + e);
    if (i < s.len) R.pairs[s.start + i] = row_pair(a, v[e]);
  }
}

// Tiles of long rows, a block each; then rows of 17 to 1,024 pairs, a warp each.  Tiles of one-tile rows go out, those to be merged back to placed.
__global__ void __launch_bounds__(kRowThreads, 4) row_long_kernel(RowLists L) {
  __shared__ unsigned word[kRowTile];
  const RowList& R = L.l[blockIdx.y];
  const unsigned n_tiles = R.ctr->n_tiles;
  const unsigned long long mask = (1ull << R.shift) - 1ull;
  const unsigned base = row_base(L, blockIdx.y);
  for (unsigned t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const RowSpan s = R.tiles[t];
    unsigned size = 2u;
    while (size < s.len) size <<= 1;
    for (unsigned e = threadIdx.x; e < size; e += kRowThreads)
      word[e] = e < s.len ? (unsigned)(R.placed[s.start + e] & mask) : 0xffffffffu;
    const unsigned long long a = R.placed[s.start] >> R.shift;
    const unsigned row_len = R.row[a] - (a == 0ull ? base : R.row[a - 1]);
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
    if (row_len <= kRowTile)
      for (unsigned e = threadIdx.x; e < s.len; e += kRowThreads) R.pairs[s.start + e] = row_pair(a, word[e]);
    else
      for (unsigned e = threadIdx.x; e < s.len; e += kRowThreads) R.placed[s.start + e] = row_pair(a, word[e]);
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
__device__ __forceinline__ unsigned row_big(const RowList& R, unsigned n_big, unsigned v) {
  unsigned lo = 0u, hi = n_big - 1u;
  while (lo < hi) {
    const unsigned mid = (lo + hi + 1u) >> 1;
    if (R.big_at[mid] <= v) lo = mid;
    else hi = mid - 1u;
  }
  return lo;
}

// Pairwise merges of the tiles of rows longer than one: every thread writes
// kRowMergeOut consecutive places, from where the merge path crosses the first.
__global__ void __launch_bounds__(kRowThreads) row_merge_kernel(RowLists L) {
  const unsigned longest = max(L.l[0].ctr->longest, L.l[1].ctr->longest);
  if (longest == 0u) return;  // the same in every block
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const unsigned stride = gridDim.x * kRowThreads, t = blockIdx.x * kRowThreads + threadIdx.x;
  int src = 0;
  for (unsigned long long width = kRowTile; width < longest; width *= 2ull) {
    for (int list = 0; list < 2; ++list) {
      const RowList& R = L.l[list];
      const unsigned long long big = R.ctr->big;
      const unsigned n_big = (unsigned)(big >> 32), total = (unsigned)big;
      const unsigned long long* from = src == 0 ? R.placed : R.pairs;
      unsigned long long* to = src == 0 ? R.pairs : R.placed;
      for (unsigned long long v0 = (unsigned long long)t * kRowMergeOut; v0 < total;
           v0 += (unsigned long long)stride * kRowMergeOut) {
        const unsigned vend = (unsigned)min((unsigned long long)total, v0 + kRowMergeOut);
        unsigned v = (unsigned)v0;
        while (v < vend) {  // pieces of one pair of runs of one row
          const unsigned r = row_big(R, n_big, v), at = R.big_at[r];
          const unsigned len = (r + 1u < n_big ? R.big_at[r + 1u] : total) - at;
          const unsigned long long pair = (unsigned long long)(v - at) / (2ull * width) * (2ull * width);
          const unsigned first = R.big_start[r] + (unsigned)pair;
          const unsigned left = (unsigned)min(width, (unsigned long long)len - pair);
          const unsigned both = (unsigned)min(2ull * width, (unsigned long long)len - pair), right = both - left;
          const unsigned d = v - at - (unsigned)pair, dend = min(both, d + (vend - v));
          const unsigned long long *ka = from + first, *kb = ka + left;
          unsigned x0 = d > right ? d - right : 0u, x1 = min(d, left);  // words of the left run before place d
          while (x0 < x1) {
            const unsigned m = (x0 + x1) >> 1;
            if (ka[m] < kb[d - 1u - m]) x0 = m + 1u;
            else x1 = m;
          }
          unsigned x = x0, y = d - x0;
          for (unsigned p = d; p < dend; ++p) {
            const bool take_left = y >= right || (x < left && ka[x] < kb[y]);
            to[first + p] = take_left ? ka[x++] : kb[y++];
          }
          v += dend - d;
        }
      }
    }
    grid.sync();
    src = 1 - src;
  }
  if (src != 0) return;  // the last merge wrote to pairs
  for (int list = 0; list < 2; ++list) {
    const RowList& R = L.l[list];
    const unsigned long long big = R.ctr->big;
    const unsigned n_big = (unsigned)(big >> 32), total = (unsigned)big;
    for (unsigned v = t; v < total; v += stride) {
      const unsigned r = row_big(R, n_big, v), p = R.big_start[r] + (v - R.big_at[r]);
      R.pairs[p] = R.placed[p];
    }
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
RowScratch carve_rows(long long rows, long long pair_cap, Take take) {
  RowScratch s;
  const size_t cap = (size_t)(pair_cap > 0 ? pair_cap : 1);
  s.zero_bytes = 256 + (size_t)(rows > 0 ? rows : 1) * 4;
  char* zero = static_cast<char*>(take(s.zero_bytes));
  s.ctr = reinterpret_cast<RowCounters*>(zero);
  s.row = reinterpret_cast<unsigned*>(zero == nullptr ? nullptr : zero + 256);
  for (int k = 0; k < 2; ++k) {
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

// Sorts both lists in place (a list of capacity 0 takes no part).
inline int launch_pair_rows(const RowScratch& w, unsigned long long* const pairs[2], const long long cap[2],
                            const unsigned long long* const count[2], const int shift[2], const long long rows[2],
                            cudaStream_t s) {
  RowLists L;
  long long most = 0;
  for (int k = 0; k < 2; ++k) {
    L.l[k] = RowList{pairs[k], w.placed[k], count[k], cap[k],   shift[k],    w.row + (k == 0 ? 0 : rows[0]),
                     rows[k],  w.ctr + k,   w.mid[k], w.tiles[k], w.big_at[k], w.big_start[k]};
    most = std::max(most, cap[k]);
  }
  if (most == 0) return P2C_OK;
  DeviceInfo info;
  if (int rc = current_device_info(&info)) return rc;
  const unsigned blocks = (unsigned)std::min<long long>((most + kRowThreads - 1) / kRowThreads, 8ll * info.sm_count);
  P2C_CUDA(cudaMemsetAsync(w.ctr, 0, w.zero_bytes, s));
  row_count_kernel<<<dim3(blocks, 2), kRowThreads, 0, s>>>(L);
  size_t bytes = w.scan_bytes;
  P2C_CUDA(cub::DeviceScan::ExclusiveSum(w.scan, bytes, w.row, w.row, (int)std::max(1ll, rows[0] + rows[1]), s));
  row_place_kernel<<<dim3(blocks, 2), kRowThreads, 0, s>>>(L);
  row_short_kernel<<<dim3(blocks, 2), kRowThreads, 0, s>>>(L);
  row_long_kernel<<<dim3((unsigned)info.sm_count * 4u, 2), kRowThreads, 0, s>>>(L);
  if (most > (long long)kRowTile) {
    void* args[] = {&L};
    P2C_CUDA(cudaLaunchCooperativeKernel((const void*)row_merge_kernel, dim3((unsigned)info.sm_count), dim3(kRowThreads),
                                         args, 0, s));
  }
  P2C_CUDA(cudaGetLastError());
  return P2C_OK;
}

}  // namespace p2c
