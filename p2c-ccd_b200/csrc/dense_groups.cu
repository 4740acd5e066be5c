// dense_groups.cu — the candidate-group early-stop replay on the device.
//
// RunDenseGroupExactEarlyStop (common/group_scheduler.cpp:60-239) replays a
// learned proposal schedule over candidate groups (one group per query id)
// against known labels, with no certificates: candidates are ordered by
// (query id, priority desc, cost asc, index) — or by (query id, index) when
// the input order is kept — and each group is walked in that order:
//
//   * a candidate whose uncertainty reaches the threshold sends the rest of
//     the group to full fallback (every candidate from there on at full cost
//     until the first colliding one);
//   * otherwise it costs its narrow cost; a colliding candidate whose
//     predicted interval meets the contact interval is a hit; a colliding
//     one that misses costs the miss penalty and, once the attempt limit is
//     reached, one full fallback call that ends the group as a collision.
//
// The binding parses the rows first (py_module.cpp:1179-1246): the
// predicted interval is the arg-max bin of eight interval scores, the full
// cost is oracle_trace[:, 5], the narrow cost full * cost_target (at least
// 1e-12) when cost_target is finite and positive, the contact interval
// oracle_trace[:, 6:8] and the label oracle_trace[:, 0] > 0.5.
//
// Device layout: one thread per row parses, validates and writes the row's
// 32-byte walk record; one stable radix sort by query id makes the groups
// contiguous; each group orders its own rows by (priority desc, cost asc,
// index) in shared memory (larger ones in tiles that are merged); one warp per
// group finds the stopping position with ballots and folds the group's sums
// row by row in order.  The reference adds its work totals one term at a time
// into double accumulators, so the totals depend on the order of the
// additions: every term goes to a slot whose position is its place in the
// reference's sequence (empty slots are +0.0, which adds exactly nothing to a
// sum that starts at +0.0 and only grows), the non-zero slots are compacted
// in order, and each total is the exact left-to-right sum formed from
// composable pieces (the ordered fold below).  Every total is therefore the
// reference's to the bit.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <cmath>

#include "p2c_internal.cuh"
#include "run_merge.cuh"

namespace p2c {
namespace {

constexpr int kThreads = 256;
constexpr int kWarpRows = 256;    // rows a warp orders
constexpr int kTileThreads = 512;
constexpr unsigned kTileRows = 4096;  // rows a block orders
constexpr int kFoldThreads = 512;
constexpr int kFoldPerThread = 8;  // consecutive terms per thread
constexpr int kFoldChunk = kFoldThreads * kFoldPerThread;
constexpr int kFoldWarps = kFoldThreads / 32;
constexpr unsigned char kColl = 1, kOverlap = 2, kHighUnc = 4;

// Integer totals, in p2c_dense_group_stats order of the counters below.
enum {
  kGroups,
  kPositive,
  kCalls,
  kFallback,
  kHit,
  kMiss,
  kTP,
  kTN,
  kFP,
  kFN,
  kReordered,
  kHighUncGroups,
  kRankSum,
  kNumCounters
};

struct DenseAcc {
  unsigned long long ctr[kNumCounters];
  unsigned long long first_error;  // (row << 2) | kind; ~0 none
  int n_groups;                    // DeviceSelect's count of group heads
  int n_terms;                     // DeviceSelect's count of non-zero work terms
  unsigned long long big;          // groups ordered in tiles (<< 32) and their rows
  unsigned next[2];                // the next group to order, to walk
  unsigned n_tiles;
  unsigned longest;                // rows of the largest group ordered in tiles
  unsigned fold_blocks[3];         // finished blocks of each total's chunk sums
};

// What the walk reads of one row: one 32-byte sector at a random place.
struct __align__(16) WalkRow {
  double full, narrow;  // PositiveCost(full, 1), PositiveCost(narrow, full)
  unsigned long long flags, pad;
};

struct Tile {
  unsigned start, len;  // len has kTileMerged set when the group has several
};
constexpr unsigned kTileMerged = 1u << 31;

// One piece of kFoldChunk terms of a total: its sum (any order, to predict the
// binade it is added in), that binade's last place, and the increments of the
// running sum for an even and an odd one.
struct FoldPieces {
  double* sum[3];
  int* ulp[3];
  ulonglong2* inc[3];
};

struct DenseLayout {
  DenseAcc* acc = nullptr;
  unsigned long long* key[2] = {nullptr, nullptr};   // sort A: priority desc | cost asc
  unsigned long long* qkey[2] = {nullptr, nullptr};  // sort B: query id
  unsigned* idx[3] = {nullptr, nullptr, nullptr};
  WalkRow* rows = nullptr;  // input order
  unsigned* g_start = nullptr;
  unsigned* big_at = nullptr;   // groups ordered in tiles: first row in the sequence of their rows
  unsigned* big_start = nullptr;
  Tile* tiles = nullptr;
  FoldPieces pieces = {};
  double* terms = nullptr;    // 2n + n slots (2 per candidate + 1 per group at most)
  double* compact = nullptr;  // the non-zero terms, in order
  double* g_full = nullptr;   // per group: the summed full costs
  double* g_cost = nullptr;   // per group: the cost before its first positive (0 when none)
  void* tmp = nullptr;
  size_t tmp_bytes = 0;
  size_t total = 0;
};

// A row whose query id differs from the one before it.
struct IsHead {
  const unsigned long long* qid;
  __device__ bool operator()(unsigned i) const { return i == 0u || qid[i] != qid[i - 1]; }
};

struct NonZeroTerm {
  __host__ __device__ bool operator()(double x) const { return x != 0.0; }
};

size_t fold_chunks(long long terms) { return (size_t)((terms + kFoldChunk - 1) / kFoldChunk); }

size_t cub_bytes(long long n) {
  const int m = (int)(n > 0 ? n : 1);
  size_t a = 0, b = 0, c = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, a, (const unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                  (const unsigned*)nullptr, (unsigned*)nullptr, m);
  cub::DeviceSelect::If(nullptr, b, thrust::counting_iterator<unsigned>(0u), (unsigned*)nullptr, (int*)nullptr, m,
                        IsHead{});
  cub::DeviceSelect::If(nullptr, c, (const double*)nullptr, (double*)nullptr, (int*)nullptr, 3 * m, NonZeroTerm{});
  return std::max(a, std::max(b, c));
}

DenseLayout carve(void* base, long long n) {
  DenseLayout L;
  char* p = static_cast<char*>(base);
  size_t off = 0;
  auto take = [&](size_t bytes) -> void* {
    off = (off + 255) & ~size_t(255);
    void* r = p ? p + off : nullptr;
    off += bytes;
    return r;
  };
  const size_t m = (size_t)(n > 0 ? n : 1);
  L.acc = (DenseAcc*)take(sizeof(DenseAcc));
  for (auto& k : L.key) k = (unsigned long long*)take(8 * m);
  for (auto& k : L.qkey) k = (unsigned long long*)take(8 * m);
  for (auto& v : L.idx) v = (unsigned*)take(4 * m);
  L.rows = (WalkRow*)take(sizeof(WalkRow) * m);
  L.g_start = (unsigned*)take(4 * m);
  L.big_at = (unsigned*)take(4 * (m / kWarpRows + 1));
  L.big_start = (unsigned*)take(4 * (m / kWarpRows + 1));
  L.tiles = (Tile*)take(sizeof(Tile) * (m / kWarpRows + 1));
  for (int k = 0; k < 3; ++k) {
    const size_t c = fold_chunks(k == 0 ? 3 * (long long)m : (long long)m);
    L.pieces.sum[k] = (double*)take(8 * c);
    L.pieces.ulp[k] = (int*)take(4 * c);
    L.pieces.inc[k] = (ulonglong2*)take(16 * c);
  }
  L.terms = (double*)take(8 * 3 * m);
  L.compact = (double*)take(8 * 3 * m);
  L.g_full = (double*)take(8 * m);
  L.g_cost = (double*)take(8 * m);
  L.tmp_bytes = cub_bytes(n);
  L.tmp = take(L.tmp_bytes);
  L.total = off;
  return L;
}

__device__ __forceinline__ unsigned float_key_asc(float f) {
  unsigned u = __float_as_uint(f == 0.0f ? 0.0f : f);  // -0 and +0 compare equal
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ double positive_cost(double v, double fallback) {  // group_scheduler.cpp:31-36
  return (!isfinite(v) || v <= 0.0) ? fallback : v;
}

struct ParseIn {
  const unsigned long long* query_id;
  const unsigned long long* candidate_id;
  const float* cost_target;
  const double* oracle_trace;  // n x 8
  const float* interval_scores;  // n x 8
  const float* priority;
  const float* cost_score;
  const float* uncertainty;
};

__global__ void init_kernel(DenseLayout L) {
  if (threadIdx.x < kNumCounters) L.acc->ctr[threadIdx.x] = 0;
  if (threadIdx.x < 3) L.acc->fold_blocks[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    L.acc->first_error = ~0ull;
    L.acc->n_groups = 0;
    L.acc->n_terms = 0;
    L.acc->big = 0;
    L.acc->next[0] = L.acc->next[1] = 0;
    L.acc->n_tiles = 0;
    L.acc->longest = 0;
  }
}

// One row: the binding's parse (py_module.cpp:1212-1244), the engine's
// validation (group_scheduler.cpp:81-88), the per-candidate costs and flags
// of the walk (:143-150, :170) and the sort keys.
__global__ void __launch_bounds__(kThreads) parse_kernel(ParseIn in, long long n, float threshold, int keep_order,
                                                         DenseLayout L) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned long long qid = in.query_id[i], cid = in.candidate_id[i];
  const float* sc = in.interval_scores + 8 * i;
  int best = 0;
  float best_score = sc[0];
#pragma unroll
  for (int k = 1; k < 8; ++k) {
    const float v = sc[k];
    if (v > best_score) {
      best_score = v;
      best = k;
    }
  }
  const double width = 1.0 / 8.0;
  const double it0 = width * (double)best;
  const double it0w = it0 + width;
  const double it1 = it0w < 1.0 ? it0w : 1.0;  // std::min(1.0, t0 + width)
  const double* tr = in.oracle_trace + 8 * i;
  const double full = tr[5];
  const float ratio = in.cost_target[i];
  double narrow = full;
  if (isfinite(ratio) && ratio > 0.0f) {
    const double x = full * (double)ratio;
    narrow = 1.0e-12 < x ? x : 1.0e-12;  // std::max(1e-12, x)
  }
  const double c0 = tr[6], c1 = tr[7];
  const float prio = in.priority[i], cost = in.cost_score[i], unc = in.uncertainty[i];
  unsigned kind = 0;
  if (qid == 0 || cid == 0)
    kind = 1;
  else if (!(isfinite(full) && isfinite(narrow) && isfinite(c0) && isfinite(c1) && isfinite(prio) &&
             isfinite(cost) && isfinite(unc)))
    kind = 2;
  if (kind) atomicMin(&L.acc->first_error, ((unsigned long long)i << 2) | kind);
  const double fc = positive_cost(full, 1.0);
  const double lo = it0 < c0 ? c0 : it0;  // std::max(interval_t0, contact_t0)
  const double hi = c1 < it1 ? c1 : it1;  // std::min(interval_t1, contact_t1)
  WalkRow row;
  row.full = fc;
  row.narrow = positive_cost(narrow, fc);
  row.flags = (tr[0] > 0.5 ? kColl : 0) | (lo <= hi ? kOverlap : 0) | (unc >= threshold ? kHighUnc : 0);
  row.pad = 0;
  L.rows[i] = row;
  L.idx[0][i] = (unsigned)i;
  L.qkey[0][i] = qid;
  if (!keep_order) L.key[0][i] = ((unsigned long long)(~float_key_asc(prio)) << 32) | float_key_asc(cost);
}

// ---- the order inside a group ----------------------------------------------
//
// Rows of a group lie together in index order; they are ordered by (key,
// index).  Groups of up to 256 rows are sorted by one warp each in registers,
// larger ones in tiles of 4096 by one block each, and the tiles are merged
// eight at a time by a launch per round (which returns at once when no group is
// larger than a tile; plain launches, so that a stream which owns part of the
// SMs only will do).  Each row's key is read once; the sort over all rows by the
// 64-bit key that this stands in for was 8 radix passes: 168 us for 1 M rows,
// the ordering kernels 52.

__device__ __forceinline__ bool entry_less(unsigned long long ka, unsigned ia, unsigned long long kb, unsigned ib) {
  return ka < kb || (ka == kb && ia < ib);
}

// Bitonic sort of a warp's 32 * E entries in registers; entry e of a lane has
// place lane * E + e, so the steps below E stay inside a lane, the others go
// between lanes.  The stages are loops, not unrolled: five sizes of straight
// code missed the instruction cache (65 us a million rows, as loops 46).
template <int E>
__device__ __forceinline__ void warp_sort(unsigned long long (&key)[E], unsigned (&idx)[E], int lane) {
#pragma unroll 1
  for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll 1
    for (int j = k >> 1; j >= E; j >>= 1) {
      const bool low = (lane & (j / E)) == 0;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const unsigned long long ok = __shfl_xor_sync(0xffffffffu, key[e], j / E);
        const unsigned oi = __shfl_xor_sync(0xffffffffu, idx[e], j / E);
        const bool up = ((lane * E + e) & k) == 0;
        if (entry_less(ok, oi, key[e], idx[e]) == (low == up)) {
          key[e] = ok;
          idx[e] = oi;
        }
      }
    }
#pragma unroll
    for (int j = E >> 1; j > 0; j >>= 1) {
      if (j >= k) continue;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if ((e & j) != 0) continue;
        const int b = e | j;
        const bool up = ((lane * E + e) & k) == 0;
        if (entry_less(key[b], idx[b], key[e], idx[e]) == up) {
          const unsigned long long tk = key[e];
          const unsigned ti = idx[e];
          key[e] = key[b];
          idx[e] = idx[b];
          key[b] = tk;
          idx[b] = ti;
        }
      }
    }
  }
}

// Orders the len <= 32 * E rows at order.
template <int E>
__device__ __forceinline__ void warp_order(unsigned* order, unsigned len, const unsigned long long* key, int lane) {
  unsigned long long k[E];
  unsigned idx[E];
#pragma unroll
  for (int e = 0; e < E; ++e) idx[e] = (unsigned)(e * 32 + lane) < len ? order[e * 32 + lane] : 0xffffffffu;
#pragma unroll
  for (int e = 0; e < E; ++e) k[e] = idx[e] != 0xffffffffu ? key[idx[e]] : ~0ull;
  warp_sort<E>(k, idx, lane);
#pragma unroll
  for (int e = 0; e < E; ++e)
    if ((unsigned)(lane * E + e) < len) order[lane * E + e] = idx[e];
}

// Bitonic sort of size (a power of two) entries by a block; 32 consecutive
// compare pairs span 64 entries, so steps of at most 32 stay within one warp's
// entries.
__device__ __forceinline__ void block_sort(unsigned long long* key, unsigned* idx, unsigned size) {
  for (unsigned k = 2; k <= size; k <<= 1) {
    for (unsigned j = k >> 1; j > 0; j >>= 1) {
      for (unsigned p = threadIdx.x; p < size / 2; p += kTileThreads) {
        const unsigned a = 2u * p - (p & (j - 1u)), b = a + j;
        const unsigned long long ka = key[a], kb = key[b];
        const unsigned ia = idx[a], ib = idx[b];
        if (entry_less(kb, ib, ka, ia) == ((a & k) == 0u)) {
          key[a] = kb;
          key[b] = ka;
          idx[a] = ib;
          idx[b] = ia;
        }
      }
      if (j > 32u) __syncthreads();
      else __syncwarp();
    }
    __syncthreads();
  }
}

// The next group of a warp: groups differ by a factor of hundreds in size, so
// warps draw them (the draw for the next one travels while one is worked on).
struct GroupDraw {
  unsigned* next;
  unsigned drawn;
  __device__ __forceinline__ GroupDraw(unsigned* n, int lane) : next(n), drawn(0u) { draw(lane); }
  __device__ __forceinline__ void draw(int lane) {
    if (lane == 0) drawn = atomicAdd(next, 1u);
  }
  __device__ __forceinline__ unsigned take(int lane) {
    const unsigned g = __shfl_sync(0xffffffffu, drawn, 0);
    draw(lane);
    return g;
  }
};

// order: rows by (query id, index) in, by (query id, key, index) out.
__global__ void __launch_bounds__(kThreads) order_small_kernel(long long n, unsigned* order, DenseLayout L) {
  const int lane = threadIdx.x & 31;
  const unsigned G = (unsigned)L.acc->n_groups;
  GroupDraw draw(&L.acc->next[0], lane);
  for (unsigned g = draw.take(lane); g < G; g = draw.take(lane)) {
    const unsigned begin = L.g_start[g];
    const unsigned len = (g + 1 < G ? L.g_start[g + 1] : (unsigned)n) - begin;
    if (len < 2u) continue;
    if (len > (unsigned)kWarpRows) {
      if (lane == 0) {
        const unsigned tiles = (len + kTileRows - 1) / kTileRows;
        const unsigned at = atomicAdd(&L.acc->n_tiles, tiles);
        for (unsigned k = 0; k < tiles; ++k)
          L.tiles[at + k] = Tile{begin + k * kTileRows, min(kTileRows, len - k * kTileRows) | (tiles > 1u ? kTileMerged : 0u)};
        if (len > kTileRows) {
          const unsigned long long b = atomicAdd(&L.acc->big, (1ull << 32) | len);
          L.big_start[b >> 32] = begin;
          L.big_at[b >> 32] = (unsigned)b;
          atomicMax(&L.acc->longest, len);
        }
      }
      continue;
    }
    if (len <= 32u) warp_order<1>(order + begin, len, L.key[0], lane);
    else if (len <= 64u) warp_order<2>(order + begin, len, L.key[0], lane);
    else if (len <= 128u) warp_order<4>(order + begin, len, L.key[0], lane);
    else warp_order<8>(order + begin, len, L.key[0], lane);
  }
}

struct OrderBuffer {
  unsigned long long* key;
  unsigned* idx;
};
// What a round reads: the last one writes (key[1], order), and they alternate.
__device__ __forceinline__ OrderBuffer merge_buffer(const DenseLayout& L, unsigned* order, int rounds, int round) {
  if (((rounds - round) & 1) == 0) return OrderBuffer{L.key[1], order};
  return OrderBuffer{L.qkey[0], L.idx[1]};
}

// One block per tile; tiles to be merged go where the first round reads, with their keys.
__global__ void __launch_bounds__(kTileThreads) order_tile_kernel(unsigned* order, DenseLayout L) {
  extern __shared__ __align__(16) unsigned char tile_raw[];
  unsigned long long* key = reinterpret_cast<unsigned long long*>(tile_raw);
  unsigned* idx = reinterpret_cast<unsigned*>(tile_raw + kTileRows * 8);
  const unsigned n = L.acc->n_tiles;
  const OrderBuffer merged = merge_buffer(L, order, merge_rounds(kTileRows, L.acc->longest), 0);
  for (unsigned t = blockIdx.x; t < n; t += gridDim.x) {
    const Tile tile = L.tiles[t];
    const unsigned len = tile.len & ~kTileMerged;
    unsigned size = 2u;
    while (size < len) size <<= 1;
    for (unsigned e = threadIdx.x; e < size; e += kTileThreads) {
      const unsigned j = e < len ? order[tile.start + e] : 0xffffffffu;
      idx[e] = j;
      key[e] = e < len ? L.key[0][j] : ~0ull;
    }
    __syncthreads();
    block_sort(key, idx, size);
    const bool merge = (tile.len & kTileMerged) != 0u;
    for (unsigned e = threadIdx.x; e < len; e += kTileThreads) {
      if (merge) merged.key[tile.start + e] = key[e];
      (merge ? merged.idx : order)[tile.start + e] = idx[e];
    }
    __syncthreads();
  }
}

// One round over the groups of more than one tile (run_merge.cuh).
__global__ void __launch_bounds__(kThreads) order_merge_kernel(unsigned* order, DenseLayout L, int round) {
  pdl_wait();
  pdl_trigger();
  const int rounds = merge_rounds(kTileRows, L.acc->longest);
  if (round >= rounds) return;
  const unsigned long long big = L.acc->big;
  const unsigned n_big = (unsigned)(big >> 32), rows = (unsigned)big;
  const OrderBuffer from = merge_buffer(L, order, rounds, round), to = merge_buffer(L, order, rounds, round + 1);
  const unsigned width = merge_width(kTileRows, round);
  for (unsigned v0 = blockIdx.x * kThreads; v0 < rows; v0 += gridDim.x * kThreads) {
    const bool live = v0 + threadIdx.x < rows;
    const unsigned v = min(v0 + threadIdx.x, rows - 1u);
    unsigned g = 0u, hi = n_big - 1u;
    while (g < hi) {
      const unsigned mid = (g + hi + 1u) >> 1;
      if (L.big_at[mid] <= v) g = mid;
      else hi = mid - 1u;
    }
    const unsigned at = L.big_at[g], len = (g + 1u < n_big ? L.big_at[g + 1u] : rows) - at, a = v - at;
    const unsigned own = a / width, run0 = own / kMergeRuns * kMergeRuns, first = L.big_start[g] + run0 * width;
    const unsigned long long* key = from.key + first;
    const unsigned* idx = from.idx + first;
    const unsigned long long my_key = key[a - run0 * width];
    const unsigned my_idx = idx[a - run0 * width];
    unsigned n[kMergeRuns];
#pragma unroll
    for (unsigned k = 0; k < kMergeRuns; ++k) {
      const unsigned long long begin = (unsigned long long)(run0 + k) * width;  // in the group
      n[k] = run0 + k == own || begin >= len ? 0u : (unsigned)min((unsigned long long)width, len - begin);
    }
    const unsigned g0 = __shfl_sync(0xffffffffu, g, 0), own0 = __shfl_sync(0xffffffffu, own, 0);
    const bool together = __all_sync(0xffffffffu, live && g == g0 && own == own0);
    const unsigned place =
        first + (a - own * width) +
        entries_before(width, n, my_key, my_idx, together, [&](unsigned k, unsigned p, unsigned long long x, unsigned i) {
          const unsigned long long other = key[k * width + p];
          return other < x || (other == x && idx[k * width + p] < i);
        });
    if (!live) continue;
    to.key[place] = my_key;
    to.idx[place] = my_idx;
  }
}

// Asynchronous copy of a row to shared memory, and the wait for all but the
// newest kAhead groups of them.
constexpr int kAhead = 3;
__device__ __forceinline__ void copy_row(WalkRow* to, const WalkRow* from) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(to);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n\tcp.async.ca.shared.global [%2], [%3], 16;" ::"r"(dst),
               "l"(from), "r"(dst + 16u), "l"(reinterpret_cast<const char*>(from) + 16)
               : "memory");
}
__device__ __forceinline__ void commit_rows() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void wait_rows() { asm volatile("cp.async.wait_group %0;" ::"n"(kAhead) : "memory"); }

// One warp per group: the walk of group_scheduler.cpp:116-232.  Rows are read
// through the order; every slot of the group's terms is written.  Bound by the
// chain of dependent additions of the two sums, so both run side by side over
// all 32 lanes (rows that add nothing add +0.0), and by the rows' latency in
// long groups, so the next three steps' rows are on their way to shared memory
// while one is worked on: one group of a million rows 28.3 -> 14.2 ms, 1 M rows
// in groups of up to 256 unchanged (their walk and the gather of sorted costs
// before it took 99 us, now 43).
__global__ void __launch_bounds__(kThreads, 4) group_kernel(const unsigned* order, long long n, unsigned limit,
                                                         double penalty, DenseLayout L) {
  __shared__ unsigned long long s_ctr[kNumCounters];
  __shared__ double2 s_add[kThreads / 32][32];
  __shared__ WalkRow s_rows[kThreads / 32][kAhead + 1][32];
  if (threadIdx.x < kNumCounters) s_ctr[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned G = (unsigned)L.acc->n_groups;
  double2* add = s_add[threadIdx.x >> 5];
  WalkRow(*ahead)[32] = s_rows[threadIdx.x >> 5];
  unsigned c[kNumCounters] = {};  // none exceeds 2 n < 2^30
  // slots past the last group's: the compaction runs over 3 n
  for (long long i = 2 * n + G + (long long)blockIdx.x * kThreads + threadIdx.x; i < 3 * n;
       i += (long long)gridDim.x * kThreads)
    L.terms[i] = 0.0;
  GroupDraw draw(&L.acc->next[1], lane);
  for (unsigned g = draw.take(lane); g < G; g = draw.take(lane)) {
    const unsigned begin = L.g_start[g];
    const unsigned end = g + 1 < G ? L.g_start[g + 1] : (unsigned)n;
    const unsigned slot0 = 2 * begin + g;  // this group's 2 * size + 1 term slots
    double gfull = 0.0, wbfp = 0.0, gcost = 0.0, last_term = 0.0;
    bool truth = false, predicted = false;
    int state = 0;  // 0 proposals, 1 full fallback, 2 resolved
    unsigned rank = 0;
    unsigned calls = 0, fallback = 0, hits = 0, misses = 0;
    bool high_group = false;
    // step k's rows go to place k mod kAhead + 1, each lane's to its own slot
    unsigned moved = 0u, j[kAhead + 1];
    auto fetch = [&](unsigned pos, unsigned row) {
      if (pos < end) {
        copy_row(&ahead[(pos - begin) / 32u % (kAhead + 1)][lane], L.rows + row);
        moved += row != pos ? 1u : 0u;
      }
      commit_rows();
    };
#pragma unroll
    for (int k = 0; k <= kAhead; ++k) j[k] = begin + 32u * k + lane < end ? order[begin + 32u * k + lane] : 0u;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) fetch(begin + 32u * k + lane, j[k]);
    unsigned next = j[kAhead];
    for (unsigned base = begin; base < end; base += 32) {
      const unsigned pos = base + lane;
      const int nvalid = (int)min(32u, end - base);
      const bool in = lane < nvalid;
      fetch(pos + 32u * kAhead, next);
      next = pos + 32u * (kAhead + 1) < end ? order[pos + 32u * (kAhead + 1)] : 0u;
      wait_rows();
      double f = 0.0, nr = 0.0;
      unsigned fl = 0;
      if (in) {
        const WalkRow r = ahead[(base - begin) / 32u % (kAhead + 1)][lane];
        f = r.full;
        nr = r.narrow;
        fl = (unsigned)r.flags;
      }
      const unsigned my_slot = slot0 + 2 * (pos - begin);
      truth = truth || __any_sync(0xffffffffu, fl & kColl);
      int from = 0;
      double term0 = 0.0, term1 = 0.0, w = 0.0;  // this row's terms; what it adds to the cost before a hit
      bool cost_here = false;                     // the group's cost is the sum so far plus `extra`s
      double extra0 = 0.0, extra1 = 0.0;
      if (state == 0) {
        const unsigned attempts = pos - begin + 1;
        const bool stop = in && ((fl & kHighUnc) || ((fl & kColl) && ((fl & kOverlap) || attempts >= limit)));
        const unsigned m = __ballot_sync(0xffffffffu, stop);
        const int t = m ? __ffs(m) - 1 : nvalid;
        const bool pre = lane < t;
        if (pre) {  // narrow call; a colliding miss adds its penalty
          term0 = nr;
          w = nr;
          if (fl & kColl) {
            term1 = f * penalty;
            w = nr + term1;
          }
        }
        calls += (unsigned)t;
        misses += __popc(__ballot_sync(0xffffffffu, pre && (fl & kColl)));
        if (m) {
          const unsigned sfl = __shfl_sync(0xffffffffu, fl, t);
          const double snr = __shfl_sync(0xffffffffu, nr, t);
          const double sf = __shfl_sync(0xffffffffu, f, t);
          rank = base + t - begin + 1;
          if (sfl & kHighUnc) {
            state = 1;
            from = t;
            high_group = true;
          } else if (sfl & kOverlap) {  // a hit inside the predicted interval
            if (lane == t) term0 = snr;
            calls += 1;
            hits += 1;
            cost_here = true;
            extra0 = snr;
            predicted = true;
            state = 2;
          } else {  // a miss at the attempt limit: penalty, then one full fallback call
            if (lane == t) {
              term0 = snr;
              term1 = sf * penalty;
            }
            last_term = sf;
            calls += 2;
            fallback += 1;
            misses += 1;
            cost_here = true;
            extra0 = snr;
            extra1 = sf;
            predicted = true;
            state = 2;
          }
        }
      }
      if (state == 1) {  // full fallback from lane `from` to the first colliding candidate
        const bool fb = in && lane >= from;
        const unsigned m = __ballot_sync(0xffffffffu, fb && (fl & kColl));
        const int q = m ? __ffs(m) - 1 : nvalid;
        const int last = m ? q + 1 : nvalid;
        if (fb && lane < last) term0 = f;
        if (fb && lane < q) w = f;
        calls += (last - from);
        fallback += (last - from);
        if (m) {
          const double qf = __shfl_sync(0xffffffffu, f, q);
          rank = base + q - begin + 1;
          cost_here = true;
          extra0 = qf;
          predicted = true;
          state = 2;
        }
      }
      if (in) {
        L.terms[my_slot] = term0;
        L.terms[my_slot + 1] = term1;
      }
      add[lane] = make_double2(f, w);
      __syncwarp();
      for (int j0 = 0; j0 < nvalid; j0 += 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const double2 a = add[j0 + j];
          gfull += a.x;
          wbfp += a.y;
        }
      }
      __syncwarp();
      if (cost_here) gcost = (wbfp + extra0) + extra1;
    }
    c[kReordered] += __reduce_add_sync(0xffffffffu, moved);
    if (lane == 0) {
      L.terms[slot0 + 2 * (end - begin)] = last_term;
      L.g_full[g] = gfull;
      L.g_cost[g] = predicted ? gcost : 0.0;
      c[kGroups] += 1;
      c[kPositive] += truth ? 1 : 0;
      c[kCalls] += calls;
      c[kFallback] += fallback;
      c[kHit] += hits;
      c[kMiss] += misses;
      c[kTP] += (truth && predicted) ? 1 : 0;
      c[kTN] += (!truth && !predicted) ? 1 : 0;
      c[kFP] += (!truth && predicted) ? 1 : 0;
      c[kFN] += (truth && !predicted) ? 1 : 0;
      c[kHighUncGroups] += high_group ? 1 : 0;
      c[kRankSum] += predicted ? rank : 0;
    }
  }
  if (lane == 0)
    for (int k = 0; k < kNumCounters; ++k)
      if (c[k]) atomicAdd(&s_ctr[k], (unsigned long long)c[k]);
  __syncthreads();
  if (threadIdx.x < kNumCounters && s_ctr[threadIdx.x]) atomicAdd(&L.acc->ctr[threadIdx.x], s_ctr[threadIdx.x]);
}

struct FoldJob {
  const double* src[3];
  const int* count[3];  // device counts
  double* out[3];
};

// ---- the ordered fold ------------------------------------------------------
//
// A sum s of non-negative doubles, added one term at a time in a fixed order
// with round-to-nearest-even, reproduced exactly with block-wide scans.
// While s stays below the top of its binade, s = S * u with u its unit in the
// last place and S an integer below 2^53, and adding a term x gives
// S + floor(x / u) + r, where r = 1 when the remainder of x / u is above one
// half, 0 below, and on an exact half the bit that makes the result even:
// r depends on S only through its parity.  Each term is therefore a pair of
// increments (for an even and for an odd S), pairs compose associatively
// ((a then b)[p] = a[p] + b[(p + a[p]) mod 2]), and a block scan gives every
// term the S in front of it.  The first term whose exact sum could reach the
// top of the binade (or an infinite term) is added with the hardware DADD;
// the fold then continues from it in the new binade.
// Each such step at least doubles s, so there are at most a few dozen of
// them.  A zero-start sum takes its first non-zero term exactly.

constexpr unsigned long long kTwo53 = 1ull << 53;

struct IncPair {
  unsigned long long e, o;  // increments of S for an even / an odd S
};

__device__ __forceinline__ IncPair compose(const IncPair& a, const IncPair& b) {  // a, then b
  IncPair c;
  c.e = a.e + ((a.e & 1ull) ? b.o : b.e);
  c.o = a.o + ((a.o & 1ull) ? b.e : b.o);
  return c;
}

__device__ __forceinline__ IncPair shfl_up_pair(const IncPair& v, int o) {
  IncPair r;
  r.e = __shfl_up_sync(0xffffffffu, v.e, o);
  r.o = __shfl_up_sync(0xffffffffu, v.o, o);
  return r;
}

__device__ __forceinline__ IncPair warp_inclusive(IncPair v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const IncPair up = shfl_up_pair(v, o);
    if (lane >= o) v = compose(up, v);
  }
  return v;
}

// The exponent of the last place of a positive double.
__device__ __forceinline__ int ulp_of(double s) { return max(ilogb(s), -1022) - 52; }

// What a term of q units adds to an even and to an odd S.
__device__ __forceinline__ IncPair term_increments(double q) {
  const double mf = floor(q);
  const double f = q - mf;
  const unsigned long long m = (unsigned long long)mf;
  const bool above = f > 0.5, tie = f == 0.5;
  IncPair c;
  c.e = m + (above ? 1ull : (tie ? (m & 1ull) : 0ull));
  c.o = m + (above ? 1ull : (tie ? ((m + 1ull) & 1ull) : 0ull));
  return c;
}

struct FoldShared {
  unsigned long long we[32], wo[32];
  double s;
  int first;
};

// x * 2^-ue as two exact factors (2^1074 alone is not a double).  A product
// that underflows is far below one half of a unit, one that overflows far above
// the binade.
struct UnitScale {
  double a, b;
  __device__ __forceinline__ explicit UnitScale(int ue) : a(ldexp(1.0, -ue / 2)), b(ldexp(1.0, -ue - -ue / 2)) {}
  __device__ __forceinline__ double operator()(double x) const { return x * a * b; }
};

// Adds the terms [begin, end) to sh.s; every thread of the block takes part.
// The terms of a chunk stay in registers over its binade steps, those already
// added count as zero.  Returns early when the sum is infinite.
__device__ __forceinline__ void fold_range(FoldShared& sh, const double* src, long long begin, long long end) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const IncPair zero{0ull, 0ull};
  double x[kFoldPerThread], nx[kFoldPerThread];
#pragma unroll
  for (int k = 0; k < kFoldPerThread; ++k) {
    const long long i = begin + t * kFoldPerThread + k;
    nx[k] = i < end ? src[i] : 0.0;
  }
  for (long long base = begin; base < end; base += kFoldChunk) {
    const int chunk = (int)min((long long)kFoldChunk, end - base);
#pragma unroll
    for (int k = 0; k < kFoldPerThread; ++k) {
      x[k] = nx[k];
      const long long i = base + kFoldChunk + t * kFoldPerThread + k;
      nx[k] = i < end ? src[i] : 0.0;
    }
    int start = 0;  // terms of the chunk already added
    while (start < chunk) {
      const double s = sh.s;
      if (isinf(s)) return;
      // the sum grows about linearly, so the next binade step is about as many
      // terms away as have been added: do not look much further
      const int len = (int)min((long long)chunk, start + max(256ll, base + start));
      if (t == 0) sh.first = len;
      __syncthreads();  // everyone read s; first is reset
      if (s == 0.0) {   // 0 + x == x: the first non-zero term starts the sum
        int mine = len;
#pragma unroll
        for (int k = kFoldPerThread - 1; k >= 0; --k) {
          const int i = t * kFoldPerThread + k;
          if (i >= start && i < len && x[k] != 0.0) mine = i;
        }
        if (mine < len) atomicMin(&sh.first, mine);
        __syncthreads();
        const int f = sh.first;
#pragma unroll
        for (int k = 0; k < kFoldPerThread; ++k)
          if (f < len && t * kFoldPerThread + k == f) sh.s = x[k];
        start = min(f + 1, len);
        __syncthreads();
        continue;
      }
      const int ue = ulp_of(s);
      const UnitScale units(ue);
      const unsigned long long S = (unsigned long long)units(s);
      IncPair inc[kFoldPerThread];
      unsigned long long m[kFoldPerThread];
      bool big[kFoldPerThread];
      IncPair incl = zero;
      const bool idle = (w + 1) * 32 * kFoldPerThread <= start || w * 32 * kFoldPerThread >= len;  // a whole warp
      if (!idle) {
        IncPair local = zero;
#pragma unroll
        for (int k = 0; k < kFoldPerThread; ++k) {
          const int i = t * kFoldPerThread + k;
          const double q = i >= start && i < len ? units(x[k]) : 0.0;
          big[k] = !(q < 9007199254740992.0);
          m[k] = 0;
          if (big[k]) {
            inc[k] = IncPair{kTwo53, kTwo53};  // never applied: the binade step comes first
          } else {
            m[k] = (unsigned long long)floor(q);
            inc[k] = term_increments(q);
          }
          local = compose(local, inc[k]);
        }
        incl = warp_inclusive(local, lane);
      }
      if (lane == 31) {
        sh.we[w] = incl.e;
        sh.wo[w] = incl.o;
      }
      __syncthreads();
      if (w == 0) {
        const IncPair v = warp_inclusive(lane < kFoldWarps ? IncPair{sh.we[lane], sh.wo[lane]} : zero, lane);
        IncPair ex = shfl_up_pair(v, 1);
        if (lane == 0) ex = zero;
        __syncwarp();
        sh.we[lane] = ex.e;
        sh.wo[lane] = ex.o;
      }
      __syncthreads();
      IncPair ein = shfl_up_pair(incl, 1);
      if (lane == 0) ein = zero;
      const IncPair wp{sh.we[w], sh.wo[w]};
      const IncPair ex = compose(wp, ein);
      unsigned long long P = S + ((S & 1ull) ? ex.o : ex.e);
      int mine = len;
      unsigned long long P_at = 0;
      if (!idle) {
#pragma unroll
        for (int k = 0; k < kFoldPerThread; ++k) {
          const bool in = t * kFoldPerThread + k < len;
          if (in && mine == len) {
            if (big[k] || P >= kTwo53 || P + m[k] >= kTwo53) {
              mine = t * kFoldPerThread + k;
              P_at = P;
            } else {
              P += (P & 1ull) ? inc[k].o : inc[k].e;
            }
          }
        }
      }
      if (mine < len) atomicMin(&sh.first, mine);
      __syncthreads();
      const int c = sh.first;
      if (c == len) {  // no binade step: the last thread holds the end of the chunk
        if (t == (len - 1) / kFoldPerThread) sh.s = ldexp((double)P, ue);
      } else if (mine == c) {
#pragma unroll
        for (int k = 0; k < kFoldPerThread; ++k)
          if (t * kFoldPerThread + k == c) sh.s = ldexp((double)P_at, ue) + x[k];
      }
      start = min(c + 1, len);
      __syncthreads();
    }
  }
}

// One block per total, its terms straight through.
__global__ void __launch_bounds__(kFoldThreads) fold_kernel(const double* src, long long cnt, double* out) {
  __shared__ FoldShared sh;
  if (threadIdx.x == 0) sh.s = 0.0;
  __syncthreads();
  fold_range(sh, src, 0, cnt);
  if (threadIdx.x == 0) *out = sh.s;
}

// The three totals of a replay, pieces of kFoldChunk terms on all SMs.  What a
// piece adds to the sum is a pair of increments once the sum's binade is
// known, and the sum of all terms before the piece, added in any order,
// predicts it.  One block per total then strings the pieces together: 512 at a
// time by a scan of their pairs, up to the first one whose prediction was
// wrong or in which the sum leaves its binade; that one is folded term by
// term.  Exact whatever the prediction.  The straight fold is a chain of one
// 4,096-term chunk after the other: 221 us for the three totals of 1 M rows,
// now 106.
__device__ __forceinline__ long long job_count(const FoldJob& job, int b) {
  const int* cp = b == 0 ? job.count[0] : (b == 1 ? job.count[1] : job.count[2]);
  return (long long)*cp;
}

// Sums of the pieces; the last block of a total turns them into the binade in
// front of each piece.
__global__ void __launch_bounds__(kFoldThreads) piece_sum_kernel(FoldJob job, FoldPieces pc, DenseAcc* acc) {
  __shared__ double warp_sum[kFoldWarps], carry;
  __shared__ bool last;
  const int b = blockIdx.y, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const double* src = b == 0 ? job.src[0] : (b == 1 ? job.src[1] : job.src[2]);
  double* sum = b == 0 ? pc.sum[0] : (b == 1 ? pc.sum[1] : pc.sum[2]);
  int* ulp = b == 0 ? pc.ulp[0] : (b == 1 ? pc.ulp[1] : pc.ulp[2]);
  const long long cnt = job_count(job, b), pieces = (cnt + kFoldChunk - 1) / kFoldChunk;
  for (long long c = blockIdx.x; c < pieces; c += gridDim.x) {
    const long long base = c * kFoldChunk;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kFoldPerThread; ++k) {
      const long long i = base + k * kFoldThreads + t;
      s += i < cnt ? src[i] : 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) warp_sum[w] = s;
    __syncthreads();
    if (t == 0) {
      double v = 0.0;
      for (int k = 0; k < kFoldWarps; ++k) v += warp_sum[k];
      sum[c] = v;
    }
    __syncthreads();
  }
  __threadfence();
  __syncthreads();
  if (t == 0) {
    last = atomicAdd(&acc->fold_blocks[b], 1u) == gridDim.x - 1;
    carry = 0.0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (long long c0 = 0; c0 < pieces; c0 += kFoldThreads) {
    const double v = c0 + t < pieces ? __ldcg(sum + c0 + t) : 0.0;
    double incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    double before = carry;
    for (int k = 0; k < w; ++k) before += warp_sum[k];
    double ex = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) ex = 0.0;
    if (c0 + t < pieces) ulp[c0 + t] = ulp_of(before + ex);
    __syncthreads();
    if (t == kFoldThreads - 1) carry = before + incl;
    __syncthreads();
  }
}

// The increments of each piece in its predicted binade; ~0 for both when a
// term is too large for their 64-bit counts (then the sum soon leaves the
// binade anyway).
__global__ void __launch_bounds__(kFoldThreads) piece_inc_kernel(FoldJob job, FoldPieces pc) {
  __shared__ IncPair warp_inc[kFoldWarps];
  const int b = blockIdx.y, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const double* src = b == 0 ? job.src[0] : (b == 1 ? job.src[1] : job.src[2]);
  const int* ulp = b == 0 ? pc.ulp[0] : (b == 1 ? pc.ulp[1] : pc.ulp[2]);
  ulonglong2* out = b == 0 ? pc.inc[0] : (b == 1 ? pc.inc[1] : pc.inc[2]);
  const long long cnt = job_count(job, b), pieces = (cnt + kFoldChunk - 1) / kFoldChunk;
  for (long long c = blockIdx.x; c < pieces; c += gridDim.x) {
    const long long base = c * kFoldChunk + t * kFoldPerThread;
    const UnitScale units(ulp[c]);
    IncPair local{0ull, 0ull};
    bool big = false;
#pragma unroll
    for (int k = 0; k < kFoldPerThread; ++k) {
      const double q = units(base + k < cnt ? src[base + k] : 0.0);
      if (!(q < 2251799813685248.0)) big = true;  // 2^51: 4096 of them stay below 2^64
      else local = compose(local, term_increments(q));
    }
    const IncPair incl = warp_inclusive(local, lane);
    if (lane == 31) warp_inc[w] = incl;
    big = __syncthreads_or(big);
    if (w == 0) {
      const IncPair v = warp_inclusive(lane < kFoldWarps ? warp_inc[lane] : IncPair{0ull, 0ull}, lane);
      if (lane == 31) out[c] = big ? make_ulonglong2(~0ull, ~0ull) : make_ulonglong2(v.e, v.o);
    }
    __syncthreads();
  }
}

// One block per total.
__global__ void __launch_bounds__(kFoldThreads) piece_fold_kernel(FoldJob job, FoldPieces pc) {
  __shared__ FoldShared sh;
  const int b = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const double* src = b == 0 ? job.src[0] : (b == 1 ? job.src[1] : job.src[2]);
  const int* ulp = b == 0 ? pc.ulp[0] : (b == 1 ? pc.ulp[1] : pc.ulp[2]);
  const ulonglong2* inc = b == 0 ? pc.inc[0] : (b == 1 ? pc.inc[1] : pc.inc[2]);
  const long long cnt = job_count(job, b), pieces = (cnt + kFoldChunk - 1) / kFoldChunk;
  const IncPair zero{0ull, 0ull};
  if (t == 0) sh.s = 0.0;
  __syncthreads();
  long long c = 0;  // pieces added
  while (c < pieces && !isinf(sh.s)) {
    const double s = sh.s;
    const int avail = (int)min((long long)kFoldThreads, pieces - c);
    int done = 0;
    if (s > 0.0) {
      const int ue = ulp_of(s);
      const unsigned long long S = (unsigned long long)UnitScale(ue)(s);
      bool fits = false;
      IncPair mine = zero;
      if (t < avail && ulp[c + t] == ue) {
        const ulonglong2 v = inc[c + t];
        fits = v.x < kTwo53 && v.y < kTwo53;
        if (fits) mine = IncPair{v.x, v.y};
      }
      if (t == 0) sh.first = avail;
      const IncPair incl = warp_inclusive(mine, lane);
      if (lane == 31) {
        sh.we[w] = incl.e;
        sh.wo[w] = incl.o;
      }
      __syncthreads();
      if (w == 0) {
        const IncPair v = warp_inclusive(lane < kFoldWarps ? IncPair{sh.we[lane], sh.wo[lane]} : zero, lane);
        IncPair ex = shfl_up_pair(v, 1);
        if (lane == 0) ex = zero;
        __syncwarp();
        sh.we[lane] = ex.e;
        sh.wo[lane] = ex.o;
      }
      __syncthreads();
      IncPair ein = shfl_up_pair(incl, 1);
      if (lane == 0) ein = zero;
      const IncPair ex = compose(IncPair{sh.we[w], sh.wo[w]}, ein);
      const unsigned long long P = S + ((S & 1ull) ? ex.o : ex.e);  // right up to the first piece that fails
      // the sum never falls, so a piece stays in the binade iff it ends in it
      const bool ok = fits && P < kTwo53 && P + ((P & 1ull) ? mine.o : mine.e) < kTwo53;
      if (t < avail && !ok) atomicMin(&sh.first, t);
      __syncthreads();
      done = sh.first;
      if (done > 0 && t == done - 1) {
        const unsigned long long end = P + ((P & 1ull) ? mine.o : mine.e);
        sh.s = ldexp((double)end, ue);
      }
      __syncthreads();
    }
    c += done;
    if (done < avail) {
      fold_range(sh, src, c * kFoldChunk, min(cnt, (c + 1) * kFoldChunk));
      ++c;
    }
  }
  if (t == 0) *(b == 0 ? job.out[0] : (b == 1 ? job.out[1] : job.out[2])) = sh.s;
}

__global__ void finish_kernel(long long n, DenseLayout L, p2c_dense_group_stats* st) {
  if (threadIdx.x != 0) return;
  const unsigned long long* c = L.acc->ctr;
  st->candidate_count = (unsigned long long)n;
  st->group_count = c[kGroups];
  st->positive_group_count = c[kPositive];
  st->no_proposal_exact_calls = (unsigned long long)n;
  st->learned_exact_calls = c[kCalls];
  st->learned_fallback_calls = c[kFallback];
  st->learned_interval_hit_count = c[kHit];
  st->learned_interval_miss_count = c[kMiss];
  st->first_positive_rank_sum = (double)c[kRankSum];
  st->tp = c[kTP];
  st->tn = c[kTN];
  st->fp = c[kFP];
  st->fn = c[kFN];
  st->reordered_count = c[kReordered];
  st->high_uncertainty_group_count = c[kHighUncGroups];
  const unsigned long long e = L.acc->first_error;
  st->error_row = e == ~0ull ? -1 : (long long)(e >> 2);
  st->error_kind = e == ~0ull ? 0 : (int)(e & 3);
  st->pad = 0;
}

int grid_for(long long n) { return (int)std::max(1ll, (n + kThreads - 1) / kThreads); }

}  // namespace
}  // namespace p2c

extern "C" {

size_t p2c_dense_group_early_stop_workspace_bytes(int64_t n) {
  if (n < 0) return 0;
  return p2c::carve(nullptr, n).total + 256;
}

int p2c_dense_group_early_stop(int64_t n, const uint64_t* query_id_dev, const uint64_t* candidate_id_dev,
                               const float* cost_target_dev, const double* oracle_trace_dev,
                               const float* interval_scores_dev, const float* priority_score_dev,
                               const float* cost_score_dev, const float* uncertainty_score_dev,
                               const p2c_dense_group_config* config, p2c_dense_group_stats* stats_dev,
                               void* workspace_dev, size_t workspace_bytes, void* stream) {
  using namespace p2c;
  if (config == nullptr) return fail(P2C_ERR_INVALID, "dense group config pointer is null");
  if (stats_dev == nullptr) return fail(P2C_ERR_INVALID, "DenseGroupEarlyStopStats pointer is null");
  if (config->representative_attempt_limit == 0u)
    return fail(P2C_ERR_INVALID, "representative_attempt_limit must be positive");
  if (!std::isfinite(config->uncertainty_fallback_threshold) || config->uncertainty_fallback_threshold < 0.0f)
    return fail(P2C_ERR_INVALID, "uncertainty_fallback_threshold must be finite and non-negative");
  if (!std::isfinite(config->interval_miss_penalty_scale) || config->interval_miss_penalty_scale < 0.0)
    return fail(P2C_ERR_INVALID, "interval_miss_penalty_scale must be finite and non-negative");
  if (n < 0 || n >= (1ll << 29))  // the 3n work-term slots are counted in int by the compaction
    return fail(P2C_ERR_INVALID, "row count must lie in [0, 2^29)");
  if (n > 0 && (query_id_dev == nullptr || candidate_id_dev == nullptr || cost_target_dev == nullptr ||
                oracle_trace_dev == nullptr || interval_scores_dev == nullptr || priority_score_dev == nullptr ||
                cost_score_dev == nullptr || uncertainty_score_dev == nullptr))
    return fail(P2C_ERR_INVALID, "input pointer is null");
  const int qbits = config->query_bits <= 0 || config->query_bits > 64 ? 64 : config->query_bits;
  const size_t need = carve(nullptr, n).total;
  if (workspace_dev == nullptr || workspace_bytes < need)
    return fail(P2C_ERR_INVALID, "dense group workspace too small: %zu < %zu bytes", workspace_bytes, need);
  // 16-byte records: the size that callers are told has room for this
  char* base = reinterpret_cast<char*>(((uintptr_t)workspace_dev + 15) & ~(uintptr_t)15);
  if ((size_t)(base - static_cast<char*>(workspace_dev)) + need > workspace_bytes)
    return fail(P2C_ERR_INVALID, "dense group workspace too small: %zu < %zu bytes", workspace_bytes, need + 16);
  DenseLayout L = carve(base, n);
  cudaStream_t s = as_stream(stream);
  init_kernel<<<1, 32, 0, s>>>(L);
  P2C_CUDA(cudaMemsetAsync(stats_dev, 0, sizeof(p2c_dense_group_stats), s));
  if (n > 0) {
    const ParseIn in{reinterpret_cast<const unsigned long long*>(query_id_dev),
                     reinterpret_cast<const unsigned long long*>(candidate_id_dev),
                     cost_target_dev,
                     oracle_trace_dev,
                     interval_scores_dev,
                     priority_score_dev,
                     cost_score_dev,
                     uncertainty_score_dev};
    const int keep = config->preserve_input_order ? 1 : 0;
    parse_kernel<<<grid_for(n), kThreads, 0, s>>>(in, n, config->uncertainty_fallback_threshold, keep, L);
    size_t tb = L.tmp_bytes;  // stable by query id
    unsigned* order = L.idx[2];
    P2C_CUDA(cub::DeviceRadixSort::SortPairs(L.tmp, tb, L.qkey[0], L.qkey[1], L.idx[0], order, (int)n, 0, qbits, s));
    tb = L.tmp_bytes;
    P2C_CUDA(cub::DeviceSelect::If(L.tmp, tb, thrust::counting_iterator<unsigned>(0u), L.g_start, &L.acc->n_groups,
                                   (int)n, IsHead{L.qkey[1]}, s));
    DeviceInfo info;
    if (int rc = current_device_info(&info)) return rc;
    const long long want = (n + (kThreads / 32) - 1) / (kThreads / 32);
    const int grid = (int)std::max(1ll, std::min(want, (long long)info.sm_count * 8));
    if (!keep) {  // priority desc, then cost asc, then index inside each group
      order_small_kernel<<<grid, kThreads, 0, s>>>(n, order, L);
      if (n > kWarpRows) {
        const size_t smem = kTileRows * 12;
        const int tiles = (int)std::min<long long>(n / kWarpRows + 1, info.sm_count * 4);
        order_tile_kernel<<<tiles, kTileThreads, smem, s>>>(order, L);
      }
      for (int round = 0; round < merge_rounds(kTileRows, (unsigned long long)n); ++round)
        P2C_CUDA(launch_pdl(order_merge_kernel, dim3((unsigned)info.sm_count * 4u), dim3(kThreads), 0, s, order, L,
                            round));
    }
    group_kernel<<<grid, kThreads, 0, s>>>(order, n, config->representative_attempt_limit,
                                           config->interval_miss_penalty_scale, L);
    FoldJob job{{L.compact, L.g_full, L.g_cost},
                {&L.acc->n_terms, &L.acc->n_groups, &L.acc->n_groups},
                {&stats_dev->learned_exact_work, &stats_dev->no_proposal_exact_work,
                 &stats_dev->cost_before_first_positive_sum}};
    tb = L.tmp_bytes;
    P2C_CUDA(cub::DeviceSelect::If(L.tmp, tb, L.terms, L.compact, &L.acc->n_terms, (int)(3 * n), NonZeroTerm{}, s));
    const dim3 pieces((unsigned)std::min<long long>((3 * n + kFoldChunk - 1) / kFoldChunk, info.sm_count * 4), 3);
    if (3 * n > kFoldChunk) {  // a first piece is folded term by term whatever its prediction
      piece_sum_kernel<<<pieces, kFoldThreads, 0, s>>>(job, L.pieces, L.acc);
      piece_inc_kernel<<<pieces, kFoldThreads, 0, s>>>(job, L.pieces);
    }
    piece_fold_kernel<<<3, kFoldThreads, 0, s>>>(job, L.pieces);
  }
  finish_kernel<<<1, 32, 0, s>>>(n, L, stats_dev);
  P2C_CUDA(cudaGetLastError());
  return P2C_OK;
}

int p2c_ordered_sum(const double* terms_dev, int64_t n, double* out_dev, void* stream) {
  using namespace p2c;
  if (n < 0) return fail(P2C_ERR_INVALID, "term count must be non-negative");
  if (out_dev == nullptr || (n > 0 && terms_dev == nullptr)) return fail(P2C_ERR_INVALID, "term or output pointer is null");
  fold_kernel<<<1, kFoldThreads, 0, as_stream(stream)>>>(terms_dev, n, out_dev);
  P2C_CUDA(cudaGetLastError());
  return P2C_OK;
}

}  // extern "C"
