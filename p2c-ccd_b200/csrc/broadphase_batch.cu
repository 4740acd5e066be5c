// broadphase_batch.cu — swept-AABB candidates of many scenes in one launch
// sequence.
//
// The column-subdivided sweep-and-prune of p2c_scene_candidates, segmented
// by scene so that a batch of N scenes costs about the launches of one
// scene instead of N times them (a 1,000-triangle scene alone is a chain of
// ~30 launches that each run for a few microseconds).  Primitives are
// indexed scene-major (scene s holds [P[s], P[s+1]): its vertices, faces,
// edges); every kernel finds a primitive's scene by binary search over P.
//   1. prep (one block): prefix offsets of primitives, vertices, pair
//      capacities and column tables per scene (minima are kept as
//      complemented keys, so the zeroed scratch starts empty);
//   2. vertex swept boxes: object envelopes and per-scene axis statistics
//      (block-level sums when a block holds one scene, warp-level otherwise);
//   3. every primitive's swept box, culled against the other objects'
//      envelopes; kept boxes appended to a compact list (often a few per cent
//      of the primitives), with per-scene, per-list extents;
//   4. one thread per scene: sweep axis, column grid (at most
//      max(64, n/4) cells for a scene of n primitives, 128 x 128 at most),
//      quantiser;
//   5. ONE radix sort, with the count read on the device, of the kept boxes'
//      keys (scene, list, column, 8-bit low field: the quantised min, with
//      the object bit of a two-body split; 24 + scene bits: 32-bit keys and 4
//      passes for up to 256 scenes, 64-bit keys beyond), a gather into one
//      struct-of-arrays in sorted order and per-scene column tables holding
//      sorted positions;
//   6. one sweep of both families over each scene's own columns, appending pairs as
//      (scene << w | packed pair), w the widest scene's packed pair, into a buffer of
//      the scenes' summed capacities (scene s owns its capacity's slice); windows of
//      large primitives are cut into pieces for a second launch;
//   7. ONE ordering of all pairs by rows (pair_rows.cuh), straight into each scene's
//      own buffer as (a << 32 | b), padded with ~0: every scene's list comes out
//      exactly as p2c_scene_candidates with sorted pairs writes it.
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <vector>

#include "broadphase.cuh"
#include "count_sort.cuh"
#include "pair_rows.cuh"

namespace p2c {

int validate_scene(const p2c_scene* sc);

namespace {

constexpr int kThreads = 256;
constexpr int kPrepThreads = 1024;
constexpr unsigned kFull = 0xffffffffu;
constexpr long long kMaxScenePrims = 1ll << 22;  // packed pairs of one scene stay below 2^44
#ifndef P2C_BATCH_QBITS
#define P2C_BATCH_QBITS 8
#endif
constexpr int kBatchQBits = P2C_BATCH_QBITS;     // quantiser of the batched key
constexpr unsigned kBatchQMax = (1u << kBatchQBits) - 1u;
constexpr int kBatchListShift = kCellBits + kBatchQBits;  // key: scene | list | column | quantised min
constexpr int kBatchSceneShift = kBatchListShift + 2;

inline unsigned grid_for(long long n, int threads) {
  const long long g = (n + threads - 1) / threads;
  return (unsigned)(g > 0 ? g : 1);
}

int bit_length(long long x) {
  int b = 0;
  while (x > 0) {
    ++b;
    x >>= 1;
  }
  return b;
}

__device__ __forceinline__ int bit_length_dev(long long x) { return x > 0 ? 64 - __clzll(x) : 0; }

// Cells of a scene's column grid per list: enough for the scene's size,
// never more than the single-scene grid.
__host__ __device__ inline long long cell_budget(long long n_prims) {
  long long c = n_prims / 4;
  if (c < 64) c = 64;
  if (c > (long long)kMaxColumns * kMaxColumns) c = (long long)kMaxColumns * kMaxColumns;
  return c;
}

struct Offsets {
  unsigned long long* prim;    // n + 1
  unsigned long long* vf_cap;  // n + 1
  unsigned long long* ee_cap;  // n + 1
  unsigned long long* cell;    // n + 1 (cells per list; a scene's tables are 3 x its budget)
  unsigned long long* vert;    // n + 1 (vertices)
  unsigned long long* edge;    // n + 1 (edges)
};

struct BatchBroad {
  const p2c_batch_scene* scenes;
  int n;
  Offsets off;
  BroadScratch* sc;          // n
  double* cbox;              // 6 x kept boxes, in compaction order
  unsigned* cprim;           // global primitive index of each kept box
  unsigned long long* keys[2];
  unsigned* keys32[2];       // the same buffers as 32-bit keys, used when key32 is set
  int key32;                 // the scene, list, column and quantiser fields fit 32 bits
  int sorted_buf;            // which of keys / vals [0] or [1] holds the sorted entries
  unsigned long long* n_keyed;  // boxes kept after culling (the compact and sorted entries)
  unsigned* vals[2];
  SortedBoxes S;             // P entries in sorted order
  unsigned* cell_begin;      // 3 x total cells
  unsigned* cell_end;
  unsigned long long* pack[2];     // vf / ee pairs as found, each scene's in its capacity's slice
  unsigned long long* sweep_next;  // next boxes of the sweep
  uint4* pieces;                   // queues of pieces of long windows: box, first entry, end
  unsigned long long* n_pieces;    // per queue
  unsigned long long piece_cap;    // pieces a queue holds
  int pair_bits[2];                // packed pair bits of the widest scene, per family
};

__device__ __forceinline__ unsigned long long pair_mask(int bits) { return (1ull << bits) - 1ull; }

// Sorted key i < *n_keyed from the 32- or 64-bit buffer.
__device__ __forceinline__ unsigned long long sorted_key(const BatchBroad& B, unsigned long long i) {
  return B.key32 ? (unsigned long long)B.keys32[B.sorted_buf][i] : B.keys[B.sorted_buf][i];
}

// Segment of g in offsets off (n segments), starting from the block's first
// segment.
__device__ __forceinline__ int scene_from(const unsigned long long* off, int n, int s_lo, unsigned long long g) {
  int s = s_lo;
  while (s + 1 < n && __ldg(off + s + 1) <= g) ++s;
  return s;
}

__device__ __forceinline__ int find_segment(const unsigned long long* off, int n, unsigned long long x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(off + mid) <= x) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ int cull_count(const p2c_batch_scene& d) {
  return (d.exclude_self && d.n_obj >= 1 && d.n_obj <= kMaxCullObjects) ? d.n_obj : 0;
}

// ---- 1. prep -----------------------------------------------------------------
__global__ void __launch_bounds__(kPrepThreads) prep_kernel(BatchBroad B) {
  using Scan = cub::BlockScan<unsigned long long, kPrepThreads>;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ unsigned long long carry[6];
  if (threadIdx.x < 6) carry[threadIdx.x] = 0ull;
  __syncthreads();
  unsigned long long* outs[6] = {B.off.prim, B.off.vf_cap, B.off.ee_cap, B.off.cell, B.off.vert, B.off.edge};
  for (int base = 0; base < B.n; base += kPrepThreads) {
    const int s = base + (int)threadIdx.x;
    unsigned long long v[6] = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
    if (s < B.n) {
      const p2c_batch_scene& d = B.scenes[s];
      const long long np = d.nv + d.nf + d.ne;
      v[0] = (unsigned long long)np;
      v[1] = (unsigned long long)d.vf_cap;
      v[2] = (unsigned long long)d.ee_cap;
      v[3] = (unsigned long long)cell_budget(np);
      v[4] = (unsigned long long)d.nv;
      v[5] = (unsigned long long)d.ne;
    }
    for (int k = 0; k < 6; ++k) {
      unsigned long long excl = 0ull, total = 0ull;
      Scan(tmp).ExclusiveSum(v[k], excl, total);
      if (s < B.n) outs[k][s] = carry[k] + excl;
      __syncthreads();
      if (threadIdx.x == 0) carry[k] += total;
      __syncthreads();
    }
  }
  if (threadIdx.x < 6) outs[threadIdx.x][B.n] = carry[threadIdx.x];
}

// ---- 2. vertex envelopes and axis statistics ----------------------------------
// One thread per vertex of the batch (scene s holds vertices [vert[s],
// vert[s + 1])): its swept box joins its object's envelope (order keys, one
// atomic per object and warp) and the scene's sums of extents, centres and
// squared centres that choose the sweep axis.  Faces and edges are boxes of
// these vertices, so the vertex pass also finds every non-finite coordinate;
// such a vertex takes no further part.
__global__ void __launch_bounds__(kThreads) envelope_kernel(BatchBroad B, unsigned long long V) {
  __shared__ double red[9][kThreads / 32];
  __shared__ int scene_lo, scene_hi, block_scene;
  const unsigned long long g = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  bool live = g < V;
  int s = -1, o = -1;
  double b[6] = {0, 0, 0, 0, 0, 0};
  if (threadIdx.x == 0) {
    const unsigned long long first = (unsigned long long)blockIdx.x * blockDim.x;
    block_scene = scene_lo = find_segment(B.off.vert, B.n, first);
    scene_hi = find_segment(B.off.vert, B.n, min(first + blockDim.x, V) - 1ull);
  }
  __syncthreads();
  if (live) {
    s = scene_from(B.off.vert, B.n, block_scene, g);
    const p2c_batch_scene& d = B.scenes[s];
    const long long i = (long long)(g - B.off.vert[s]);
    live = swept_box<1>(d.v_t0, d.v_t1, nullptr, i, d.thickness, b);
    if (!live) atomicOr(&B.sc[s].error_word, 1ull);
    if (live && cull_count(d) > 0) o = d.v_obj[i];
  }
  // object envelopes: per (scene, object) one atomic per warp
  {
    const bool mine0 = o >= 0 && s >= 0 && o < kMaxCullObjects;
    unsigned remaining = __ballot_sync(kFull, mine0);
    while (remaining) {
      const int leader = __ffs((int)remaining) - 1;
      const int ls = __shfl_sync(kFull, s, leader), lo_obj = __shfl_sync(kFull, o, leader);
      const bool mine = mine0 && s == ls && o == lo_obj;
      remaining &= ~__ballot_sync(kFull, mine);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        unsigned long long kmin = mine ? order_key(b[a]) : ~0ull;
        unsigned long long kmax = mine ? order_key(b[3 + a]) : 0ull;
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) {
          kmin = min(kmin, __shfl_xor_sync(kFull, kmin, sh));
          kmax = max(kmax, __shfl_xor_sync(kFull, kmax, sh));
        }
        if (lane == leader) {
          atomicMax(&B.sc[ls].obj_nlo[lo_obj][a], ~kmin);
          atomicMax(&B.sc[ls].obj_hi[lo_obj][a], kmax);
        }
      }
    }
  }
  // axis statistics: sums of extents, centres and squared centres
  double vals[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (live) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double c = 0.5 * (b[3 + a] + b[a]);
      vals[a] = b[3 + a] - b[a];
      vals[3 + a] = c;
      vals[6 + a] = c * c;
    }
  }
  if (scene_lo == scene_hi) {  // one scene in the block: block sums, 10 atomics
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      double v = vals[k];
#pragma unroll
      for (int sh = 16; sh > 0; sh >>= 1) v += __shfl_down_sync(kFull, v, sh);
      if (lane == 0) red[k][threadIdx.x >> 5] = v;
    }
    const unsigned cnt = __popc(__ballot_sync(kFull, live));
    __syncthreads();
    BroadScratch& sc = B.sc[scene_lo];
    if (threadIdx.x < 9) {
      double t = 0.0;
      for (int w = 0; w < kThreads / 32; ++w) t += red[threadIdx.x][w];
      double* dst = threadIdx.x < 3 ? &sc.extent_sum[threadIdx.x]
                    : threadIdx.x < 6 ? &sc.center_sum[threadIdx.x - 3]
                                      : &sc.center_sq_sum[threadIdx.x - 6];
      atomicAdd(dst, t);
    }
    if (lane == 0 && cnt) atomicAdd(&sc.count, (unsigned long long)cnt);
  } else {  // scene boundary inside the block: per warp and scene
    unsigned todo = __ballot_sync(kFull, live);
    while (todo) {
      const int leader = __ffs((int)todo) - 1;
      const int ls = __shfl_sync(kFull, s, leader);
      const bool mine = live && s == ls;
      todo &= ~__ballot_sync(kFull, mine);
      BroadScratch& sc = B.sc[ls];
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        double v = mine ? vals[k] : 0.0;
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) v += __shfl_xor_sync(kFull, v, sh);
        if (lane == leader) {
          double* dst = k < 3 ? &sc.extent_sum[k] : k < 6 ? &sc.center_sum[k - 3] : &sc.center_sq_sum[k - 6];
          atomicAdd(dst, v);
        }
      }
      const unsigned cnt = __popc(__ballot_sync(kFull, mine));
      if (lane == leader) atomicAdd(&sc.count, (unsigned long long)cnt);
    }
  }
}

// ---- 3. swept boxes, culling, compaction and per-list extents ------------------
__device__ __forceinline__ void max_if_larger(unsigned long long* p, unsigned long long v) {
  if (v > *reinterpret_cast<volatile unsigned long long*>(p)) atomicMax(p, v);
}

// One thread per primitive: its swept box; kept unless it is a vertex in no
// face, has a non-finite coordinate or (self pairs excluded) lies outside
// every other object's envelope.  Kept boxes are appended (one atomic per warp) to a compact list
// of (box, primitive) entries that everything after works on, and their
// extents per (scene, list) size the column grids.
// A block takes kCullSpan consecutive primitives: its start (the search for its
// scene, then the scene's table entry) is a chain of dependent loads that 256
// primitives alone do not cover (64 uneven scenes, 7.2 M primitives: 130 us with
// 256 a block, 118 with 1024).
constexpr unsigned kCullSpan = 4 * kThreads;

__global__ void __launch_bounds__(kThreads) cull_kernel(BatchBroad B, unsigned long long P) {
  __shared__ int block_scene;
  const unsigned long long block_first = (unsigned long long)blockIdx.x * kCullSpan;
  if (threadIdx.x == 0) block_scene = find_segment(B.off.prim, B.n, block_first);
  __syncthreads();
  for (unsigned long long g = block_first + threadIdx.x; g - threadIdx.x < min(P, block_first + kCullSpan);
       g += kThreads) {
    bool keep = false, other = false;
    int s = -1, l = 3;
    double b[6] = {0, 0, 0, 0, 0, 0};
    if (g < P) {
      s = scene_from(B.off.prim, B.n, block_scene, g);
      const p2c_batch_scene& d = B.scenes[s];
      const long long loc = (long long)(g - B.off.prim[s]);
      l = loc < d.nv ? 0 : (loc < d.nv + d.nf ? 1 : 2);
      const long long i = l == 0 ? loc : (l == 1 ? loc - d.nv : loc - d.nv - d.nf);
      const int o = (l == 0 ? d.v_obj : (l == 1 ? d.f_obj : d.e_obj))[i];
      keep = !(l == 0 && o < 0);
      const bool finite = l == 0   ? swept_box<1>(d.v_t0, d.v_t1, nullptr, i, d.thickness, b)
                          : l == 1 ? swept_box<3>(d.v_t0, d.v_t1, d.faces, i, d.thickness, b)
                                   : swept_box<2>(d.v_t0, d.v_t1, d.edges, i, d.thickness, b);
      keep = keep && finite;
      const int cull = cull_count(d);
      if (keep && cull > 0) {
        const BroadScratch& sc = B.sc[s];
        bool near_other = false;
        for (int q = 0; q < cull && !near_other; ++q) {
          if (q == o || sc.obj_hi[q][0] == 0ull) continue;
          bool ov = true;
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const double olo = unorder_key(~sc.obj_nlo[q][a]), ohi = unorder_key(sc.obj_hi[q][a]);
            ov = ov && b[a] <= ohi && olo <= b[3 + a];
          }
          near_other = ov;
        }
        keep = near_other;
      }
      other = keep && o != 0 && o != 1 && d.exclude_self && d.n_obj == 2;
    }
    if (__any_sync(kFull, other) && other) atomicOr(&B.sc[s].obj_other, 1ull);  // only malformed two-object scenes
    // compaction of the kept boxes
    {
      const unsigned m = __ballot_sync(kFull, keep);
      if (m != 0u) {
        const int lane = threadIdx.x & 31;
        const int leader = __ffs((int)m) - 1;
        unsigned long long base = 0;
        if (lane == leader) base = atomicAdd(B.n_keyed, (unsigned long long)__popc(m));
        base = __shfl_sync(kFull, base, leader);
        if (keep) {
          const unsigned long long c = base + (unsigned long long)__popc(m & ((1u << lane) - 1u));
          double* dst = B.cbox + 6 * c;
#pragma unroll
          for (int k = 0; k < 6; ++k) dst[k] = b[k];
          B.cprim[c] = (unsigned)g;
        }
      }
    }
    // per (scene, list) extents; most warps hold one scene and one list
    unsigned todo = __ballot_sync(kFull, keep);
    while (todo) {
      const int leader = __ffs((int)todo) - 1;
      const int ls = __shfl_sync(kFull, s, leader), ll = __shfl_sync(kFull, l, leader);
      const bool mine = keep && s == ls && l == ll;
      const unsigned mask = __ballot_sync(kFull, mine);
      todo &= ~mask;
      ListStats& S = B.sc[ls].list[ll];
      if ((threadIdx.x & 31) == leader) atomicAdd(&S.active, (unsigned long long)__popc(mask));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        unsigned long long ext = mine ? (unsigned long long)__double_as_longlong(b[3 + a] - b[a]) : 0ull;
        unsigned long long lo = mine ? order_key(b[a]) : ~0ull;
        unsigned long long hi = mine ? order_key(b[3 + a]) : 0ull;
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) {
          ext = max(ext, __shfl_xor_sync(kFull, ext, sh));
          lo = min(lo, __shfl_xor_sync(kFull, lo, sh));
          hi = max(hi, __shfl_xor_sync(kFull, hi, sh));
        }
        if ((threadIdx.x & 31) == leader) {
          max_if_larger(&S.ext_max[a], ext);
          max_if_larger(&S.nlo_min[a], ~lo);
          max_if_larger(&S.hi_max[a], hi);
        }
      }
    }
  }
}

// ---- 4. per-scene grid (one thread per scene) ---------------------------------
__global__ void grid_kernel(BatchBroad B) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= B.n) return;
  BroadScratch& sc = B.sc[s];
  const long long budget = (long long)(B.off.cell[s + 1] - B.off.cell[s]);
  int max_cols = (int)floor(sqrt((double)budget));
  if (max_cols > kMaxColumns) max_cols = kMaxColumns;
  if (max_cols < 1) max_cols = 1;
  const double n = sc.count > 0 ? (double)sc.count : 1.0;
  int axis = 0;
  double best = INFINITY;
  for (int a = 0; a < 3; ++a) {
    const double mean = sc.center_sum[a] / n;
    const double var = fmax(sc.center_sq_sum[a] / n - mean * mean, 0.0);
    const double score = (sc.extent_sum[a] / n) / (sqrt(var) + 1e-300);
    if (score < best) {
      best = score;
      axis = a;
    }
  }
  Grid g;
  g.axis = axis;
  g.a1 = axis == 0 ? 1 : 0;
  g.a2 = axis == 2 ? 1 : 2;
  const p2c_batch_scene& d = B.scenes[s];
  const bool split = d.exclude_self && d.n_obj == 2 && sc.obj_other == 0ull;
  g.split_shift = split ? kBatchQBits - 1 : -1;
  g.qmax = split ? (kBatchQMax >> 1) : kBatchQMax;
  const int ax[3] = {g.a1, g.a2, axis};
  double base[3], inv[3];
  int cols[2] = {1, 1};
  for (int k = 0; k < 3; ++k) {
    double lo = INFINITY, hi = -INFINITY, reach = 0.0;
    for (int l = 0; l < 3; ++l) {
      const ListStats& L = sc.list[l];
      const double r = L.active ? __longlong_as_double((long long)L.ext_max[ax[k]]) : 0.0;
      if (k < 2) (k == 0 ? g.reach1 : g.reach2)[l] = r;
      if (L.active == 0) continue;
      lo = fmin(lo, unorder_key(~L.nlo_min[ax[k]]));
      hi = fmax(hi, unorder_key(L.hi_max[ax[k]]));
      reach = fmax(reach, r);
    }
    const double range = (hi > lo) ? hi - lo : 0.0;
    base[k] = isfinite(lo) ? lo : 0.0;
    if (k < 2) {
      double width = fmax(reach, range / max_cols);
      if (!(width > 0.0) || !isfinite(width)) width = 1.0;
      int c = (int)fmin((double)max_cols, floor(range / width) + 1.0);
      cols[k] = c < 1 ? 1 : c;
      inv[k] = 1.0 / width;
    } else {
      inv[k] = (range > 0.0 && isfinite(range)) ? (double)g.qmax / range : 0.0;
    }
  }
  g.base1 = base[0];
  g.base2 = base[1];
  g.inv1 = inv[0];
  g.inv2 = inv[1];
  g.g1 = cols[0];
  g.g2 = cols[1];
  g.base0 = base[2];
  g.scale0 = inv[2];
  g.seg[0] = 0;
  g.seg[1] = sc.list[0].active;
  g.seg[2] = g.seg[1] + sc.list[1].active;
  g.seg[3] = g.seg[2] + sc.list[2].active;
  sc.grid = g;
}

// ---- 5. keys, sort, gather ---------------------------------------------------------
// Sort key of every kept box (compact entry c, value c): the order of the
// compact entries does not matter, they are sorted on their full keys and
// the pairs are sorted at the end.
// With pad_to > 0 the entries [kept, pad_to) get the key ~0, after every box
// (its list field, 3, names no list), for a sort sized on the host.
__global__ void __launch_bounds__(kThreads) keys_kernel(BatchBroad B, unsigned long long pad_to) {
  const unsigned long long n = *B.n_keyed;
  for (unsigned long long c = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; c < pad_to;
       c += (unsigned long long)gridDim.x * blockDim.x)
    if (c >= n) {
      if (B.key32) B.keys32[0][c] = ~0u;
      else B.keys[0][c] = ~0ull;
      B.vals[0][c] = (unsigned)c;
    }
  for (unsigned long long c = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; c < n;
       c += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long g = B.cprim[c];
    const int s = find_segment(B.off.prim, B.n, g);
    const p2c_batch_scene& d = B.scenes[s];
    const long long loc = (long long)(g - B.off.prim[s]);
    const int l = loc < d.nv ? 0 : (loc < d.nv + d.nf ? 1 : 2);
    const Grid& G = B.sc[s].grid;
    const double* b = B.cbox + 6 * c;
    const unsigned cell = (unsigned)(column(b[G.a1], G.base1, G.inv1, G.g1) * G.g2 +
                                     column(b[G.a2], G.base2, G.inv2, G.g2));
    int32_t o = 0;
    if (G.split_shift >= 0) {
      const long long j = l == 0 ? loc : (l == 1 ? loc - d.nv : loc - d.nv - d.nf);
      o = (l == 0 ? d.v_obj : (l == 1 ? d.f_obj : d.e_obj))[j];
    }
    const unsigned long long key = ((unsigned long long)s << kBatchSceneShift) |
                                   ((unsigned long long)l << kBatchListShift) |
                                   ((unsigned long long)cell << kBatchQBits) |
                                   split_field(G, o, quantise(b[G.axis], G));
    if (B.key32) B.keys32[0][c] = (unsigned)key;
    else B.keys[0][c] = key;
    B.vals[0][c] = (unsigned)c;
  }
}

__device__ __forceinline__ unsigned* cell_table(const BatchBroad& B, unsigned* base, int s, int l) {
  const unsigned long long c0 = B.off.cell[s], budget = B.off.cell[s + 1] - c0;
  return base + 3ull * c0 + (unsigned long long)l * budget;
}

__device__ __forceinline__ void gather_one(const BatchBroad& B, const unsigned* __restrict__ order,
                                           unsigned long long i, unsigned long long n) {
  const unsigned long long key = sorted_key(B, i);
  const int s = (int)(key >> kBatchSceneShift);
  const int l = (int)((key >> kBatchListShift) & 3ull);
  const p2c_batch_scene& d = B.scenes[s];
  const Grid& G = B.sc[s].grid;
  const unsigned c = order[i];
  const unsigned long long g = B.cprim[c];
  const long long loc = (long long)(g - B.off.prim[s]);
  const long long j = l == 0 ? loc : (l == 1 ? loc - d.nv : loc - d.nv - d.nf);
  const double* b = B.cbox + 6 * (unsigned long long)c;
  B.S.lo[i] = b[G.axis];
  B.S.hi[i] = b[3 + G.axis];
  B.S.alo[i] = b[G.a1];
  B.S.ahi[i] = b[3 + G.a1];
  B.S.blo[i] = b[G.a2];
  B.S.bhi[i] = b[3 + G.a2];
  B.S.q[i] = (unsigned)(key & kBatchQMax);
  B.S.fb[i] = fbox_entry(b[G.a1], b[3 + G.a1], b[G.a2], b[3 + G.a2]);
  B.S.id[i] = (int32_t)j;
  B.S.obj[i] = (l == 0 ? d.v_obj : (l == 1 ? d.f_obj : d.e_obj))[j];
  const unsigned long long head = key >> kBatchQBits;  // scene, list and column
  const unsigned cell = (unsigned)(head & ((1ull << kCellBits) - 1ull));
  if (i == 0 || (sorted_key(B, i - 1) >> kBatchQBits) != head) cell_table(B, B.cell_begin, s, l)[cell] = (unsigned)i;
  if (i + 1 == n || (sorted_key(B, i + 1) >> kBatchQBits) != head)
    cell_table(B, B.cell_end, s, l)[cell] = (unsigned)(i + 1);
}

__global__ void __launch_bounds__(kThreads) gather_kernel(BatchBroad B) {
  const unsigned long long n = *B.n_keyed;
  const unsigned* __restrict__ order = B.vals[B.sorted_buf];
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x)
    gather_one(B, order, i, n);
}

// ---- 6. sweeps -------------------------------------------------------------------
// Pairs a warp has found, packed with their scenes, written 64 at a time with
// one atomic for each scene among 32 of them.
struct ScenePairBuffer {
  unsigned long long* slots;  // shared, 96
  unsigned n;                 // warp-uniform

  __device__ __forceinline__ void flush(unsigned count, const BatchBroad& B, int family) {
    const int lane = threadIdx.x & 31, bits = B.pair_bits[family];
    const unsigned long long* cap_off = family == 0 ? B.off.vf_cap : B.off.ee_cap;
    __syncwarp();
    for (unsigned k0 = 0; k0 < count; k0 += 32u) {
      const bool live = k0 + (unsigned)lane < count;
      const unsigned long long key = live ? slots[k0 + (unsigned)lane] : 0ull;
      const int s = live ? (int)(key >> bits) : -1;
      const unsigned same = __match_any_sync(kFull, s);
      const int leader = __ffs((int)same) - 1;
      unsigned long long base = 0;
      if (live && lane == leader)
        base = atomicAdd(family == 0 ? &B.sc[s].vf_count : &B.sc[s].ee_count, (unsigned long long)__popc(same));
      base = __shfl_sync(kFull, base, leader);
      if (live) {
        const unsigned long long slot = base + (unsigned long long)__popc(same & ((1u << lane) - 1u));
        if (slot < cap_off[s + 1] - cap_off[s]) B.pack[family][cap_off[s] + slot] = key;
      }
    }
    __syncwarp();
    if (count + (unsigned)lane < n) {  // at most 31 stay
      const unsigned long long rest = slots[count + (unsigned)lane];
      slots[lane] = rest;
    }
    n -= count;
    __syncwarp();
  }
  __device__ __forceinline__ void append(bool found, unsigned long long key, const BatchBroad& B, int family) {
    const unsigned mask = __ballot_sync(kFull, found);
    if (mask == 0u) return;
    if (found) slots[n + (unsigned)__popc(mask & ((1u << (threadIdx.x & 31)) - 1u))] = key;
    n += (unsigned)__popc(mask);
    if (n >= 64u) flush(64u, B, family);
  }
};

// Lanes that share one scanning box: they look its columns' windows up side by
// side and walk all of them as one list, as the single-scene sweep does.
constexpr int kSweepLanes = 8;
// A column of at most this many entries is walked without a search (4 / 8 / 16 /
// 64: 64 uneven scenes 609 / 609 / 610 / 629 us a step, 51,200 proxies 511 / 511 /
// 517 / 550).
constexpr unsigned kWholeRun = 8;

// A window longer than kLongWindow goes to a queue in pieces of kPiece entries,
// which a second launch spreads over the whole GPU.  A primitive that is large
// against the others of its scene (a ground quad under a mesh) has all of them
// in one window: walked by its eight lanes alone it sets the length of the
// launch.  Candidates of a sheet of 96,800 triangles over one quad: 36,400 us
// by the eight lanes, 530 with the queues; 64 uneven scenes, which hardly use
// them, pay 3 us for their empty launch.  Windows from 128 / 256 / 512 entries
// on differ by 2 %, pieces of 32 / 64 / 128 entries by 3 %.
// A full queue leaves a window to its lanes.  Windows are queued by length, one
// queue for each factor of four, so that the many middling ones of a dense
// scene never take the room of the longest (four self-colliding sheets over
// quads: 4,030 us when they do, 560 when not).
#ifndef P2C_BATCH_LONG_WINDOW
#define P2C_BATCH_LONG_WINDOW 256
#endif
#ifndef P2C_BATCH_PIECE
#define P2C_BATCH_PIECE 64
#endif
constexpr unsigned kLongWindow = P2C_BATCH_LONG_WINDOW;
constexpr unsigned kPiece = P2C_BATCH_PIECE;
constexpr int kPieceQueues = 4;
// A queue holds one piece per eight primitives of the batch, within [4096, 2^20]
// (a small batch keeps a small workspace).
__host__ __device__ inline unsigned long long piece_cap_for(unsigned long long prims) {
  const unsigned long long c = prims / 8;
  return c < 4096ull ? 4096ull : (c > (1ull << 20) ? (1ull << 20) : c);
}

// A scanning box: its list, scene and primitive, and what its walk tests
// first.  The exact bounds are read again for an entry that passes.
struct ScanBox {
  unsigned i;
  int l, s, id, obj;
  double lo, hi;
  FBox pf;
};

// Entry j is a pair that the box owns.  Vertex-face pairs: a vertex owns the
// pairs whose face minimum is >= its minimum, a face the others.  Edge-edge
// pairs: an edge owns the pairs whose partner minimum is larger (ties: larger
// index).
__device__ __forceinline__ bool test_entry(const BatchBroad& B, const ScanBox& x, unsigned j, unsigned long long& key) {
  const float4 qf = B.S.fb[j];
  const double qlo = B.S.lo[j];
  if (!(qlo >= x.lo && qlo <= x.hi && fmay_overlap(x.pf, qf))) return false;
  const int qid = B.S.id[j];
  const bool own = x.l == 0 || qlo > x.lo || (x.l == 2 && qid > x.id);
  if (!own || !overlap3(box_at(B.S, (long long)x.i), qlo, B.S, j)) return false;
  const p2c_batch_scene& d = B.scenes[x.s];
  if (B.S.obj[j] == x.obj) {  // the reference's object rules
    if (d.exclude_self) return false;
    if (x.l == 2) {
      const int32_t* ea = d.edges + 2 * (long long)x.id;
      const int32_t* eb = d.edges + 2 * (long long)qid;
      const int a0 = __ldg(ea), a1 = __ldg(ea + 1), b0 = __ldg(eb), b1 = __ldg(eb + 1);
      if (a0 == b0 || a0 == b1 || a1 == b0 || a1 == b1) return false;
    } else {
      const int vtx = x.l == 0 ? x.id : qid;
      const int32_t* fv = d.faces + 3 * (long long)(x.l == 0 ? qid : x.id);
      if (__ldg(fv) == vtx || __ldg(fv + 1) == vtx || __ldg(fv + 2) == vtx) return false;
    }
  }
  const int shift = max(1, bit_length_dev(x.l == 2 ? d.ne : d.nf));
  const unsigned a = x.l == 2 ? (unsigned)min(x.id, qid) : (unsigned)(x.l == 0 ? x.id : qid);
  const unsigned b = x.l == 2 ? (unsigned)max(x.id, qid) : (unsigned)(x.l == 0 ? qid : x.id);
  key = ((unsigned long long)x.s << B.pair_bits[x.l == 2 ? 1 : 0]) | pair_key(a, b, shift);
  return true;
}

// Queues the window [offset, offset + len) of box i, if it is long and fits.
// Of the last queue, whose windows have no largest length, a window takes at
// most a kQueueShare-th of what is free, in longer pieces if need be: 30,000
// triangles among 20 larger ones have 140 windows of 30,000 to 90,000 entries,
// more than the queue holds in short pieces (28.4 ms then, 5.6 so).
constexpr unsigned kQueueShare = 32;

__device__ __forceinline__ bool queue_window(uint4* pieces, unsigned long long* n_pieces, unsigned long long cap,
                                             unsigned i, unsigned offset, unsigned len) {
  if (len <= kLongWindow) return false;
  const int q = (len > 4u * kLongWindow) + (len > 16u * kLongWindow) + (len > 64u * kLongWindow);
  pieces += (unsigned long long)q * cap;
  n_pieces += q;
  unsigned long long at = *reinterpret_cast<volatile unsigned long long*>(n_pieces);
  unsigned piece = kPiece, n = (len + kPiece - 1u) / kPiece;
  if (q < kPieceQueues - 1) {
    if (at >= cap) return false;
    at = atomicAdd(n_pieces, (unsigned long long)n);
    if (at + n > cap) {
      for (unsigned long long k = at; k < cap; ++k) pieces[k] = make_uint4(0u, 0u, 0u, 0u);  // empty
      return false;
    }
  } else {
    for (unsigned long long seen = at;; at = seen) {  // ends: another window's success changes the count, never past cap
      const unsigned most = (unsigned)(cap - at) / kQueueShare;
      if (most == 0u) return false;
      piece = max(kPiece, (len + most - 1u) / most);
      n = (len + piece - 1u) / piece;
      seen = atomicCAS(n_pieces, at, at + n);
      if (seen == at) break;
    }
  }
  for (unsigned k = 0; k < n; ++k)
    pieces[at + k] = make_uint4(i, offset + k * piece, offset + min(len, (k + 1u) * piece), 0u);
  return true;
}

// Both families in one launch.  Bound by dependent loads.  Two lanes per box,
// an atomic for every step that found a pair and four launches: 379 us for a
// served group of eight scenes, 83 for 64 uneven scenes; now 178 and 63.
__global__ void __launch_bounds__(kThreads, 4) sweep_kernel(BatchBroad B, int vf_on, int ee_on) {
  __shared__ unsigned long long slots[2][kThreads / 32][96];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int member = lane & (kSweepLanes - 1), sub = lane / kSweepLanes;
  constexpr unsigned kBoxes = 32 / kSweepLanes;
  ScenePairBuffer vfb{slots[0][warp], 0u}, eeb{slots[1][warp], 0u};
  const unsigned n = (unsigned)*B.n_keyed, steps = (n + kBoxes - 1u) / kBoxes;
  const unsigned take = max(1u, min(32u, steps / (gridDim.x * (kThreads / 32) * 8u)));
  for (;;) {
    unsigned first = 0;
    if (lane == 0) first = (unsigned)atomicAdd(B.sweep_next, (unsigned long long)take);
    first = __shfl_sync(kFull, first, 0);
    if (first >= steps) break;
    for (unsigned t = first; t < min(first + take, steps); ++t) {
      ScanBox x{t * kBoxes + (unsigned)sub, 0, 0, 0, 0, 0.0, 0.0, FBox{0.f, 0.f, 0.f, 0.f}};
      bool live = x.i < n;
      if (live) {
        const unsigned long long key = sorted_key(B, x.i);
        x.l = (int)((key >> kBatchListShift) & 3ull);
        x.s = (int)(key >> kBatchSceneShift);
        live = x.l == 2 ? ee_on != 0 : (x.l <= 1 && vf_on != 0);
      }
      const int partner = x.l == 2 ? 2 : 1 - x.l;
      int c1a = 0, c2a = 0, n2 = 1, columns = 0;
      unsigned q_lo = 0, q_hi = 0;
      if (live) {
        const Grid& g = B.sc[x.s].grid;
        const Box6 pb = box_at(B.S, (long long)x.i);
        Walker w;
        walker_init(w, g, pb.lo, pb.hi, pb.alo, pb.ahi, pb.blo, pb.bhi, g.reach1[partner], g.reach2[partner]);
        x.id = B.S.id[x.i];
        x.obj = B.S.obj[x.i];
        x.lo = pb.lo;
        x.hi = pb.hi;
        x.pf = fbox_of(pb);
        c1a = w.c1;
        c2a = w.c2_begin;
        n2 = w.c2_end - w.c2_begin + 1;
        columns = (w.c1_end - w.c1 + 1) * n2;
        q_lo = w.q_lo + split_prefix(g, x.obj);
        q_hi = w.q_hi + split_prefix(g, x.obj);
      }
      const unsigned* begins = cell_table(B, B.cell_begin, x.s, partner);
      const unsigned* ends = cell_table(B, B.cell_end, x.s, partner);
      for (int c = member; __any_sync(kFull, c - member < columns); c += kSweepLanes) {
        unsigned offset = 0, len = 0;
        if (c < columns) {
          const int cell = (c1a + c / n2) * B.sc[x.s].grid.g2 + c2a + c % n2;
          unsigned b = begins[cell], e = ends[cell];
          if (e - b > kWholeRun) {
            const unsigned end = e;
            while (b < e) {  // first entry with q >= q_lo
              const unsigned m = (b + e) >> 1;
              if (B.S.q[m] < q_lo) b = m + 1;
              else e = m;
            }
            offset = b;
            e = end;
            while (b < e) {  // first one with q > q_hi
              const unsigned m = (b + e) >> 1;
              if (B.S.q[m] <= q_hi) b = m + 1;
              else e = m;
            }
            len = run_length(offset, b);
            if (queue_window(B.pieces, B.n_pieces, B.piece_cap, x.i, offset, len)) len = 0u;
          } else {
            offset = b;
            len = run_length(b, e);
          }
        }
        unsigned before = len;  // inclusive, then exclusive sum of the windows over the box's lanes
#pragma unroll
        for (int d = 1; d < kSweepLanes; d <<= 1) {
          const unsigned up = __shfl_up_sync(kFull, before, d, kSweepLanes);
          if (member >= d) before += up;
        }
        const unsigned entries = __shfl_sync(kFull, before, kSweepLanes - 1, kSweepLanes);
        before -= len;
        offset -= before;
        for (unsigned k = (unsigned)member; __any_sync(kFull, k - (unsigned)member < entries); k += kSweepLanes) {
          int run = 0;  // the last window that starts at or before entry k
#pragma unroll
          for (int d = kSweepLanes / 2; d > 0; d >>= 1) {
            const unsigned at = __shfl_sync(kFull, before, run + d, kSweepLanes);
            if (at <= k) run += d;
          }
          const unsigned j = __shfl_sync(kFull, offset, run, kSweepLanes) + k;
          unsigned long long key = 0;
          const bool found = k < entries && test_entry(B, x, j, key);
          vfb.append(found && x.l != 2, key, B, 0);
          eeb.append(found && x.l == 2, key, B, 1);
        }
      }
    }
  }
  if (vfb.n != 0u) vfb.flush(vfb.n, B, 0);
  if (eeb.n != 0u) eeb.flush(eeb.n, B, 1);
}

// The queued pieces, each by the lanes of one group.
__global__ void __launch_bounds__(kThreads, 4) piece_kernel(BatchBroad B) {
  __shared__ unsigned long long slots[2][kThreads / 32][96];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned member = (unsigned)lane & (kSweepLanes - 1), sub = (unsigned)lane / kSweepLanes;
  constexpr unsigned kBoxes = 32 / kSweepLanes;
  ScenePairBuffer vfb{slots[0][warp], 0u}, eeb{slots[1][warp], 0u};
  for (int q = kPieceQueues - 1; q >= 0; --q) {
    const unsigned n = (unsigned)min(B.n_pieces[q], B.piece_cap);
    const uint4* pieces = B.pieces + (unsigned long long)q * B.piece_cap;
    for (unsigned first = (blockIdx.x * (kThreads / 32) + (unsigned)warp) * kBoxes; first < n;
         first += gridDim.x * (kThreads / 32) * kBoxes) {
      uint4 piece = make_uint4(0u, 0u, 0u, 0u);
      if (first + sub < n) piece = pieces[first + sub];
      ScanBox x{piece.x, 0, 0, 0, 0, 0.0, 0.0, FBox{0.f, 0.f, 0.f, 0.f}};
      if (piece.z > piece.y) {
        const unsigned long long key = sorted_key(B, x.i);
        const Box6 pb = box_at(B.S, (long long)x.i);
        x.l = (int)((key >> kBatchListShift) & 3ull);
        x.s = (int)(key >> kBatchSceneShift);
        x.id = B.S.id[x.i];
        x.obj = B.S.obj[x.i];
        x.lo = pb.lo;
        x.hi = pb.hi;
        x.pf = fbox_of(pb);
      }
      for (unsigned j = piece.y + member; __any_sync(kFull, j - member < piece.z); j += kSweepLanes) {
        unsigned long long key = 0;
        const bool found = j < piece.z && test_entry(B, x, j, key);
        vfb.append(found && x.l != 2, key, B, 0);
        eeb.append(found && x.l == 2, key, B, 1);
      }
    }
  }
  if (vfb.n != 0u) vfb.flush(vfb.n, B, 0);
  if (eeb.n != 0u) eeb.flush(eeb.n, B, 1);
}

// ---- 7. pairs into the scenes' buffers, in order ------------------------------
// All scenes' pairs of one family as rows of all their vertices or edges
// (pair_rows.cuh).
struct BatchRows {
  const p2c_batch_scene* scenes;
  const BroadScratch* sc;
  unsigned long long* pack;
  const unsigned long long* cap_off;
  const unsigned long long* row_base;  // off.vert or off.edge
  int n, bits, family;
  long long cap;
  __device__ __forceinline__ int shift(int s) const {
    return max(1, bit_length_dev(family == 0 ? scenes[s].nf : scenes[s].ne));
  }
  __device__ __forceinline__ bool live(long long i) const {
    const int s = find_segment(cap_off, n, (unsigned long long)i);
    return (unsigned long long)i - cap_off[s] < (family == 0 ? sc[s].vf_count : sc[s].ee_count);
  }
  __device__ __forceinline__ bool load(long long i, unsigned long long& key) const {
    if (!live(i)) return false;
    key = pack[i];
    return true;
  }
  __device__ __forceinline__ unsigned long long row(unsigned long long key) const {
    const int s = (int)(key >> bits);
    return row_base[s] + ((key & pair_mask(bits)) >> shift(s));
  }
  __device__ __forceinline__ unsigned long long b_mask(unsigned long long key) const {
    return (1ull << shift((int)(key >> bits))) - 1ull;
  }
  __device__ __forceinline__ unsigned long long* out(int s) const {
    return reinterpret_cast<unsigned long long*>(family == 0 ? scenes[s].vf_pairs : scenes[s].ee_pairs);
  }
  __device__ __forceinline__ void pad(long long i) const {
    const int s = find_segment(cap_off, n, (unsigned long long)i);
    out(s)[(unsigned long long)i - cap_off[s]] = ~0ull;
  }
  __device__ __forceinline__ void store(unsigned place, unsigned long long key, const unsigned* rows) const {
    const int s = (int)(key >> bits), sh = shift(s);
    const unsigned base = family == 0 ? 0u : rows[-1];
    const unsigned first = row_base[s] == 0ull ? 0u : rows[(long long)row_base[s] - 1] - base;  // the scene's first place
    out(s)[place - first] = ((key & pair_mask(bits)) >> sh << 32) | (key & ((1ull << sh) - 1ull));
  }
  __device__ __forceinline__ unsigned long long* input() const { return pack; }
};

__global__ void export_counts_kernel(BatchBroad B) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= B.n) return;
  const BroadScratch& sc = B.sc[s];
  unsigned long long* c = reinterpret_cast<unsigned long long*>(B.scenes[s].counts);
  c[0] = sc.vf_count;
  c[1] = sc.ee_count;
  c[2] = sc.error_word;
  c[3] = (unsigned long long)sc.grid.axis | ((unsigned long long)sc.grid.g1 << 8) |
         ((unsigned long long)sc.grid.g2 << 24) | (sc.grid.seg[3] << 40);
}

// ---- workspace ---------------------------------------------------------------------
struct Totals {
  unsigned long long P = 0, V = 0, E = 0, vf = 0, ee = 0, cells = 0;
  int pair_bits[2] = {2, 2};  // widest packed pair of any scene: vf, ee
  long long most_in_row[2] = {0, 0};  // most pairs of one vertex, of one edge
};

Totals totals_of(const p2c_batch_scene* h, int n) {
  Totals t;
  for (int s = 0; s < n; ++s) {
    const long long np = h[s].nv + h[s].nf + h[s].ne;
    t.P += (unsigned long long)np;
    t.V += (unsigned long long)h[s].nv;
    t.E += (unsigned long long)h[s].ne;
    t.vf += (unsigned long long)h[s].vf_cap;
    t.ee += (unsigned long long)h[s].ee_cap;
    t.cells += (unsigned long long)cell_budget(np);
    t.pair_bits[0] = std::max(t.pair_bits[0], bit_length(h[s].nv) + std::max(1, bit_length(h[s].nf)));
    t.most_in_row[0] = std::max<long long>(t.most_in_row[0], h[s].nf);
    t.most_in_row[1] = std::max<long long>(t.most_in_row[1], h[s].ne);
    t.pair_bits[1] = std::max(t.pair_bits[1], bit_length(h[s].ne) + std::max(1, bit_length(h[s].ne)));
  }
  return t;
}

size_t sort_temp_bytes(const Totals& t) {
  size_t a32 = 0, a64 = 0;
  const int np = (int)std::max<unsigned long long>(t.P, 1ull);
  cub::DeviceRadixSort::SortPairs(nullptr, a32, (const unsigned*)nullptr, (unsigned*)nullptr, (const unsigned*)nullptr,
                                  (unsigned*)nullptr, np);
  cub::DeviceRadixSort::SortPairs(nullptr, a64, (const unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                  (const unsigned*)nullptr, (unsigned*)nullptr, np);
  return std::max(count_sort_scratch_bytes((long long)np), std::max(a32, a64));
}

struct Carve {
  BatchBroad B;
  RowScratch rows = {};
  size_t zero_bytes = 0;  // from the scratch on
  void* tmp = nullptr;
  size_t tmp_bytes = 0;
  size_t total = 0;
};

Carve carve(void* base, const p2c_batch_scene* scenes_dev, int n, const Totals& t) {
  Carve C;
  size_t off = 0;
  char* b = static_cast<char*>(base);
  auto take = [&](size_t bytes) -> void* {
    void* p = b == nullptr ? nullptr : b + off;
    off += (std::max<size_t>(bytes, 1) + 255) & ~size_t(255);
    return p;
  };
  const size_t P = (size_t)std::max<unsigned long long>(t.P, 1ull);
  BatchBroad& B = C.B;
  B.scenes = scenes_dev;
  B.n = n;
  B.off.prim = static_cast<unsigned long long*>(take(8 * (size_t)(n + 1)));
  B.off.vf_cap = static_cast<unsigned long long*>(take(8 * (size_t)(n + 1)));
  B.off.ee_cap = static_cast<unsigned long long*>(take(8 * (size_t)(n + 1)));
  B.off.cell = static_cast<unsigned long long*>(take(8 * (size_t)(n + 1)));
  const size_t zero_at = off;  // scratch, counters and column tables start at zero
  B.sc = static_cast<BroadScratch*>(take(sizeof(BroadScratch) * (size_t)n));
  B.n_keyed = static_cast<unsigned long long*>(take(8 * (2 + kPieceQueues)));
  B.sweep_next = B.n_keyed + 1;
  B.n_pieces = B.n_keyed + 2;
  B.cell_begin = static_cast<unsigned*>(take(4 * 3 * (size_t)t.cells));
  B.cell_end = static_cast<unsigned*>(take(4 * 3 * (size_t)t.cells));
  C.zero_bytes = off - zero_at;
  B.off.vert = static_cast<unsigned long long*>(take(8 * (size_t)(n + 1)));
  B.off.edge = static_cast<unsigned long long*>(take(8 * (size_t)(n + 1)));
  B.cbox = static_cast<double*>(take(48 * P));
  B.cprim = static_cast<unsigned*>(take(4 * P));
  B.keys[0] = static_cast<unsigned long long*>(take(8 * P));
  B.keys[1] = static_cast<unsigned long long*>(take(8 * P));
  B.keys32[0] = reinterpret_cast<unsigned*>(B.keys[0]);
  B.keys32[1] = reinterpret_cast<unsigned*>(B.keys[1]);
  B.key32 = 0;
  B.sorted_buf = 0;
  B.piece_cap = piece_cap_for(t.P);
  B.pieces = static_cast<uint4*>(take(sizeof(uint4) * (size_t)(B.piece_cap * kPieceQueues)));
  B.vals[0] = static_cast<unsigned*>(take(4 * P));
  B.vals[1] = static_cast<unsigned*>(take(4 * P));
  B.S.lo = static_cast<double*>(take(8 * P));
  B.S.hi = static_cast<double*>(take(8 * P));
  B.S.alo = static_cast<double*>(take(8 * P));
  B.S.ahi = static_cast<double*>(take(8 * P));
  B.S.blo = static_cast<double*>(take(8 * P));
  B.S.bhi = static_cast<double*>(take(8 * P));
  B.S.q = static_cast<unsigned*>(take(4 * P));
  B.S.fb = static_cast<float4*>(take(16 * P));
  B.S.id = static_cast<int32_t*>(take(4 * P));
  B.S.obj = static_cast<int32_t*>(take(4 * P));
  B.pack[0] = static_cast<unsigned long long*>(take(8 * (size_t)std::max<unsigned long long>(t.vf, 1ull)));
  B.pack[1] = static_cast<unsigned long long*>(take(8 * (size_t)std::max<unsigned long long>(t.ee, 1ull)));
  const long long caps[2] = {(long long)t.vf, (long long)t.ee};
  C.rows = carve_rows((long long)(t.V + t.E), caps, take);
  C.tmp_bytes = sort_temp_bytes(t);
  C.tmp = take(C.tmp_bytes);
  C.total = off;
  return C;
}

int validate_table(const p2c_batch_scene* h, int n) {
  for (int s = 0; s < n; ++s) {
    const p2c_batch_scene& d = h[s];
    p2c_scene sc{d.v_t0, d.v_t1, d.faces, d.edges, d.v_obj, d.f_obj, d.e_obj, d.nv, d.nf, d.ne, d.thickness,
                 d.exclude_self, d.n_obj};
    const int rc = validate_scene(&sc);
    if (rc != P2C_OK) return fail(rc, "scene %d: %s", s, p2c_last_error());
    if (d.nv >= kMaxScenePrims || d.nf >= kMaxScenePrims || d.ne >= kMaxScenePrims)
      return fail(P2C_ERR_INVALID, "scene %d: batched candidates need nv, nf, ne < 2^22", s);
    if (d.counts == nullptr) return fail(P2C_ERR_INVALID, "scene %d: counts pointer is null", s);
    if (d.vf_cap < 0 || d.ee_cap < 0) return fail(P2C_ERR_INVALID, "scene %d: pair capacities must be non-negative", s);
    if ((d.vf_cap > 0 && d.vf_pairs == nullptr) || (d.ee_cap > 0 && d.ee_pairs == nullptr))
      return fail(P2C_ERR_INVALID, "scene %d: pair output pointer is null", s);
  }
  return P2C_OK;
}

}  // namespace

// Blocks of a loop over device-counted work: exactly what the device holds at
// once (SMs x resident blocks of this kernel).  All blocks then run side by
// side and each pass of the loop covers one contiguous stretch of the sorted
// entries, so the partners they read stay in the L2 (a larger grid runs its
// blocks in waves that each walk their own far-apart stretches).
template <class K>
unsigned resident_grid(K kernel, const DeviceInfo& info) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  return (unsigned)std::max(1, info.sm_count) * (unsigned)per_sm;
}

int launch_batch_candidates(const p2c_batch_scene* h, const p2c_batch_scene* dev, int n, void* ws, size_t ws_bytes,
                            cudaStream_t s) {
  const Totals t = totals_of(h, n);
  if (t.P >= (1ull << 31) || t.vf >= (1ull << 31) || t.ee >= (1ull << 31))
    return fail(P2C_ERR_INVALID, "batch too large for one candidate launch (primitives and capacities < 2^31)");
  const Carve need = carve(nullptr, dev, n, t);
  if (ws == nullptr || ws_bytes < need.total)
    return fail(P2C_ERR_INVALID, "batch candidate workspace too small: %zu < %zu bytes", ws_bytes, need.total);
  Carve C = carve(ws, dev, n, t);
  BatchBroad& B = C.B;
  const int scene_bits = std::max(1, bit_length(n - 1));
  const int key_bits = kBatchSceneShift + scene_bits;
  B.key32 = key_bits <= 32 ? 1 : 0;  // up to 256 scenes: 32-bit keys halve the key traffic of the sort
  B.pair_bits[0] = t.pair_bits[0];
  B.pair_bits[1] = t.pair_bits[1];
  P2C_CUDA(cudaMemsetAsync(B.sc, 0, C.zero_bytes, s));
  prep_kernel<<<1, kPrepThreads, 0, s>>>(B);
  P2C_CUDA(cudaGetLastError());
  const unsigned long long P = t.P;
  if (t.V > 0) envelope_kernel<<<grid_for((long long)t.V, kThreads), kThreads, 0, s>>>(B, t.V);
  if (P > 0) cull_kernel<<<grid_for((long long)P, kCullSpan), kThreads, 0, s>>>(B, P);
  grid_kernel<<<grid_for(n, 128), 128, 0, s>>>(B);
  P2C_CUDA(cudaGetLastError());
  DeviceInfo info;
  int rc = current_device_info(&info);
  if (rc != P2C_OK) return rc;
  bool any_cull = false;
  for (int k = 0; k < n && !any_cull; ++k)
    any_cull = h[k].exclude_self && h[k].n_obj >= 1 && h[k].n_obj <= kMaxCullObjects;
  if (P > 0) {
    // No scene culls: nearly every box is kept, and the library's onesweep
    // sort over all P entries (the others padded to sort last) beats ranking
    // them with the count sort; otherwise only the kept boxes are ranked.
    keys_kernel<<<std::min(grid_for((long long)P, kThreads), resident_grid(keys_kernel, info)), kThreads, 0, s>>>(B, any_cull ? 0ull : P);
    P2C_CUDA(cudaGetLastError());
    bool second = false;
    if (!any_cull) {
      size_t tb = C.tmp_bytes;
      if (B.key32) {
        cub::DoubleBuffer<unsigned> k(B.keys32[0], B.keys32[1]);
        cub::DoubleBuffer<unsigned> v(B.vals[0], B.vals[1]);
        P2C_CUDA(cub::DeviceRadixSort::SortPairs(C.tmp, tb, k, v, (int)P, 0, key_bits, s));
        second = k.selector == 1;
      } else {
        cub::DoubleBuffer<unsigned long long> k(B.keys[0], B.keys[1]);
        cub::DoubleBuffer<unsigned> v(B.vals[0], B.vals[1]);
        P2C_CUDA(cub::DeviceRadixSort::SortPairs(C.tmp, tb, k, v, (int)P, 0, key_bits, s));
        second = k.selector == 1;
      }
    } else {
      rc = B.key32 ? count_sort_pairs(B.keys32[0], B.vals[0], B.keys32[1], B.vals[1], B.n_keyed, (long long)P,
                                      key_bits, C.tmp, C.tmp_bytes, s, &second)
                   : count_sort_pairs(B.keys[0], B.vals[0], B.keys[1], B.vals[1], B.n_keyed, (long long)P, key_bits,
                                      C.tmp, C.tmp_bytes, s, &second);
      if (rc != P2C_OK) return rc;
    }
    B.sorted_buf = second ? 1 : 0;
    gather_kernel<<<std::min(grid_for((long long)P, kThreads), resident_grid(gather_kernel, info)), kThreads, 0,
                    s>>>(B);
    P2C_CUDA(cudaGetLastError());
  }
  if (P > 0 && (t.vf > 0 || t.ee > 0)) {
    sweep_kernel<<<std::min(grid_for((long long)P * kSweepLanes, kThreads), resident_grid(sweep_kernel, info)), kThreads,
                   0, s>>>(B, t.vf > 0 ? 1 : 0, t.ee > 0 ? 1 : 0);
    P2C_CUDA(cudaGetLastError());
    if (P > kLongWindow) {
      piece_kernel<<<resident_grid(piece_kernel, info), kThreads, 0, s>>>(B);
      P2C_CUDA(cudaGetLastError());
    }
  }
  const BatchRows vf{B.scenes, B.sc, B.pack[0], B.off.vf_cap, B.off.vert, n, B.pair_bits[0], 0, (long long)t.vf};
  const BatchRows ee{B.scenes, B.sc, B.pack[1], B.off.ee_cap, B.off.edge, n, B.pair_bits[1], 1, (long long)t.ee};
  const long long rows[2] = {(long long)t.V, (long long)t.E};
  rc = launch_pair_rows(C.rows, vf, ee, rows, t.most_in_row, s);
  if (rc != P2C_OK) return rc;
  export_counts_kernel<<<grid_for(n, 128), 128, 0, s>>>(B);
  P2C_CUDA(cudaGetLastError());
  return P2C_OK;
}

}  // namespace p2c

extern "C" {

size_t p2c_batch_candidates_workspace_bytes(const p2c_batch_scene* scenes_host, int32_t n_scenes) {
  if (scenes_host == nullptr || n_scenes < 1) return 0;
  const p2c::Totals t = p2c::totals_of(scenes_host, n_scenes);
  return p2c::carve(nullptr, nullptr, n_scenes, t).total;
}

int p2c_batch_candidates(const p2c_batch_scene* scenes_host, const p2c_batch_scene* scenes_dev, int32_t n_scenes,
                         void* workspace_dev, size_t workspace_bytes, void* stream) {
  if (scenes_host == nullptr || scenes_dev == nullptr) return p2c::fail(P2C_ERR_INVALID, "scene table pointer is null");
  if (n_scenes < 1 || n_scenes > (1 << 20))
    return p2c::fail(P2C_ERR_INVALID, "batch scene count must lie in [1, 2^20]");
  const int rc = p2c::validate_table(scenes_host, n_scenes);
  if (rc != P2C_OK) return rc;
  return p2c::launch_batch_candidates(scenes_host, scenes_dev, n_scenes, workspace_dev, workspace_bytes,
                                      p2c::as_stream(stream));
}

}  // extern "C"
