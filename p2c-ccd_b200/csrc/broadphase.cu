// broadphase.cu — swept-AABB candidate generation on a binned grid.
//
// Replaces the reference's CPU candidate builders: the brute-force
// BuildMeshExactCertificateQuery pair loops (cpp/certificate/
// mesh_exact_query.cpp:211-317) and the scene tool's SweepPairs /
// BuildVFCandidates / BuildEECandidates (tools/
// scene_object_envelope_native_ti_walltime.cpp:603-699).  The pair SET is
// identical: inclusive double-precision overlap on all three axes, no vertex
// against a face that contains it and no edges sharing a vertex inside one
// object, optionally no pairs inside one object at all.
//
// A one-axis sweep over a surface mesh scans windows of ~sqrt(n) boxes (a
// whole slice of surface projects onto the axis).  Here the two non-sweep
// axes are cut into columns about as wide as a typical box and every column
// into bins along the sweep axis; a box is filed under the bin of its min
// corner, ordinary and oversized boxes apart, and scans one contiguous run of
// bins in each column that an overlapping partner's min corner can lie in.
// Steps, all on the caller's stream without host synchronisation:
//   1. vertex swept boxes (t0 and t1 positions, +thickness): object
//      envelopes and per-axis statistics;
//   2. swept boxes of every vertex, face and edge and culling: with self
//      pairs excluded, a primitive outside every other object's envelope
//      cannot have a candidate (the scene tool's object-pair permission,
//      PrepareScene :521-545, used as a filter); kept boxes are appended to a
//      compact list, often a few per cent of the scene.  The launch's last
//      block chooses the sweep axis (smallest mean extent relative to the
//      spread of centres) and the bins;
//   3. counting sort into the bins: each box's rank in its bin (one atomic per
//      warp and bin), each column's place, then the boxes to their places.  The
//      order inside a bin does not matter, so no radix passes are needed;
//   4. one sweep launch for both families: 8 lanes share a box, look up its
//      columns' runs side by side and walk the runs' entries together;
//   5. pair lists that fit are ranked by counting smaller keys (all SMs at
//      once); longer ones are put into rows by their first primitive, and
//      each row orders itself (pair_rows.cuh).
// Overlapping boxes of different objects imply overlapping object envelopes
// (each box lies inside its object's envelope), so beyond culling only the
// same-object rule remains.
#include <algorithm>
#include <cmath>

#include "broadphase.cuh"
#include "pair_rows.cuh"

namespace p2c {
namespace {

constexpr int kThreads = 256;
constexpr unsigned kFull = 0xffffffffu;

inline unsigned grid_for(long long n, int threads) {
  const long long g = (n + threads - 1) / threads;
  return (unsigned)(g > 0 ? g : 1);
}

struct Lists {
  long long off[4];  // global index g: list l holds [off[l], off[l + 1])
  const int32_t* prim[3];
  const int32_t* obj[3];
  __device__ __forceinline__ int list_of(long long g) const { return g < off[1] ? 0 : (g < off[2] ? 1 : 2); }
};

constexpr int kMaxCols = 256;                   // columns per non-sweep axis
constexpr int kMinBinsZ = 8, kMaxBinsZ = 512;   // bins of a column along the sweep axis (a power of two)

// Bins of one list, size class and side: about one per four primitives of the scene.
inline long long bin_budget(long long n) {
  long long b = 1ll << 13;
  while (b < n / 4 && b < (1ll << 18)) b <<= 1;
  return b;
}

// Extents of the kept boxes of one list, as float keys rounded outward (the
// grid needs bounds, not exact values): raised by atomicMax, zero = empty.
struct ListExtent {
  unsigned active;   // boxes kept
  unsigned ext[3];   // up(largest extent)
  unsigned nlo[3];   // ~down(smallest min)
  unsigned hi[3];    // up(largest max)
};

// Size classes: where nine boxes in ten are at most half as long along a1 (a2)
// as the longest one, a box above that length limit1 (limit2) is filed apart,
// so that a scene's few oversized boxes do not widen what every other box has
// to scan (a 624k-triangle cloth on a sphere of four times larger triangles).
struct BinGrid {
  int axis, a1, a2, g1, g2;
  int classes;       // 2, or 1 when no kept box is oversized
  double limit1, limit2;
  int cols;          // g1 * g2
  int gz, zshift;    // bins per column and their log2
  // Two-body split: with self pairs excluded and exactly two objects (ids 0
  // and 1) each object has its own bins and a box walks only the other's.
  int sides;         // 2 split, 1 not
  double base1, base2, inv1, inv2;  // column = floor((x - base) * inv)
  double base0, inv0;               // bin along the sweep axis: floor((x - base0) * inv0)
  double reach1[2][3], reach2[2][3];  // per class and list: the largest extent along a1 / a2
  unsigned seg[4];                  // list l's binned entries are [seg[l], seg[l + 1])
};

// Extents by half octave from 2^-24 to 2^8 (clamped): the float's exponent
// and first mantissa bit.
constexpr int kExtentBins = 64, kExtentFirst = (127 - 24) * 2;
__device__ __forceinline__ int extent_bin(double ext) {
  const int i = (int)(__float_as_uint(__double2float_ru(ext)) >> 22) - kExtentFirst;
  return i < 0 ? 0 : (i >= kExtentBins ? kExtentBins - 1 : i);
}

struct SceneScratch {
  double extent_sum[3], center_sum[3], center_sq_sum[3];
  unsigned ext_hist[3][kExtentBins];  // kept boxes by extent (a sample of the blocks)
  unsigned long long count;
  unsigned long long obj_nlo[kMaxCullObjects][3];  // ~order keys of the objects' swept-box minima (zero = empty)
  unsigned long long obj_hi[kMaxCullObjects][3];
  ListExtent list[3];  // 0 vertices, 1 faces, 2 edges
  BinGrid grid;
  unsigned long long vf_count;
  unsigned long long ee_count;
  unsigned long long error_word;  // bit 0: non-finite coordinate
  unsigned obj_other;             // non-zero: a kept primitive's object id is neither 0 nor 1
  unsigned keyed;                 // boxes kept after culling (compact entries)
  unsigned blocks_done;           // cull blocks finished (the last sizes the grid)
  unsigned placed[3];             // entries given a place, per list
  unsigned sweep_next;            // next box of the sweep
};

// The binned boxes: per entry two 16-byte records for the float prefilter, the
// bins it scans and the exact box.
struct Binned {
  float4* cols;    // non-sweep bounds rounded outward: (alo down, ahi up, blo down, bhi up)
  float4* tag;     // (lo down, hi down, id, object)
  uint4* span;     // per class (first column's bins, columns along a2, columns, first bin | last bin << 16)
  double* box;     // 6: lo, hi along the sweep axis, alo, ahi, blo, bhi
  unsigned* count; // bins
  unsigned* start;
};

__device__ __forceinline__ int bin_z(double x, const BinGrid& g) {
  return clamp_floor((x - g.base0) * g.inv0, g.gz - 1);  // monotone in x: the runs rely on it
}
__device__ __forceinline__ unsigned first_bin(const BinGrid& g, int list, int cls, int side, int col) {
  return (unsigned)(((list * g.classes + cls) * g.sides + side) * g.cols + col) << g.zshift;
}

// A maximum that rarely grows: most calls only read it.
__device__ __forceinline__ void raise_max(unsigned* p, unsigned v) {
  if (v > *reinterpret_cast<volatile unsigned*>(p)) atomicMax(p, v);
}
__device__ __forceinline__ void raise_max(unsigned long long* p, unsigned long long v) {
  if (v > *reinterpret_cast<volatile unsigned long long*>(p)) atomicMax(p, v);
}
__device__ __forceinline__ double bound_of(unsigned key) {  // the float behind a key, as double
  return (double)__uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
}

// Block sums of the per-axis statistics that choose the sweep axis (extents,
// centres and squared centres of the boxes), ten atomics per block.
__device__ __forceinline__ void axis_stats(const double b[6], bool live, SceneScratch* sc) {
  __shared__ double red[9][kThreads / 32];
  const int lane = threadIdx.x & 31;
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
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    double v = vals[k];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(kFull, v, s);
    if (lane == 0) red[k][threadIdx.x >> 5] = v;
  }
  const unsigned cnt = __popc(__ballot_sync(kFull, live));
  __syncthreads();
  if (threadIdx.x < 9) {
    double s = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) s += red[threadIdx.x][w];
    double* dst = threadIdx.x < 3 ? &sc->extent_sum[threadIdx.x]
                  : threadIdx.x < 6 ? &sc->center_sum[threadIdx.x - 3]
                                    : &sc->center_sq_sum[threadIdx.x - 6];
    atomicAdd(dst, s);
  }
  if (lane == 0 && cnt) atomicAdd(&sc->count, (unsigned long long)cnt);
}

// Vertex swept boxes (Extend/Expand/SweptPointBox,
// scene_object_envelope_native_ti_walltime.cpp:256-301): each joins its
// object's envelope (the union of the object's vertex boxes; one atomic per
// object per warp) and the per-axis statistics that choose the sweep axis.
// Faces and edges are boxes of these vertices, so this pass also finds
// every non-finite coordinate; such a vertex takes no further part.
__global__ void __launch_bounds__(kThreads) envelope_kernel(const double* __restrict__ v_t0,
                                                            const double* __restrict__ v_t1,
                                                            const int32_t* __restrict__ v_obj, long long nv,
                                                            double thickness, int cull_objects, SceneScratch* sc) {
  pdl_wait();
  pdl_trigger();
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  double b[6] = {0, 0, 0, 0, 0, 0};
  bool live = g < nv;
  int o = -1;
  if (live) {
    live = swept_box<1>(v_t0, v_t1, nullptr, g, thickness, b);
    if (!live) atomicOr(&sc->error_word, 1ull);
    o = v_obj[g];
  }
  if (cull_objects > 0) {
    const bool mine0 = live && o >= 0 && o < cull_objects;
    unsigned remaining = __ballot_sync(kFull, mine0);
    while (remaining) {
      const int leader = __ffs((int)remaining) - 1;
      const int lo_obj = __shfl_sync(kFull, o, leader);
      const bool mine = mine0 && o == lo_obj;
      remaining &= ~__ballot_sync(kFull, mine);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        unsigned long long kmin = mine ? order_key(b[a]) : ~0ull;
        unsigned long long kmax = mine ? order_key(b[3 + a]) : 0ull;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
          kmin = min(kmin, __shfl_xor_sync(kFull, kmin, s));
          kmax = max(kmax, __shfl_xor_sync(kFull, kmax, s));
        }
        if (lane == leader) {
          raise_max(&sc->obj_nlo[lo_obj][a], ~kmin);
          raise_max(&sc->obj_hi[lo_obj][a], kmax);
        }
      }
    }
  }
  axis_stats(b, live, sc);
}

// What the grid is computed from: one warp per axis gathers it.
struct AxisInfo {
  double score;        // mean extent over the spread of centres (vertices)
  double base, range;  // where the kept boxes lie
  double reach;        // longest kept box
  double half, ninety; // extents that half / nine tenths of the kept boxes do not exceed
};
struct GridInput {
  AxisInfo axis[3];
};

// Upper edge of the histogram bin that holds the given tenth of the boxes;
// lane i holds bins 2i and 2i + 1.
__device__ __forceinline__ double extent_quantile(unsigned h0, unsigned h1, unsigned tenths) {
  const int lane = threadIdx.x & 31;
  unsigned incl = h0 + h1;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned t = __shfl_up_sync(kFull, incl, d);
    if (lane >= d) incl += t;
  }
  const unsigned want = __shfl_sync(kFull, incl, 31) / 10u * tenths;
  const unsigned at0 = __ballot_sync(kFull, incl - h1 >= want), at1 = __ballot_sync(kFull, incl >= want);
  const int i = min(at0 != 0u ? 2 * (__ffs((int)at0) - 1) : kExtentBins - 1,
                    at1 != 0u ? 2 * (__ffs((int)at1) - 1) + 1 : kExtentBins - 1);
  return (double)__uint_as_float((unsigned)(kExtentFirst + i + 1) << 22);
}

// By the first three warps of a block (read past L1: other blocks wrote it).
__device__ __forceinline__ void load_grid_input(const SceneScratch* sc, GridInput& in) {
  const int a = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (a < 3) {
    const unsigned h0 = __ldcg(&sc->ext_hist[a][2 * lane]), h1 = __ldcg(&sc->ext_hist[a][2 * lane + 1]);
    const double half = extent_quantile(h0, h1, 5u), ninety = extent_quantile(h0, h1, 9u);
    if (lane == 0) {
      AxisInfo x;
      double lo = INFINITY, top = -INFINITY;
      x.reach = 0.0;
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        if (__ldcg(&sc->list[l].active) == 0u) continue;
        lo = fmin(lo, bound_of(~__ldcg(&sc->list[l].nlo[a])));
        top = fmax(top, bound_of(__ldcg(&sc->list[l].hi[a])));
        x.reach = fmax(x.reach, bound_of(__ldcg(&sc->list[l].ext[a])));
      }
      x.base = isfinite(lo) ? lo : 0.0;
      x.range = (top > lo) ? top - lo : 0.0;
      const double n = sc->count > 0 ? (double)sc->count : 1.0;
      const double mean = sc->center_sum[a] / n;
      const double var = fmax(sc->center_sq_sum[a] / n - mean * mean, 0.0);
      x.score = (sc->extent_sum[a] / n) / (sqrt(var) + 1e-300);
      x.half = half;
      x.ninety = ninety;
      in.axis[a] = x;
    }
  }
  __syncthreads();
}

// Sweep axis, columns and bins, by one thread of the last block of the cull
// launch.  two_body: self pairs are excluded and the scene has two objects, so
// the bins split by object unless an id other than 0 and 1 was kept.  budget:
// bins of one list, class and side.
__device__ void compute_grid(SceneScratch* sc, const GridInput& in, int budget, int two_body) {
  int axis = 0;
  double best = INFINITY;
  for (int a = 0; a < 3; ++a)
    if (in.axis[a].score < best) {
      best = in.axis[a].score;
      axis = a;
    }
  BinGrid g;
  g.axis = axis;
  g.a1 = axis == 0 ? 1 : 0;
  g.a2 = axis == 2 ? 1 : 2;
  g.sides = two_body != 0 && __ldcg(&sc->obj_other) == 0u ? 2 : 1;
  const unsigned active[3] = {__ldcg(&sc->list[0].active), __ldcg(&sc->list[1].active), __ldcg(&sc->list[2].active)};
  const unsigned most = max(max(active[0], active[1]), max(active[2], 1u));
  // about two columns per box of the largest list at most
  const double col_limit = fmin((double)kMaxCols, ceil(sqrt(2.0 * (double)most)) + 7.0);
  double inv[2], limit[2];
  int cols[2] = {1, 1};
  bool oversized = false;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const AxisInfo& x = in.axis[k == 0 ? g.a1 : g.a2];
    const double half = fmin(x.reach, x.half);
    limit[k] = x.ninety <= 0.5 * x.reach ? x.ninety : x.reach;
    oversized = oversized || limit[k] < x.reach;
    // a usual box then meets about four columns per axis, one per lane of its
    // group; an axis along which it would scan most of the scene all the same
    // is not cut
    const double most_cols = k == 0 ? col_limit : fmin(col_limit, floor((double)(budget / kMinBinsZ) / (double)cols[0]));
    double width = fmax((half + limit[k]) * (1.0 / 3.0), x.range / most_cols);
    if (half + limit[k] + width > 0.6 * x.range) width = 2.0 * x.range;
    if (!(width > 0.0) || !isfinite(width)) width = 1.0;
    const int c = (int)fmin(most_cols, floor(x.range / width) + 1.0);
    cols[k] = c < 1 ? 1 : c;
    inv[k] = 1.0 / width;
  }
  g.classes = oversized ? 2 : 1;
  g.limit1 = limit[0];
  g.limit2 = limit[1];
  for (int l = 0; l < 3; ++l) {
    const double r1 = active[l] ? bound_of(__ldcg(&sc->list[l].ext[g.a1])) : 0.0;
    const double r2 = active[l] ? bound_of(__ldcg(&sc->list[l].ext[g.a2])) : 0.0;
    g.reach1[0][l] = fmin(limit[0], r1);
    g.reach2[0][l] = fmin(limit[1], r2);
    g.reach1[1][l] = r1;
    g.reach2[1][l] = r2;
  }
  g.g1 = cols[0];
  g.g2 = cols[1];
  g.cols = cols[0] * cols[1];
  g.gz = kMinBinsZ;
  g.zshift = 3;
  while (g.gz < kMaxBinsZ && 2 * g.gz * g.cols <= budget && (double)g.gz * (double)g.cols < 4.0 * (double)most) {
    g.gz *= 2;
    g.zshift += 1;
  }
  const AxisInfo& z = in.axis[axis];
  g.base1 = in.axis[g.a1].base;
  g.base2 = in.axis[g.a2].base;
  g.inv1 = inv[0];
  g.inv2 = inv[1];
  g.base0 = z.base;
  g.inv0 = (z.range > 0.0 && isfinite(z.range)) ? (double)g.gz / z.range : 0.0;
  g.seg[0] = 0u;
  g.seg[1] = active[0];
  g.seg[2] = g.seg[1] + active[1];
  g.seg[3] = g.seg[2] + active[2];
  sc->grid = g;
}

__global__ void grid_kernel(SceneScratch* sc, int budget, int two_body) {
  pdl_wait();
  pdl_trigger();
  __shared__ GridInput in;
  load_grid_input(sc, in);
  if (threadIdx.x == 0) compute_grid(sc, in, budget, two_body);
}

// Every primitive's swept box (Swept*Box, :256-301), kept unless it is a
// vertex in no face, has a non-finite coordinate or (self pairs excluded) lies
// outside every other object's envelope.  Kept boxes are appended (one atomic per warp) to a
// compact list of (box, primitive) entries that everything after works on;
// their extents per list size the grid.  The extents are 32-bit keys reduced
// by one instruction per warp and in shared memory per block: with 64-bit keys
// reduced by shuffles and ten global atomics per warp this launch took 352 us
// for the 1.9 M primitives of a 624k-triangle scene (now 89 us, 90 MB written),
// all of it waiting on the same few addresses.
__global__ void __launch_bounds__(kThreads, 4) cull_kernel(const double* __restrict__ v_t0,
                                                        const double* __restrict__ v_t1, Lists L, double thickness,
                                                        int cull_objects, int ordered, double* __restrict__ cbox,
                                                        unsigned* __restrict__ cprim, SceneScratch* sc, int budget,
                                                        int two_body) {
  pdl_wait();
  pdl_trigger();
  __shared__ ListExtent ext[3];
  __shared__ unsigned hist[3 * kExtentBins];
  __shared__ GridInput in;
  __shared__ double envelope[kMaxCullObjects][6];  // every object's, read once per block
  for (int k = threadIdx.x; k < 3 * kExtentBins; k += kThreads) hist[k] = 0u;
  for (int k = threadIdx.x; k < 3 * cull_objects; k += kThreads) {
    const int q = k / 3, a = k - 3 * q;
    const unsigned long long top = sc->obj_hi[q][a];  // zero: no vertex, an envelope nothing overlaps
    envelope[q][a] = top != 0ull ? unorder_key(~sc->obj_nlo[q][a]) : INFINITY;
    envelope[q][3 + a] = top != 0ull ? unorder_key(top) : -INFINITY;
  }
  const bool sample = blockIdx.x % (gridDim.x / 512u + 1u) == 0u;
  for (int k = threadIdx.x; k < (int)(3 * sizeof(ListExtent) / 4); k += kThreads) reinterpret_cast<unsigned*>(ext)[k] = 0u;
  __syncthreads();
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  bool keep = false, other = false;
  int l = 3;
  double b[6] = {0, 0, 0, 0, 0, 0};
  if (g < L.off[3]) {
    l = L.list_of(g);
    const long long i = g - L.off[l];
    const int o = L.obj[l][i];
    keep = !(l == 0 && o < 0);
    const bool finite = l == 0   ? swept_box<1>(v_t0, v_t1, nullptr, i, thickness, b)
                        : l == 1 ? swept_box<3>(v_t0, v_t1, L.prim[1], i, thickness, b)
                                 : swept_box<2>(v_t0, v_t1, L.prim[2], i, thickness, b);
    keep = keep && finite;
    if (keep && cull_objects > 0) {
      bool near_other = false;
      for (int q = 0; q < cull_objects && !near_other; ++q) {
        if (q == o) continue;
        bool ov = true;
#pragma unroll
        for (int a = 0; a < 3; ++a) ov = ov && b[a] <= envelope[q][3 + a] && envelope[q][a] <= b[3 + a];
        near_other = ov;
      }
      keep = near_other;
    }
    other = keep && o != 0 && o != 1;
  }
  if (__any_sync(kFull, other) && lane == 0) atomicOr(&sc->obj_other, 1u);
  if (ordered) {  // nothing is culled: every entry in place (one that is not kept is marked)
    if (g < L.off[3]) {
      double* dst = cbox + 6 * g;
#pragma unroll
      for (int k = 0; k < 6; ++k) dst[k] = b[k];
      cprim[g] = keep ? (unsigned)g : ~0u;
    }
  } else {
    const unsigned m = __ballot_sync(kFull, keep);
    if (m != 0u) {
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(&sc->keyed, (unsigned)__popc(m));
      base = __shfl_sync(kFull, base, 0);
      if (keep) {
        const unsigned c = base + (unsigned)__popc(m & ((1u << lane) - 1u));
        double* dst = cbox + 6ull * c;
#pragma unroll
        for (int k = 0; k < 6; ++k) dst[k] = b[k];
        cprim[c] = (unsigned)g;
      }
    }
  }
  // per-list extents: warp, block, then at most ten atomics per block and list
  for (int ll = 0; ll < 3; ++ll) {
    const bool mine = keep && l == ll;
    const unsigned mask = __ballot_sync(kFull, mine);
    if (mask == 0u) continue;
    if (lane == 0) atomicAdd(&ext[ll].active, (unsigned)__popc(mask));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const unsigned e = __reduce_max_sync(kFull, mine ? fkey_up(b[3 + a] - b[a]) : 0u);
      const unsigned lo = __reduce_max_sync(kFull, mine ? ~fkey_down(b[a]) : 0u);
      const unsigned hi = __reduce_max_sync(kFull, mine ? fkey_up(b[3 + a]) : 0u);
      if (lane == 0) {
        atomicMax(&ext[ll].ext[a], e);
        atomicMax(&ext[ll].nlo[a], lo);
        atomicMax(&ext[ll].hi[a], hi);
      }
    }
  }
  if (sample && keep)
    for (int a = 0; a < 3; ++a) atomicAdd(&hist[a * kExtentBins + extent_bin(b[3 + a] - b[a])], 1u);
  __syncthreads();
  if (sample)
    for (int k = threadIdx.x; k < 3 * kExtentBins; k += kThreads)
      if (hist[k] != 0u) atomicAdd(&sc->ext_hist[0][0] + k, hist[k]);
  if (threadIdx.x < 30) {
    const int ll = threadIdx.x / 10, k = threadIdx.x % 10;
    const unsigned v = reinterpret_cast<const unsigned*>(&ext[ll])[k];
    unsigned* dst = reinterpret_cast<unsigned*>(&sc->list[ll]) + k;
    if (v != 0u) {
      if (k == 0) atomicAdd(dst, v);
      else raise_max(dst, v);
    }
  }
  // the last block to finish sizes the grid from everyone's extents
  __shared__ bool last_block;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last_block = atomicAdd(&sc->blocks_done, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (last_block) {
    __threadfence();
    load_grid_input(sc, in);
    if (threadIdx.x == 0) compute_grid(sc, in, budget, two_body);
  }
}

// Bin and rank in it of every kept box (compact entry c).  Lanes of a warp
// that meet in a bin take their ranks with one atomic.
__global__ void __launch_bounds__(kThreads) bin_kernel(Lists L, const double* __restrict__ cbox,
                                                       const unsigned* __restrict__ cprim, uint2* __restrict__ spot,
                                                       unsigned* __restrict__ bin_count, const SceneScratch* sc,
                                                       unsigned ordered_n) {
  pdl_wait();
  pdl_trigger();
  const BinGrid& G = sc->grid;
  const unsigned n = ordered_n != 0u ? ordered_n : sc->keyed;
  for (unsigned base = blockIdx.x * kThreads; base < n; base += gridDim.x * kThreads) {
    const unsigned c = base + threadIdx.x;
    unsigned bin = ~0u;
    if (c < n && cprim[c] != ~0u) {
      const long long g = cprim[c];
      const int l = L.list_of(g);
      const double* b = cbox + 6ull * c;
      const int col = column(b[G.a1], G.base1, G.inv1, G.g1) * G.g2 + column(b[G.a2], G.base2, G.inv2, G.g2);
      const int side = G.sides == 2 ? L.obj[l][g - L.off[l]] : 0;
      const int cls = G.classes == 2 && (b[3 + G.a1] - b[G.a1] > G.limit1 || b[3 + G.a2] - b[G.a2] > G.limit2) ? 1 : 0;
      bin = first_bin(G, l, cls, side, col) + (unsigned)bin_z(b[G.axis], G);
    }
    const unsigned same = __match_any_sync(kFull, bin);
    const int lane = threadIdx.x & 31, leader = __ffs((int)same) - 1;
    unsigned rank = 0;
    if (lane == leader && bin != ~0u) rank = atomicAdd(bin_count + bin, (unsigned)__popc(same));
    rank = __shfl_sync(kFull, rank, leader) + (unsigned)__popc(same & ((1u << lane) - 1u));
    if (c < n) spot[c] = make_uint2(bin, rank);
  }
}

// Places of the bins: a warp takes 512 consecutive ones (whole columns, as a
// column has 8 to 512), eight per lane and half, and reserves their entries with one
// atomic per list it touches.  Columns land in any order; a column's bins are
// contiguous, which is all the sweep needs.
__global__ void __launch_bounds__(kThreads) place_kernel(Binned B, SceneScratch* sc) {
  pdl_wait();
  pdl_trigger();
  const BinGrid& G = sc->grid;
  const unsigned per_list = (unsigned)(G.classes * G.sides * G.cols) << G.zshift, bins = 3u * per_list;
  const int lane = threadIdx.x & 31;
  for (unsigned base = (blockIdx.x * kThreads + threadIdx.x) / 32u * 512u; base < bins;
       base += gridDim.x * kThreads * 16u) {
    uint4 v[2][2];
    unsigned sum[2], incl[2], place[2] = {0u, 0u};
    int l[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned bin = base + 256u * (unsigned)h + 8u * (unsigned)lane;
      v[h][0] = v[h][1] = make_uint4(0u, 0u, 0u, 0u);
      l[h] = 3;
      if (bin < bins) {
        v[h][0] = *reinterpret_cast<const uint4*>(B.count + bin);
        v[h][1] = *reinterpret_cast<const uint4*>(B.count + bin + 4);
        l[h] = bin < per_list ? 0 : (bin < 2u * per_list ? 1 : 2);
      }
      sum[h] = v[h][0].x + v[h][0].y + v[h][0].z + v[h][0].w + v[h][1].x + v[h][1].y + v[h][1].z + v[h][1].w;
      incl[h] = sum[h];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned t = __shfl_up_sync(kFull, incl[h], d);
        if (lane >= d) incl[h] += t;
      }
    }
    incl[1] += __shfl_sync(kFull, incl[0], 31);
    for (int ll = 0; ll < 3; ++ll) {
      // entries of this list among the warp's bins, and before them
      const unsigned m0 = __ballot_sync(kFull, l[0] == ll), m1 = __ballot_sync(kFull, l[1] == ll);
      if ((m0 | m1) == 0u) continue;
      const int f0 = __ffs((int)m0) - 1, f1 = __ffs((int)m1) - 1, e0 = 31 - __clz((int)m0), e1 = 31 - __clz((int)m1);
      const unsigned before0 = __shfl_sync(kFull, incl[0] - sum[0], max(f0, 0));
      const unsigned before1 = __shfl_sync(kFull, incl[1] - sum[1], max(f1, 0));
      const unsigned last0 = __shfl_sync(kFull, incl[0], max(e0, 0)), last1 = __shfl_sync(kFull, incl[1], max(e1, 0));
      const unsigned before = m0 != 0u ? before0 : before1;
      const unsigned total = (m1 != 0u ? last1 : last0) - before;
      unsigned at = 0;
      if (lane == 0 && total != 0u) at = atomicAdd(&sc->placed[ll], total);
      at = G.seg[ll] + __shfl_sync(kFull, at, 0) - before;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (l[h] == ll) place[h] = at + incl[h] - sum[h];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned bin = base + 256u * (unsigned)h + 8u * (unsigned)lane;
      if (bin >= bins) continue;
      uint4 p, q;
      p.x = place[h];
      p.y = p.x + v[h][0].x;
      p.z = p.y + v[h][0].y;
      p.w = p.z + v[h][0].z;
      q.x = p.w + v[h][0].w;
      q.y = q.x + v[h][1].x;
      q.z = q.y + v[h][1].y;
      q.w = q.z + v[h][1].z;
      *reinterpret_cast<uint4*>(B.start + bin) = p;
      *reinterpret_cast<uint4*>(B.start + bin + 4) = q;
    }
  }
}

// Kept boxes to their places.
__global__ void __launch_bounds__(kThreads) scatter_kernel(Lists L, const double* __restrict__ cbox,
                                                           const unsigned* __restrict__ cprim,
                                                           const uint2* __restrict__ spot, Binned B,
                                                           const SceneScratch* sc, unsigned ordered_n) {
  pdl_wait();
  pdl_trigger();
  const BinGrid& G = sc->grid;
  const unsigned n = ordered_n != 0u ? ordered_n : sc->keyed;
  for (unsigned c = blockIdx.x * kThreads + threadIdx.x; c < n; c += gridDim.x * kThreads) {
    const uint2 at = spot[c];
    if (at.x == ~0u) continue;
    const long long g = cprim[c];
    const int l = L.list_of(g);
    const long long j = g - L.off[l];
    const unsigned i = B.start[at.x] + at.y;
    const double* b = cbox + 6ull * c;
    const double lo = b[G.axis], hi = b[3 + G.axis], alo = b[G.a1], ahi = b[3 + G.a1], blo = b[G.a2], bhi = b[3 + G.a2];
    B.cols[i] = fbox_entry(alo, ahi, blo, bhi);
    B.tag[i] = make_float4(__double2float_rd(lo), __double2float_rd(hi), __int_as_float((int)j),
                           __int_as_float(L.obj[l][j]));
    double2* x = reinterpret_cast<double2*>(B.box + 6ull * i);
    x[0] = make_double2(lo, hi);
    x[1] = make_double2(alo, ahi);
    x[2] = make_double2(blo, bhi);
    // The columns its partners' min corners can lie in, per class; the lower
    // ones are widened by a relative 2^-40 so that the rounding of alo - reach
    // never skips one.  One thread per box here; in the sweep every lane of the
    // box's group would repeat it.
    const int target = l == 2 ? 2 : 1 - l, side = G.sides == 2 ? 1 - L.obj[l][j] : 0;
    const int e1 = column(ahi, G.base1, G.inv1, G.g1), e2 = column(bhi, G.base2, G.inv2, G.g2);
    const unsigned z = (unsigned)bin_z(lo, G) | ((unsigned)bin_z(hi, G) << 16);
    for (int cls = 0; cls < 2; ++cls) {
      uint4 span = make_uint4(0u, 1u, 0u, 0u);
      if (cls < G.classes) {
        const double r1 = G.reach1[cls][target], r2 = G.reach2[cls][target];
        const int c1 = column(alo - r1 - (fabs(alo) + r1) * 0x1p-40, G.base1, G.inv1, G.g1);
        const int c2 = column(blo - r2 - (fabs(blo) + r2) * 0x1p-40, G.base2, G.inv2, G.g2);
        span = make_uint4(first_bin(G, target, cls, side, c1 * G.g2 + c2), (unsigned)(e2 - c2 + 1),
                          (unsigned)((e1 - c1 + 1) * (e2 - c2 + 1)), z);
      }
      B.span[2ull * i + cls] = span;
    }
  }
}

// Lanes that share one scanning box: they look its columns' runs up side by
// side and walk all runs as one list, eight entries at a time.  A 624k-triangle
// cloth's candidates with 4 / 8 / 16 / 32 lanes per box: 1.89 / 1.81 / 1.96 /
// 2.24 ms; five resident blocks (48 registers) against four: 1.81 and 1.91 ms.
#ifndef P2C_SWEEP_LANES
#define P2C_SWEEP_LANES 8
#endif
constexpr int kSweepLanes = P2C_SWEEP_LANES;
#ifndef P2C_SWEEP_BLOCKS
#define P2C_SWEEP_BLOCKS 5
#endif

struct PairOut {
  unsigned long long* out;
  unsigned long long cap;
  int shift;
  int on;
};

// Bound by dependent loads and issue (DRAM idle, 40 % of issue slots): per
// entry two 16-byte loads and a float test, exact doubles only for survivors,
// pairs staged per warp.  624k-triangle cloth, 1.9 M boxes, 50 M entries
// scanned, 3.1 M pairs: 1.14 ms for both families, against 2.63 ms for two
// launches that binary-searched radix-sorted columns with one lane per column;
// 27 bodies of 20,000 triangles, 10.5 M pairs: 5.6 -> 1.2 ms.
//
// Vertex-face pairs: vertices scan faces and own the pairs whose face minimum
// is >= the vertex minimum, faces scan vertices and own the others; keys
// (vertex, face).  Edge-edge pairs: an edge owns the pairs whose partner
// minimum is larger (ties: larger edge index); keys (lower, higher).
__global__ void __launch_bounds__(kThreads, P2C_SWEEP_BLOCKS)
    sweep_kernel(Binned B, const int32_t* __restrict__ faces, const int32_t* __restrict__ edges, int exclude_self,
                 PairOut vf, PairOut ee, SceneScratch* sc) {
  pdl_wait();
  pdl_trigger();
  __shared__ unsigned long long slots[2][kThreads / 32][96];
  const BinGrid& g = sc->grid;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int member = lane & (kSweepLanes - 1), sub = lane / kSweepLanes;
  constexpr unsigned kBoxes = 32 / kSweepLanes;
  PairBuffer vfb{slots[0][warp], 0u}, eeb{slots[1][warp], 0u};
  const unsigned vf_end = g.seg[2], all_end = g.seg[3], stride = (unsigned)g.g2;
  const int zshift = g.zshift;
  // steps of kBoxes boxes, one family each
  const unsigned vf_steps = vf.on ? (vf_end + kBoxes - 1u) / kBoxes : 0u;
  const unsigned steps = vf_steps + (ee.on ? (all_end - vf_end + kBoxes - 1u) / kBoxes : 0u);
  const unsigned chunk = max(1u, min(32u, steps / (gridDim.x * (kThreads / 32) * 8u)));
  for (;;) {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&sc->sweep_next, chunk);
    base = __shfl_sync(kFull, base, 0);
    if (base >= steps) break;
    for (unsigned t = base; t < min(base + chunk, steps); ++t) {
      const bool is_vf = t < vf_steps;
      const unsigned i = is_vf ? t * kBoxes + (unsigned)sub : vf_end + (t - vf_steps) * kBoxes + (unsigned)sub;
      const bool live = i < (is_vf ? vf_end : all_end);
      const bool from_vertex = is_vf && i < g.seg[1];
      int id = 0, obj = 0, columns = 0;
      float4 pc = make_float4(0.f, 0.f, 0.f, 0.f), pt = pc;
      uint4 span = make_uint4(0u, 1u, 0u, 0u), large = span;
      if (live) {
        pc = B.cols[i];
        pt = B.tag[i];
        span = B.span[2ull * i];
        large = B.span[2ull * i + 1];
        id = __float_as_int(pt.z);
        obj = __float_as_int(pt.w);
        columns = (int)(span.z + large.z);
      }
      for (int c = member; __any_sync(kFull, c - member < columns); c += kSweepLanes) {
        unsigned offset = 0, len = 0;
        if (c < columns) {
          const bool ordinary = (unsigned)c < span.z;
          const unsigned k = ordinary ? (unsigned)c : (unsigned)c - span.z, n2 = ordinary ? span.y : large.y;
          const unsigned d1 = k / n2;
          const unsigned bin = (ordinary ? span.x : large.x) + ((d1 * stride + k - d1 * n2) << zshift);
          const unsigned last = bin + (span.w >> 16);
          offset = B.start[bin + (span.w & 0xffffu)];
          len = run_length(offset, B.start[last] + B.count[last]);
        }
        unsigned before = len;  // inclusive, then exclusive sum of the runs' lengths over the box's lanes
#pragma unroll
        for (int d = 1; d < kSweepLanes; d <<= 1) {
          const unsigned t = __shfl_up_sync(kFull, before, d, kSweepLanes);
          if (member >= d) before += t;
        }
        const unsigned entries = __shfl_sync(kFull, before, kSweepLanes - 1, kSweepLanes);
        before -= len;
        offset -= before;
        for (unsigned k = (unsigned)member; __any_sync(kFull, k < entries); k += kSweepLanes) {
          int run = 0;  // the last run that starts at or before entry k
#pragma unroll
          for (int d = kSweepLanes / 2; d > 0; d >>= 1) {
            const unsigned at = __shfl_sync(kFull, before, run + d, kSweepLanes);
            if (at <= k) run += d;
          }
          const unsigned j = __shfl_sync(kFull, offset, run, kSweepLanes) + k;
          bool found = false;
          unsigned long long key = 0;
          if (k < entries) {
            const float4 qt = B.tag[j], qc = B.cols[j];
            const int qid = __float_as_int(qt.z), qobj = __float_as_int(qt.w);
            // rounding down is monotone: a partner minimum below lo or above hi
            // shows in the floats or passes to the exact test
            const bool maybe = !(qt.x < pt.x) && !(qt.x > pt.y) && !(exclude_self && qobj == obj) &&
                               fmay_overlap(FBox{pc.x, pc.y, pc.z, pc.w}, qc);
            if (maybe) {
              // this box's own bounds are read again here (from L1): kept in
              // registers through the walk they cost a resident block
              const double2* x = reinterpret_cast<const double2*>(B.box + 6ull * j);
              const double2* y = reinterpret_cast<const double2*>(B.box + 6ull * i);
              const double2 q0 = x[0], q1 = x[1], q2 = x[2], p0 = y[0], p1 = y[1], p2 = y[2];
              const bool own = is_vf ? (from_vertex ? q0.x >= p0.x : q0.x > p0.x)
                                     : q0.x > p0.x || (q0.x == p0.x && qid > id);
              found = own && p0.x <= q0.y && q0.x <= p0.y && p1.x <= q1.y && q1.x <= p1.y && p2.x <= q2.y &&
                      q2.x <= p2.y;
              if (found && qobj == obj) {  // no self exclusion: the mesh's own adjacency is no contact
                if (is_vf) {
                  const int vtx = from_vertex ? id : qid;
                  const int32_t* fv = faces + 3 * (long long)(from_vertex ? qid : id);
                  found = !(__ldg(fv) == vtx || __ldg(fv + 1) == vtx || __ldg(fv + 2) == vtx);
                } else {
                  const int32_t* ea = edges + 2 * (long long)id;
                  const int32_t* eb = edges + 2 * (long long)qid;
                  const int a0 = __ldg(ea), a1 = __ldg(ea + 1), b0 = __ldg(eb), b1 = __ldg(eb + 1);
                  found = !(a0 == b0 || a0 == b1 || a1 == b0 || a1 == b1);
                }
              }
              if (found)
                key = is_vf ? pair_key((unsigned)(from_vertex ? id : qid), (unsigned)(from_vertex ? qid : id), vf.shift)
                            : pair_key((unsigned)min(id, qid), (unsigned)max(id, qid), ee.shift);
            }
          }
          if (is_vf) vfb.append(found, key, vf.out, vf.cap, &sc->vf_count);
          else eeb.append(found, key, ee.out, ee.cap, &sc->ee_count);
        }
      }
    }
  }
  if (vfb.n != 0u) vfb.flush(vfb.n, vf.out, vf.cap, &sc->vf_count);
  if (eeb.n != 0u) eeb.flush(eeb.n, ee.out, ee.cap, &sc->ee_count);
}

__device__ __forceinline__ unsigned long long unpack_pair(unsigned long long k, int shift) {
  return ((k >> shift) << 32) | (k & ((1ull << shift) - 1ull));
}

__device__ __forceinline__ void export_counts(const SceneScratch* sc, unsigned long long* counts) {
  counts[0] = sc->vf_count;
  counts[1] = sc->ee_count;
  counts[2] = sc->error_word;
  counts[3] = (unsigned long long)sc->grid.axis | ((unsigned long long)sc->grid.g1 << 8) |
              ((unsigned long long)sc->grid.g2 << 24) | ((unsigned long long)sc->grid.seg[3] << 40);
}

// Pair lists whose capacities are at most kRankSortCap are sorted by rank, in
// one launch for both families: a key's place is the number of smaller keys
// (keys are unique), counted by eight threads per key over tiles of the list
// in shared memory, on as many blocks as there are 32-key groups.  n^2
// comparisons, but spread over the GPU: 3,700 edge pairs take 10.7 us where one
// block's radix sort took 20.5 us (both with cold caches).  The line: all
// candidates of a scene by ranks / by rows, both lists' buffers as large as the
// larger list: 1,554 pairs 58 / 87 us, 3,770 89 / 91, 7,388 136 / 103, 18,629 251 / 122.
// Buffers have room to spare (1.25 to 1.4 times and more), so 8,192 places hold
// the lists that ranks suit.
constexpr long long kRankSortCap = 8192;
constexpr int kRankKeys = 32;
constexpr int kRankTile = 2048;

struct RankList {
  const unsigned long long* src;
  unsigned long long* dst;
  long long cap;
  int shift;
};

__global__ void __launch_bounds__(kRankKeys * 8) rank_sort_kernel(RankList vf, RankList ee, unsigned vf_blocks,
                                                                  const SceneScratch* sc,
                                                                  unsigned long long* counts) {
  pdl_wait();
  pdl_trigger();
  __shared__ unsigned long long tile[kRankTile];
  if (blockIdx.x == 0 && threadIdx.x == 0) export_counts(sc, counts);  // final once the sweep is done
  const bool is_vf = blockIdx.x < vf_blocks;
  const RankList R = is_vf ? vf : ee;
  const long long count = (long long)(is_vf ? sc->vf_count : sc->ee_count);
  const int n = (int)(count < R.cap ? count : R.cap);
  const int k = (int)(blockIdx.x - (is_vf ? 0u : vf_blocks)) * kRankKeys + (int)(threadIdx.x >> 3);
  const int part = threadIdx.x & 7;
  if (k - (int)(threadIdx.x >> 3) >= n) {  // no key in this block, only padding
    if (part == 0 && k < R.cap) R.dst[k] = ~0ull;
    return;
  }
  const unsigned long long mine = k < n ? R.src[k] : 0ull;
  unsigned smaller = 0;
  for (int base = 0; base < n; base += kRankTile) {
    const int m = min(kRankTile, n - base);
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += kRankKeys * 8) tile[i] = R.src[base + i];
    __syncthreads();
    int i = part;
    for (; i + 24 < m; i += 32)
      smaller += (unsigned)(tile[i] < mine) + (unsigned)(tile[i + 8] < mine) + (unsigned)(tile[i + 16] < mine) +
                 (unsigned)(tile[i + 24] < mine);
    for (; i < m; i += 8) smaller += (unsigned)(tile[i] < mine);
  }
#pragma unroll
  for (int d = 4; d > 0; d >>= 1) smaller += __shfl_xor_sync(kFull, smaller, d);
  if (part != 0) return;
  if (k < n) R.dst[smaller] = unpack_pair(mine, R.shift);
  else if (k < R.cap) R.dst[k] = ~0ull;
}

__global__ void export_counts_kernel(const SceneScratch* sc, unsigned long long* counts) {
  pdl_wait();
  pdl_trigger();
  export_counts(sc, counts);
}

// ---- workspace carving -----------------------------------------------------
struct Carver {
  char* base;
  size_t off = 0;
  bool dry;
  template <class T>
  T* take(long long count) {
    off = (off + 255) & ~size_t(255);
    T* p = dry ? nullptr : reinterpret_cast<T*>(base + off);
    off += sizeof(T) * (size_t)(count > 0 ? count : 1);
    return p;
  }
};

struct Layout {
  SceneScratch* sc;
  size_t zero_bytes;  // the scratch and the bin counts behind it start at zero
  long long budget;   // bins of one list and side
  Binned bins;
  double* cbox;       // kept boxes, compaction order
  unsigned* cprim;    // their primitive indices
  uint2* spot;        // their bins and ranks
  unsigned long long* unsorted[2];  // pair lists before the rank sort
  RowScratch rows;                  // for longer lists
  size_t total;
};

Layout carve(void* base, long long nv, long long nf, long long ne, long long pair_cap, bool dry) {
  Carver c{static_cast<char*>(base), 0, dry};
  Layout L;
  const long long n = nv + nf + ne;
  L.budget = bin_budget(n);
  L.sc = c.take<SceneScratch>(1);
  L.bins.count = c.take<unsigned>(12 * L.budget);
  L.zero_bytes = c.off;
  L.bins.start = c.take<unsigned>(12 * L.budget);
  L.bins.cols = c.take<float4>(n);
  L.bins.tag = c.take<float4>(n);
  L.bins.span = c.take<uint4>(2 * n);
  L.bins.box = c.take<double>(6 * n);
  L.cbox = c.take<double>(6 * n);
  L.cprim = c.take<unsigned>(n);
  L.spot = c.take<uint2>(n);
  L.unsorted[0] = c.take<unsigned long long>(std::min(pair_cap, kRankSortCap));
  L.unsorted[1] = c.take<unsigned long long>(std::min(pair_cap, kRankSortCap));
  const long long caps[2] = {pair_cap, pair_cap};
  if (pair_cap > kRankSortCap) L.rows = carve_rows(nv + ne, caps, [&](size_t b) { return (void*)c.take<char>((long long)b); });
  L.total = c.off + 256;
  return L;
}

int bit_length(long long x) {
  int b = 0;
  while (x > 0) {
    ++b;
    x >>= 1;
  }
  return b;
}

}  // namespace

int validate_scene(const p2c_scene* sc) {
  if (sc == nullptr) return fail(P2C_ERR_INVALID, "scene pointer is null");
  if (sc->nv < 0 || sc->nf < 0 || sc->ne < 0) return fail(P2C_ERR_INVALID, "scene counts must be non-negative");
  if (sc->nv + sc->nf + sc->ne >= (1ll << 31)) return fail(P2C_ERR_INVALID, "scene primitive count must stay below 2^31");
  if (!(sc->thickness >= 0.0) || !std::isfinite(sc->thickness))
    return fail(P2C_ERR_INVALID, "scene thickness must be finite and non-negative");
  if (sc->n_obj < 0) return fail(P2C_ERR_INVALID, "scene n_obj must be non-negative");
  if (sc->nv > 0 && (sc->v_t0 == nullptr || sc->v_t1 == nullptr || sc->v_obj == nullptr))
    return fail(P2C_ERR_INVALID, "scene vertex arrays are null");
  if (sc->nf > 0 && (sc->faces == nullptr || sc->f_obj == nullptr))
    return fail(P2C_ERR_INVALID, "scene face arrays are null");
  if (sc->ne > 0 && (sc->edges == nullptr || sc->e_obj == nullptr))
    return fail(P2C_ERR_INVALID, "scene edge arrays are null");
  return P2C_OK;
}

size_t broadphase_workspace_bytes(long long nv, long long nf, long long ne, long long pair_cap) {
  return carve(nullptr, nv, nf, ne, pair_cap, true).total;
}


// Blocks of a loop over device-counted work: what the device holds at once.
template <class K>
unsigned resident_grid(K kernel, const DeviceInfo& info) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  return (unsigned)std::max(1, info.sm_count) * (unsigned)per_sm;
}

// Candidate generation; counts_dev receives {vf_count, ee_count, error_word,
// axis | g1 << 8 | g2 << 24 | kept boxes << 40}.
int launch_broadphase(const p2c_scene& scene, unsigned long long* vf_out, long long vf_cap,
                      unsigned long long* ee_out, long long ee_cap, unsigned long long* counts_dev, bool sort_out,
                      void* ws, size_t ws_bytes, cudaStream_t s) {
  const long long pair_cap = std::max(vf_cap, ee_cap);
  const size_t need = broadphase_workspace_bytes(scene.nv, scene.nf, scene.ne, pair_cap);
  if (ws == nullptr || ws_bytes < need)
    return fail(P2C_ERR_INVALID, "candidate workspace too small: %zu < %zu bytes", ws_bytes, need);
  Layout L = carve(ws, scene.nv, scene.nf, scene.ne, pair_cap, false);
  const long long n = scene.nv + scene.nf + scene.ne;
  const int cull = (scene.exclude_self && scene.n_obj >= 1 && scene.n_obj <= kMaxCullObjects) ? scene.n_obj : 0;
  const bool ordered = cull == 0;  // nothing culled: entries stay in primitive order, no compaction
  Lists lists;
  lists.off[0] = 0;
  lists.off[1] = scene.nv;
  lists.off[2] = scene.nv + scene.nf;
  lists.off[3] = n;
  lists.prim[0] = nullptr;
  lists.prim[1] = scene.faces;
  lists.prim[2] = scene.edges;
  lists.obj[0] = scene.v_obj;
  lists.obj[1] = scene.f_obj;
  lists.obj[2] = scene.e_obj;
  DeviceInfo info;
  int rc = current_device_info(&info);
  if (rc != P2C_OK) return rc;
  P2C_CUDA(cudaMemsetAsync(L.sc, 0, L.zero_bytes, s));
  if (scene.nv > 0)
    P2C_CUDA(launch_pdl(envelope_kernel, dim3(grid_for(scene.nv, kThreads)), dim3(kThreads), 0, s, scene.v_t0,
                        scene.v_t1, scene.v_obj, (long long)scene.nv, scene.thickness, cull, L.sc));
  const int two_body = scene.exclude_self && scene.n_obj == 2 ? 1 : 0;
  const bool do_vf = scene.nv + scene.nf > 0 && vf_out != nullptr;
  const bool do_ee = scene.ne > 0 && ee_out != nullptr;
  // with sorting, pairs are emitted packed so that the sort touches fewer bits
  const int vf_shift = sort_out ? std::max(1, bit_length(scene.nf)) : 0;
  const int ee_shift = sort_out ? std::max(1, bit_length(scene.ne)) : 0;
  const bool rank_sort = sort_out && pair_cap <= kRankSortCap;
  if (n > 0) {
    P2C_CUDA(launch_pdl(cull_kernel, dim3(grid_for(n, kThreads)), dim3(kThreads), 0, s, scene.v_t0, scene.v_t1,
                        lists, scene.thickness, cull, ordered ? 1 : 0, L.cbox, L.cprim, L.sc, (int)L.budget,
                        two_body));
    const unsigned ordered_n = ordered ? (unsigned)n : 0u;
    const unsigned loop_grid = std::min(grid_for(n, kThreads), resident_grid(scatter_kernel, info));
    P2C_CUDA(launch_pdl(bin_kernel, dim3(loop_grid), dim3(kThreads), 0, s, lists, (const double*)L.cbox,
                        (const unsigned*)L.cprim, L.spot, L.bins.count, (const SceneScratch*)L.sc, ordered_n));
    P2C_CUDA(launch_pdl(place_kernel, dim3(std::min(grid_for(12 * L.budget, 16 * kThreads), 8u * info.sm_count)),
                        dim3(kThreads), 0, s, L.bins, L.sc));
    P2C_CUDA(launch_pdl(scatter_kernel, dim3(loop_grid), dim3(kThreads), 0, s, lists, (const double*)L.cbox,
                        (const unsigned*)L.cprim, (const uint2*)L.spot, L.bins, (const SceneScratch*)L.sc,
                        ordered_n));
    if (do_vf || do_ee) {
      const PairOut vf{rank_sort ? L.unsorted[0] : vf_out, (unsigned long long)vf_cap, vf_shift, do_vf ? 1 : 0};
      const PairOut ee{rank_sort ? L.unsorted[1] : ee_out, (unsigned long long)ee_cap, ee_shift, do_ee ? 1 : 0};
      P2C_CUDA(launch_pdl(sweep_kernel, dim3(std::min(grid_for(n * kSweepLanes, kThreads), resident_grid(sweep_kernel, info))),
                          dim3(kThreads), 0, s, L.bins, scene.faces, scene.edges, scene.exclude_self, vf, ee, L.sc));
    }
  } else {  // no primitive, no cull launch: the (empty) grid on its own
    P2C_CUDA(launch_pdl(grid_kernel, dim3(1), dim3(96), 0, s, L.sc, (int)L.budget, two_body));
  }
  if (rank_sort) {
    const unsigned vf_blocks = vf_cap > 0 ? grid_for(vf_cap, kRankKeys) : 0u;
    const unsigned ee_blocks = ee_cap > 0 ? grid_for(ee_cap, kRankKeys) : 0u;
    P2C_CUDA(launch_pdl(rank_sort_kernel, dim3(std::max(1u, vf_blocks + ee_blocks)), dim3(kRankKeys * 8), 0, s,
                        RankList{L.unsorted[0], vf_out, vf_cap, vf_shift},
                        RankList{L.unsorted[1], ee_out, ee_cap, ee_shift}, vf_blocks, (const SceneScratch*)L.sc,
                        counts_dev));
  } else if (sort_out) {
    const long long rows[2] = {scene.nv, scene.ne}, most_in_row[2] = {scene.nf, scene.ne};
    rc = launch_pair_rows(L.rows, SceneRows{vf_out, &L.sc->vf_count, vf_cap, vf_shift},
                          SceneRows{ee_out, &L.sc->ee_count, ee_cap, ee_shift}, rows, most_in_row, s);
    if (rc != P2C_OK) return rc;
  }
  if (!rank_sort)  // the rank sort writes the counts itself
    P2C_CUDA(launch_pdl(export_counts_kernel, dim3(1), dim3(1), 0, s, (const SceneScratch*)L.sc, counts_dev));
  P2C_CUDA(cudaGetLastError());
  return P2C_OK;
}

}  // namespace p2c

extern "C" {

size_t p2c_scene_candidates_workspace_bytes(int64_t nv, int64_t nf, int64_t ne, int64_t vf_cap, int64_t ee_cap) {
  return p2c::broadphase_workspace_bytes(nv, nf, ne, vf_cap > ee_cap ? vf_cap : ee_cap);
}

int p2c_scene_candidates(const p2c_scene* scene, uint64_t* vf_pairs_dev, int64_t vf_cap, uint64_t* ee_pairs_dev,
                         int64_t ee_cap, uint64_t* counts_dev, int sort_pairs, void* workspace_dev,
                         size_t workspace_bytes, void* stream) {
  int rc = p2c::validate_scene(scene);
  if (rc != P2C_OK) return rc;
  if (counts_dev == nullptr) return p2c::fail(P2C_ERR_INVALID, "counts pointer is null");
  if (vf_cap < 0 || ee_cap < 0) return p2c::fail(P2C_ERR_INVALID, "pair capacities must be non-negative");
  if ((vf_cap > 0 && vf_pairs_dev == nullptr) || (ee_cap > 0 && ee_pairs_dev == nullptr))
    return p2c::fail(P2C_ERR_INVALID, "pair output pointer is null");
  return p2c::launch_broadphase(*scene, reinterpret_cast<unsigned long long*>(vf_pairs_dev), vf_cap,
                                reinterpret_cast<unsigned long long*>(ee_pairs_dev), ee_cap,
                                reinterpret_cast<unsigned long long*>(counts_dev), sort_pairs != 0, workspace_dev,
                                workspace_bytes, p2c::as_stream(stream));
}

}  // extern "C"
