// certify_engine.cuh — the persistent warp engine of the interval certifier.
//
// A query is one interval tree (one primitive over one interval).  A warp
// keeps up to kSlots queries in shared memory and ONE stack of their pending
// nodes.  Every iteration pops up to 32 nodes, one per lane, takes each node's
// midpoint sample, and pushes the two children of every node that splits,
// left child on top: lanes are never tied to a tree, so none idles while the
// warp holds 32 nodes, and nothing is handed from lane to lane.  A node needs
// only its midpoint sample: its endpoints are midpoints or endpoints of
// ancestors, already known to be farther than eps_space (otherwise the
// ancestor would be a collision leaf and would not have been split).  A root
// takes three samples (t0, t1, mid) on three lanes.
//
// When the stack holds few nodes, the idle lanes sample the nodes' descendants
// in the same iteration: one node and its next four levels fill 31 lanes, two
// nodes and three levels 30, and so on.  A descendant counts only if every
// ancestor in the group turns out to split (a ballot and at most four bit
// tests), so results are unchanged, and the chain of dependent samples of a
// deep tree shortens by up to five: a warp's instructions cost the same
// whether one lane or all take part.
//
// Across warps: when some warp has nothing to do, a warp holding
// more nodes than one iteration takes publishes its shallowest ones to a
// global pool that idle warps drain, so one deep tree is bisected by many
// warps.
//
// The reduction of a tree reproduces the recursion's result exactly: the
// leftmost collision leaf in depth-first order wins (keys are left-aligned
// paths with a sentinel bit below the last level, so disjoint nodes compare
// in depth-first order and the key encodes the leaf), else any undecided leaf
// makes the tree undecided, else separation with the minimum leaf margin.  A
// tree's reduction lives in its warp's slot; once one of its nodes leaves the
// warp, every warp that held part of it adds its slot's reduction to a pooled
// record, and the last one writes the result.  Nodes right of a known
// collision are pruned: the recursion never reaches them.
//
// Bound by instruction issue and the latency of dependent FP64 chains, not by
// memory: on a 156k-triangle cloth's fallback trees (edge-edge) 51 % of the issue
// slots and 31 % of the FP64 pipe are busy, DRAM idle, four warps per scheduler
// (128 registers).  So a full iteration has a path of its own without the
// groups' bookkeeping, the sample is one out-of-line function for both paths,
// and all warps work on one family at a time: the code is 67 KB, and
// instruction fetch stalls cost up to 20 % otherwise.  Against the engine
// that tied a lane to a subtree and handed subtrees between lanes, on a B200:
// two 40,960-triangle spheres 75 -> 33 us (12 iterations on the longest warp
// instead of 27), 20,000 plain queries 365 -> 180 us, a 60,000-triangle cloth's
// 295,000 self candidates 780 -> 420 us, a 624k-triangle cloth's 1.9 M any-hit
// certificates 10.3 -> 8.5 ms, 64 uneven scenes 283 -> 190 us; slower only where
// each warp has one deep tree of the same size from the start (1,200 of 8,191
// nodes 362 -> 459, of a launch that shares none).  Idle warps hold a
// ticket each and poll their own pool entry: with one shared head that they
// advanced by compare-and-swap the 20,000 queries took 1,200 us.  A bracket of
// the distance in single precision that spared 95 % of the FP64 samples made
// the loop longer, not shorter (cloth 445 -> 690 us), and was dropped.
//
// No wait in this engine is unbounded: the loop checks the launch's device
// time budget (CertParams::budget_ns, never zero); on expiry the engine
// returns false and the launcher reports P2C_ERR_TIMEOUT.
#pragma once

#include "certify_core.cuh"

namespace p2c {

// Global reduction record of a tree whose subtrees left its warp.
struct TreeAgg {
  unsigned long long coll_key;     // min leaf_key over collision leaves (~0: none)
  unsigned long long margin_bits;  // min separation margin (bit pattern of a non-negative double)
  unsigned int undecided;          // any undecided leaf
  unsigned int outstanding;        // live units: warps holding part of it + pooled nodes
};

struct SubtreeTask {
  unsigned long long path;  // the node's leaf key (path and depth)
  unsigned long long tag;   // 1 + (q << 24 | agg index (16 bits) << 8 | family - 1); 0 = unpublished
};

// Launch-wide counters, one 128-byte line each: idle warps poll some of them
// while busy warps update others.
struct alignas(128) PaddedCounter {
  unsigned long long v;
  unsigned long long pad[15];
};

struct EngineState {
  PaddedCounter queue_head[2];  // next query of each family
  PaddedCounter finalized;      // queries finished (both families)
  PaddedCounter task_reserve;   // pooled nodes published (or about to be)
  PaddedCounter task_head;      // tickets of warps that took or wait for one
  PaddedCounter agg_next;       // TreeAgg records handed out
  PaddedCounter helpers;        // idle warps allowed to stay and wait
};

struct EnginePools {
  TreeAgg* aggs = nullptr;        // capacity agg_cap
  SubtreeTask* tasks = nullptr;   // capacity task_cap
  unsigned long long agg_cap = 0;
  unsigned long long task_cap = 0;
  unsigned long long helper_cap = 0;  // idle warps that wait for subtrees
};

constexpr int kMaxTreeDepth = 63;  // leaf keys need one bit below the deepest level

// Shape of the loop below (compile-time), with the times of other values, us a
// pass after an L2 flush: 20,000 plain queries / two spheres of 40,960 triangles
// / a 60,000-triangle cloth's self candidates / a 624k-triangle cloth's any-hit.
// As set: 213 / 140 / 634 / 10,540; repeats differ by 1 % in the first, 0.2 % in
// the others.
//   P2C_ENGINE_SLOTS   queries a warp keeps in flight (at most 32).
//                      8: 215 / 140 / 676 / 9,728; 32: 192 / 138 / 693 / 13,213
//                      (three blocks an SM);
//   P2C_ENGINE_STACK   pending nodes a warp can hold (a power of two).
//                      512: 183 / 138 / 695 / 10,585 (three blocks an SM);
//   P2C_ROOT_BATCH     queries fetched together (three root samples each).
//                      5: 213 / 140 / 664 / 10,000;
//   P2C_EXPORT_LANES   nodes one warp may publish to the pool per reading of its
//                      counters.  1: 302 / 140 / 665 / 10,933; 3: 264 / 140 / 649 / 10,645;
//   P2C_OVERSUPPLY     unclaimed nodes the pool may hold before warps stop
//                      publishing.  64: 213 / 140 / 638 / 10,543;
//   P2C_BACKOFF        longest sleep between two polls of an idle warp (ns).
//                      64: 215 / 140 / 637 / 10,525; 1,024: 211 / 140 / 633 / 10,537;
//   P2C_EXPORT_ABOVE   a warp publishes nodes beyond this many.
//                      16: 219 / 140 / 644 / 10,614; 64: 207 / 140 / 631 / 10,507;
//   P2C_FINISH_BATCH   finished queries a warp collects before it writes their
//                      results together (their writes are chains of dependent
//                      loads, stores and atomics).
//                      1: 215 / 140 / 695 / 10,846; 16: 215 / 140 / 639 / 9,500;
//   P2C_GUIDED         a warp claims at most 1 / (P2C_GUIDED * warps) of the
//                      queries left in a queue (and one more).
//                      2: 207 / 143 / 634 / 10,546; 4: 221 / 143 / 641 / 10,532;
//   P2C_HUNGRY_PERIOD  iterations between reads of the pool's counters (a
//                      power of two).  1: 233 / 142 / 656 / 10,603; 8: 221 / 140 / 631 / 10,543.
// P2C_HELPERS_PER_SM (certify_launch.cuh, 8): 2: 199 / 138 / 649 / 10,814; 16: 241 / 145 /
// 648 / 10,617.  P2C_CERTIFY_BLOCKS (4): 3: 193 / 138 / 688 / 12,259; 5: 224 / 142 / 674 /
// 11,001.  No value is best at all four; these lose least.
#ifndef P2C_ENGINE_SLOTS
#define P2C_ENGINE_SLOTS 16
#endif
#ifndef P2C_ENGINE_STACK
#define P2C_ENGINE_STACK 256
#endif
#ifndef P2C_ROOT_BATCH
#define P2C_ROOT_BATCH 10
#endif
#ifndef P2C_EXPORT_LANES
#define P2C_EXPORT_LANES 6
#endif
#ifndef P2C_OVERSUPPLY
#define P2C_OVERSUPPLY 0
#endif
#ifndef P2C_BACKOFF
#define P2C_BACKOFF 256u
#endif
#ifndef P2C_EXPORT_ABOVE
#define P2C_EXPORT_ABOVE 32
#endif
#ifndef P2C_GUIDED
#define P2C_GUIDED 1u
#endif
#ifndef P2C_FINISH_BATCH
#define P2C_FINISH_BATCH 8
#endif
#ifndef P2C_HUNGRY_PERIOD
#define P2C_HUNGRY_PERIOD 2
#endif
constexpr int kSlots = P2C_ENGINE_SLOTS;
constexpr unsigned kStack = P2C_ENGINE_STACK;
constexpr int kRootBatch = P2C_ROOT_BATCH;
static_assert(kSlots <= 32, "slots are one warp mask");
static_assert(kRootBatch <= 10, "three lanes per root");
static_assert((kStack & (kStack - 1)) == 0 && kStack >= 160, "64 entries stay free for a depth-first descent");
static_assert((P2C_HUNGRY_PERIOD & (P2C_HUNGRY_PERIOD - 1)) == 0, "P2C_HUNGRY_PERIOD must be a power of two");

// Phase clock of one warp iteration, compiled only with -DP2C_ENGINE_PROFILE
// (a measurement build; the library is built without it): lane 0 of every
// warp adds the SM clock cycles spent in each phase of the loop below to
// g_engine_prof (0 fetch, 1 pop, 2 pool take, 3 idle wait, 4 distance sample,
// 5 classify, 6 record, 7 push, 8 export, 9 finalise, 10 budget check,
// 11 iterations).
#ifdef P2C_ENGINE_PROFILE
static __device__ unsigned long long g_engine_prof[16];
#define P2C_PROF_DECL              \
  unsigned long long prof_t = 0;   \
  unsigned long long prof_acc[12]; \
  for (int _k = 0; _k < 12; ++_k) prof_acc[_k] = 0ull;
#define P2C_PROF_START() prof_t = clock64();
#define P2C_PROF_MARK(k)                               \
  {                                                    \
    __syncwarp();                                      \
    const unsigned long long _now = clock64();         \
    prof_acc[k] += _now - prof_t;                      \
    prof_t = _now;                                     \
  }
#define P2C_PROF_FLUSH()                                                               \
  if ((threadIdx.x & 31) == 0)                                                         \
    for (int _k = 0; _k < 12; ++_k) atomicAdd(&g_engine_prof[_k], prof_acc[_k]);
#define P2C_PROF_COUNT(k) prof_acc[k] += 1ull;
#else
#define P2C_PROF_DECL
#define P2C_PROF_START()
#define P2C_PROF_MARK(k)
#define P2C_PROF_FLUSH()
#define P2C_PROF_COUNT(k)
#endif

__device__ __forceinline__ unsigned long long leaf_key(unsigned long long path, int depth) {
  return path | (1ull << (63 - depth));
}

// Publication of pooled nodes and the last decrement of a shared tree: a
// release store of the task tag and an acquire load by its taker, and an
// acquire-release decrement of the tree's outstanding units.
__device__ __forceinline__ void store_release(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long load_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned decrement_acq_rel(unsigned* p) {  // returns the value before
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(0xffffffffu) : "memory");
  return old;
}

__device__ __forceinline__ unsigned long long volatile_load(const unsigned long long* p) {
  return *reinterpret_cast<const volatile unsigned long long*>(p);
}
__device__ __forceinline__ unsigned volatile_load(const unsigned* p) {
  return *reinterpret_cast<const volatile unsigned*>(p);
}

// A warp's shared state: its queries (struct-of-arrays [k][slot], so lanes
// reading different slots hit different banks and lanes reading one slot
// broadcast), their reductions, and the stack of pending nodes.
struct EngineShared {
  double p0[12][kSlots];
  double p1[12][kSlots];
  double nrm[4][kSlots];                 // motion norms (MotionRadius factors)
  double rate[2][kSlots];                // the two that the radius takes, once the largest are chosen
  double T0[kSlots], T1[kSlots];
  unsigned long long coll_key[kSlots];   // leftmost collision leaf known to this warp (~0: none)
  unsigned long long margin[kSlots];     // min separation margin (bits); a colliding root's time of impact
  long long qidx[kSlots];
  int family[kSlots];
  int undecided[kSlots];
  int outstanding[kSlots];               // the query's nodes on this warp's stack
  int gidx[kSlots];                      // TreeAgg index once shared, else -1
  int batch[32];                         // slots of the roots fetched together
  unsigned long long nkey[kStack];       // stack: leaf keys (path and depth), intervals, slots
  double nt0[kStack], nt1[kStack];
  unsigned short nmeta[kStack];          // slot | depth << 8
};

constexpr unsigned long long kRootKey = 1ull << 63;  // leaf_key of the root

__device__ __forceinline__ void fill_slot(EngineShared& sh, int s, const Geo& g, double T0, double T1, int family,
                                          long long q, unsigned long long coll_key, int gidx) {
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    sh.p0[i][s] = g.p0[i];
    sh.p1[i][s] = g.p1[i];
  }
  double nrm[4];
  NoCount nc;
  motion_norms(SlotGeo<EngineShared>{sh, s}, nrm, nc);
#pragma unroll
  for (int i = 0; i < 4; ++i) sh.nrm[i][s] = nrm[i];
  sh.rate[0][s] = family == 1 ? nrm[0] : max_std(nrm[0], nrm[1]);
  sh.rate[1][s] = family == 1 ? max_std(max_std(nrm[1], nrm[2]), nrm[3]) : max_std(nrm[2], nrm[3]);
  sh.T0[s] = T0;
  sh.T1[s] = T1;
  sh.coll_key[s] = coll_key;
  sh.margin[s] = 0x7ff0000000000000ull;  // +inf
  sh.qidx[s] = q;
  sh.family[s] = family;
  sh.undecided[s] = 0;
  sh.outstanding[s] = 1;
  sh.gidx[s] = gidx;
}

// Motion radius of slot s over [t0, t1].  A product with a positive half width
// rounds monotonically, so the largest of the reference's products is the
// product with the largest norm, bit for bit; a zero half width (a zero-width
// root) takes the reference's own order, which an infinite norm can tell apart.
__device__ __forceinline__ double slot_radius(const EngineShared& sh, int s, double t0, double t1) {
  const double h = mul(0.5, max_std(0.0, sub(t1, t0)));
  if (h > 0.0) return add(mul(h, sh.rate[0][s]), mul(h, sh.rate[1][s]));
  NoCount ops;
  const double nrm[4] = {sh.nrm[0][s], sh.nrm[1][s], sh.nrm[2][s], sh.nrm[3][s]};
  return sh.family[s] == 1 ? motion_radius<1>(nrm, t0, t1, ops) : motion_radius<2>(nrm, t0, t1, ops);
}

// One FP64 sample.  Out of line: inlined into both paths of the loop it cost
// 15 % where both families are certified.
static __device__ __noinline__ double slot_distance(const EngineShared& sh, int s, int family, double t) {
  NoCount ops;
  const SlotGeo<EngineShared> g{sh, s};
  return family == 1 ? distance_at<1>(g, t, ops) : distance_at<2>(g, t, ops);
}

// A node goes to stack entry e.
__device__ __forceinline__ void put_node(EngineShared& sh, unsigned e, unsigned long long key, double t0, double t1,
                                         int slot, int depth) {
  e &= kStack - 1u;
  sh.nkey[e] = key;
  sh.nt0[e] = t0;
  sh.nt1[e] = t1;
  sh.nmeta[e] = (unsigned short)(slot | (depth << 8));
}

// Both children of a split node, the left one on top.
__device__ __forceinline__ void push_children(EngineShared& sh, unsigned e, unsigned long long key, double t0,
                                              double mid, double t1, int slot, int depth) {
  const unsigned long long half = (1ull << 62) >> depth;  // the sentinel bit of the children
  put_node(sh, e, key + half, mid, t1, slot, depth + 1);
  put_node(sh, e + 1u, key - half, t0, mid, slot, depth + 1);
}

// A leaf joins its tree's reduction here: a collision, a separation's margin.
__device__ __forceinline__ void record_collision(EngineShared& sh, int slot, unsigned long long key,
                                                 const EnginePools& pools) {
  if (key < sh.coll_key[slot]) {
    atomicMin(&sh.coll_key[slot], key);
    const int gi = sh.gidx[slot];
    if (gi >= 0) atomicMin(&pools.aggs[gi].coll_key, key);
  }
}
__device__ __forceinline__ void record_margin(EngineShared& sh, int slot, double margin) {
  const unsigned long long mb = (unsigned long long)__double_as_longlong(margin);
  if (mb < sh.margin[slot]) atomicMin(&sh.margin[slot], mb);
}

// The tree's result from its reduction.
__device__ __forceinline__ Outcome tree_outcome(unsigned long long coll_key, unsigned long long margin, bool undecided,
                                                double T0, double T1) {
  Outcome o{P2C_STATUS_SEPARATION, T0, T1, T1, __longlong_as_double((long long)margin)};
  if (coll_key != ~0ull) {
    o.status = P2C_STATUS_COLLISION;
    o.margin = 0.0;
    if (coll_key == kRootKey) {
      o.toi = __longlong_as_double((long long)margin);
    } else {  // the leaf is recovered from its key
      const int d = 64 - __ffsll((long long)coll_key);
      replay(T0, T1, coll_key & ~(1ull << (63 - d)), d, o.t0, o.t1);
      o.toi = mul(0.5, add(o.t0, o.t1));
    }
  } else if (undecided) {
    o.status = P2C_STATUS_UNDECIDED;
    o.margin = 0.0;
  }
  return o;
}

// The problem a launch certifies: both families' queries.  P provides
//   long long n(int family) const;
//   bool skip(int family, long long q) const;   // drop q unevaluated (a cancelled candidate)
//   void load(int family, long long q, Geo&, double& T0, double& T1, int& bad) const;
//   void finish(int family, long long q, const Outcome&) const;
//   void invalid(int family, long long q, int bad, double T0, double T1) const;
template <class P>
__device__ bool run_engine(const P& prob, const CertParams& prm, int fetch1, int fetch2,
                           EngineShared& sh, WarpStats& st, EngineState* es, const EnginePools& pools,
                           unsigned long long t_start) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  const long long n1 = prob.n(1), n2 = prob.n(2);
  const unsigned long long n_total = (unsigned long long)(n1 + n2);

  unsigned top = 0u, bottom = 0u;          // stack [bottom, top), indices modulo kStack
  unsigned free_mask = kSlots == 32 ? FULL : (1u << kSlots) - 1u;
  // Family whose queue this warp drains: edge-edge, then vertex-face, the same
  // on every warp, so that the instruction caches hold one family's sample at a
  // time (odd warps starting with the other family cost 6 % on a cloth's two queues).
  int cur = 2;
  unsigned exhausted = (n1 == 0 ? 1u : 0u) | (n2 == 0 ? 2u : 0u);  // bit f-1: family f's queue is empty
  bool helper = false;                     // this warp is counted in es->helpers
  bool waiting = false;                    // this warp holds the ticket of a pool entry
  unsigned long long ticket = 0;
  unsigned backoff = 64;                   // ns slept per idle poll (doubles up to P2C_BACKOFF)
  unsigned long long published = 0, tickets = 0;  // the pool's counters, as last read
  unsigned done_mask = 0u;                 // slots whose query is finished here, result not yet written
  long long claimed1 = 0, claimed2 = 0;    // queue positions known to be claimed
  const unsigned warps = gridDim.x * (blockDim.x >> 5);
  bool ok = true;
  P2C_PROF_DECL

  P2C_PROF_START()
  for (unsigned iter = 0;; ++iter) {
    if ((iter & 63u) == 0u) {
      int over = 0;
      if (lane == 0) over = (global_ns() - t_start) > prm.budget_ns;
      if (__shfl_sync(FULL, over, 0)) {
        ok = false;
        break;
      }
    }
    P2C_PROF_MARK(10)
    const unsigned size = top - bottom;
    // ---- results of finished queries, several at a time ------------------------
    if (done_mask != 0u && (size == 0u || __popc(done_mask) >= P2C_FINISH_BATCH)) {
      bool finish = (done_mask >> lane) & 1u;
      if (finish) {
        const int gi = sh.gidx[lane];
        unsigned long long ck = sh.coll_key[lane], mb = sh.margin[lane];
        bool und = sh.undecided[lane] != 0;
        if (gi >= 0) {  // shared: add this warp's part; the last part writes the result
          TreeAgg& A = pools.aggs[gi];
          atomicMin(&A.margin_bits, mb);
          if (und) atomicOr(&A.undecided, 1u);
          finish = decrement_acq_rel(&A.outstanding) == 1u;
          if (finish) {
            ck = volatile_load(&A.coll_key);
            mb = volatile_load(&A.margin_bits);
            und = volatile_load(&A.undecided) != 0u;
          }
        }
        if (finish)
          prob.finish(sh.family[lane], sh.qidx[lane], tree_outcome(ck, mb, und, sh.T0[lane], sh.T1[lane]));
      }
      const unsigned finished = __ballot_sync(FULL, finish);
      if (finished != 0u && lane == 0) atomicAdd(&es->finalized.v, (unsigned long long)__popc(finished));
      free_mask |= done_mask;
      done_mask = 0u;
      __syncwarp();
    }
    P2C_PROF_MARK(9)
    const bool read_pool = (iter & (P2C_HUNGRY_PERIOD - 1u)) == 0u;
    if (read_pool) {  // read here, used at the end of the iteration
      published = volatile_load(&es->task_reserve.v);
      tickets = volatile_load(&es->task_head.v);
    }
    bool roots = false;
    int fetched = 0;
    // ---- (A) new queries from the per-family queues -------------------------
    if (size < 32u && exhausted != 3u) {
      if (exhausted & (1u << (cur - 1))) cur = 3 - cur;
      const int limit = min(cur == 1 ? fetch1 : fetch2, kSlots);
      const long long nc = cur == 1 ? n1 : n2;
      // smaller batches as the queue runs out, so that no warp is left with many queries at the end
      const unsigned left = (unsigned)min(max(nc - (cur == 1 ? claimed1 : claimed2), 0ll), 1ll << 30);
      const int share = (int)min((unsigned)kRootBatch, left / (P2C_GUIDED * warps) + 1u);
      const int want = min(limit - (kSlots - __popc(free_mask)), share);
      // wait for a full batch of free slots while there are nodes to work on
      if (want > 0 && (size == 0u || 2 * want >= min(limit, share))) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&es->queue_head[cur - 1].v, (unsigned long long)want);
        base = __shfl_sync(FULL, base, 0);
        (cur == 1 ? claimed1 : claimed2) = (long long)base + want;
        if ((long long)base + want >= nc) exhausted |= 1u << (cur - 1);
        const long long q = (long long)base + lane;
        bool fresh = false, gone = false;
        int s = 0;
        if (lane < want && q < nc) {
          if (prob.skip(cur, q)) {
            gone = true;
          } else {
            Geo g;
            double T0, T1;
            int bad = 0;
            prob.load(cur, q, g, T0, T1, bad);
            if (bad != 0) {
              prob.invalid(cur, q, bad, T0, T1);
              gone = true;
            } else {
              s = nth_set_bit(free_mask, lane);
              fill_slot(sh, s, g, T0, T1, cur, q, ~0ull, -1);
              fresh = true;
            }
          }
        }
        const unsigned dropped = __ballot_sync(FULL, gone), got = __ballot_sync(FULL, fresh);
        if (dropped != 0u && lane == 0) atomicAdd(&es->finalized.v, (unsigned long long)__popc(dropped));
        if (got == 0u) continue;
        free_mask &= ~__reduce_or_sync(FULL, fresh ? (1u << s) : 0u);
        if (fresh) sh.batch[__popc(got & lt_mask)] = s;
        __syncwarp();
        fetched = __popc(got);
        st.queries += (unsigned)fetched;
        roots = true;
      }
    }
    P2C_PROF_MARK(0)
    if (!roots) {
      if (size == 0u) {
        // ---- (B) no node and no query left: a node from the global pool ------
        // A ticket names the pool entry this warp gets; it polls that entry
        // alone, so waiting warps do not contend.
        if (!waiting) {
          if (!helper) {  // at most helper_cap idle warps stay to take nodes; the others leave
            int stay = 0;
            if (lane == 0) stay = atomicAdd(&es->helpers.v, 1ull) < pools.helper_cap;
            helper = __shfl_sync(FULL, stay, 0) != 0;
            if (!helper) break;
          }
          if (lane == 0) ticket = atomicAdd(&es->task_head.v, 1ull);
          ticket = __shfl_sync(FULL, ticket, 0);
          waiting = true;
          backoff = 64u;
        }
        SubtreeTask* tk = pools.tasks + (ticket & (pools.task_cap - 1ull));
        unsigned long long tag = 0;
        int all_done = 0;  // one lane's read for the warp: the lanes leave together
        if (lane == 0) {
          tag = load_acquire(&tk->tag);
          all_done = tag == 0ull && volatile_load(&es->finalized.v) >= n_total;
        }
        tag = __shfl_sync(FULL, tag, 0);
        if (tag == 0ull) {
          if (__shfl_sync(FULL, all_done, 0)) break;
          __nanosleep(backoff);
          backoff = min(backoff * 2u, P2C_BACKOFF);
          P2C_PROF_MARK(3)
          continue;
        }
        waiting = false;
        if (lane == 0) {  // into slot 0: every slot and the whole stack are free
          tag -= 1ull;
          const int f = (int)(tag & 1ull) + 1;
          const int gi = (int)((tag >> 8) & 0xffffull);
          const long long q = (long long)(tag >> 24);
          const unsigned long long key = volatile_load(&tk->path);
          store_release(&tk->tag, 0ull);  // the entry is free for the pool's next lap
          Geo g;
          int bad = 0;
          double T0, T1, a, b;
          prob.load(f, q, g, T0, T1, bad);
          fill_slot(sh, 0, g, T0, T1, f, q, volatile_load(&pools.aggs[gi].coll_key), gi);
          const int d = 64 - __ffsll((long long)key);
          replay(T0, T1, key & ~(1ull << (63 - d)), d, a, b);
          put_node(sh, 0u, key, a, b, 0, d);
        }
        free_mask &= ~1u;
        bottom = 0u;
        top = 1u;
        __syncwarp();
        P2C_PROF_MARK(2)
        continue;
      }
    }
    P2C_PROF_COUNT(11)
    st.iters += 1u;
    const double eps_space = prm.eps_space;
    // Up to ten nodes fill the lanes with their descendants; with groups up to
    // four or six nodes only, two spheres take 149 or 143 us instead of 140.
    if (!roots && size > 10u) {
      // ---- (C) up to 32 nodes, one per lane -----------------------------------------
      const int count = max(1, min((int)min(size, 32u), (int)(kStack - 64u) - (int)size));  // room for a descent
      top -= (unsigned)count;
      const bool in = lane < count;
      int slot = 0, depth = 0;
      unsigned long long key = 0;
      double t0 = 0.0, t1 = 0.0;
      if (in) {
        const unsigned e = (top + (unsigned)(count - 1 - lane)) & (kStack - 1u);  // lane 0 takes the topmost
        const unsigned meta = sh.nmeta[e];
        slot = (int)(meta & 0xffu);
        depth = (int)(meta >> 8);
        key = sh.nkey[e];
        t0 = sh.nt0[e];
        t1 = sh.nt1[e];
      }
      const double mid = mul(0.5, add(t0, t1));
      P2C_PROF_MARK(1)
      bool split = false;
      const bool eval = in && !(sh.coll_key[slot] < key);  // a node right of a known collision is never needed
      if (eval) {
        const double d = slot_distance(sh, slot, sh.family[slot], mid);
        if (d <= eps_space) {
          record_collision(sh, slot, key, pools);
        } else {
          const double lb = sub(d, slot_radius(sh, slot, t0, t1));
          if (lb > eps_space) record_margin(sh, slot, max_std(0.0, sub(lb, eps_space)));
          else if (depth >= prm.max_depth || sub(t1, t0) <= prm.eps_time) sh.undecided[slot] = 1;
          else split = true;
        }
      }
      P2C_PROF_MARK(4)
      const unsigned pushers = __ballot_sync(FULL, split);
      st.nodes += (unsigned)__popc(__ballot_sync(FULL, eval));
      if (split)
        push_children(sh, top + 2u * (unsigned)__popc(pushers & (0xfffffffeu << lane)), key, t0, mid, t1, slot, depth);
      top += 2u * (unsigned)__popc(pushers);
      P2C_PROF_MARK(7)
      const unsigned same = __match_any_sync(FULL, in ? slot : -1);
      bool done = false;
      if (in && (same & lt_mask) == 0u) {  // one lane per query
        const int left = sh.outstanding[slot] + 2 * __popc(pushers & same) - __popc(same);
        sh.outstanding[slot] = left;
        done = left == 0;
      }
      if (__any_sync(FULL, done)) done_mask |= __reduce_or_sync(FULL, done ? 1u << slot : 0u);
      __syncwarp();
    } else {
      // ---- (D) roots, or a few nodes with their descendants: groups of lanes --------
      int levels, groups;
      if (roots) {
        groups = fetched;
        levels = groups == 1 ? 4 : (groups <= 3 ? 3 : (groups <= 6 ? 2 : 1));
      } else {
        groups = (int)size;
        levels = size == 1u ? 5 : (size == 2u ? 4 : (size <= 4u ? 3 : 2));
        top -= size;
      }
      const int width = (1 << levels) + (roots ? 1 : -1);
      const int group = (int)((unsigned)(lane * (65536 / width + 1)) >> 16);
      const int first = group * width;  // lane of the group's node
      const bool in = group < groups;
      int h = lane - first + 1, slot = 0, depth = 0;
      if (roots && h >= width - 1) h = h == width ? -1 : 0;  // endpoints t1 (-1) and t0 (0)
      unsigned long long key = kRootKey;
      double t0 = 0.0, t1 = 0.0;
      if (in) {
        if (roots) {
          slot = sh.batch[group];
          t0 = sh.T0[slot];
          t1 = sh.T1[slot];
        } else {
          const unsigned e = (top + (unsigned)(groups - 1 - group)) & (kStack - 1u);  // group 0 is the topmost
          const unsigned meta = sh.nmeta[e];
          slot = (int)(meta & 0xffu);
          depth = (int)(meta >> 8);
          key = sh.nkey[e];
          t0 = sh.nt0[e];
          t1 = sh.nt1[e];
        }
      }
      const bool eval = in && !(sh.coll_key[slot] < key);
      double mid = mul(0.5, add(t0, t1));
#pragma unroll 1
      for (int b = 30 - __clz(max(h, 1)); b >= 0; --b) {  // down to this lane's descendant
        const unsigned long long half = depth < 63 ? (1ull << 62) >> depth : 0ull;
        depth += 1;
        if ((h >> b) & 1) {
          t0 = mid;
          key += half;
        } else {
          t1 = mid;
          key -= half;
        }
        mid = mul(0.5, add(t0, t1));
      }
      P2C_PROF_MARK(1)
      double d = 0.0;
      if (eval) d = slot_distance(sh, slot, sh.family[slot], h > 0 ? mid : (h == 0 ? t0 : t1));
      P2C_PROF_MARK(4)
      // classify: 0 none, 1 collision, 2 separation, 3 undecided
      const bool hit = eval && d <= eps_space;
      int leaf = 0;
      double margin = 0.0;
      bool split = false, root_hit = false;
      if (roots) {
        const unsigned hits = __ballot_sync(FULL, hit);
        if (eval && h == 1) {
          const bool hit0 = (hits >> (first + width - 2)) & 1u, hit1 = (hits >> (first + width - 1)) & 1u;
          if (hit0 || hit || hit1) {  // the root is the only node; its time of impact is the first hit of t0, mid, t1
            root_hit = true;
            sh.coll_key[slot] = kRootKey;
            sh.margin[slot] = (unsigned long long)__double_as_longlong(hit0 ? t0 : (hit ? mid : t1));
          }
        }
      }
      if (eval && h > 0 && !root_hit) {
        if (hit) {
          leaf = 1;
        } else {
          const double lb = sub(d, slot_radius(sh, slot, t0, t1));
          if (lb > eps_space) {
            leaf = 2;
            margin = max_std(0.0, sub(lb, eps_space));
          } else if (depth >= prm.max_depth || sub(t1, t0) <= prm.eps_time) {
            leaf = 3;
          } else {
            split = true;
          }
        }
      }
      bool reached = eval && h > 0;
      if (levels > 1) {
        const unsigned splits = __ballot_sync(FULL, split);
#pragma unroll 1
        for (int a = h >> 1; a > 0; a >>= 1) reached = reached && ((splits >> (first + a - 1)) & 1u);
      }
      st.nodes += (unsigned)__popc(__ballot_sync(FULL, reached));
      P2C_PROF_MARK(5)
      if (reached) {
        if (leaf == 1) record_collision(sh, slot, key, pools);
        else if (leaf == 2) record_margin(sh, slot, margin);
        else if (leaf == 3) sh.undecided[slot] = 1;
      }
      P2C_PROF_MARK(6)
      const bool push = reached && split && h >= (1 << (levels - 1));
      const unsigned pushers = __ballot_sync(FULL, push);
      if (push)
        push_children(sh, top + 2u * (unsigned)__popc(pushers & (0xfffffffeu << lane)), key, t0, mid, t1, slot, depth);
      top += 2u * (unsigned)__popc(pushers);
      P2C_PROF_MARK(7)
      const unsigned same = __match_any_sync(FULL, in ? slot : -1);
      const unsigned popped = __ballot_sync(FULL, in && lane == first);
      unsigned done = 0u;
      if (in && (same & lt_mask) == 0u) {  // one lane per query
        const int left = sh.outstanding[slot] + 2 * __popc(pushers & same) - __popc(popped & same);
        sh.outstanding[slot] = left;
        if (left == 0) done = 1u << slot;
      }
      done_mask |= __reduce_or_sync(FULL, done);
      __syncwarp();
    }
    // ---- (I) publish the shallowest nodes to hungry warps ---------------------------
    // Waiting warps hold the tickets past the published count.  Only what one
    // iteration cannot take is given away, at most P2C_EXPORT_LANES nodes per
    // reading of the counters and none while P2C_OVERSUPPLY are unclaimed, so
    // the unclaimed entries (at most P2C_OVERSUPPLY + P2C_EXPORT_LANES per
    // warp) never reach the ring's size.
    if (read_pool) {
      const bool give = tickets + P2C_OVERSUPPLY > published && top - bottom > P2C_EXPORT_ABOVE;
      if (__any_sync(FULL, give)) {  // the lanes' reads of the counters may differ
        int count = min(max((int)(top - bottom) - P2C_EXPORT_ABOVE, 0), P2C_EXPORT_LANES);
        const unsigned e = (bottom + (unsigned)lane) & (kStack - 1u);
        const int es_slot = lane < count ? (int)(sh.nmeta[e] & 0xffu) : -1;
        unsigned mine = __match_any_sync(FULL, es_slot);
        const bool lead = lane < count && (mine & lt_mask) == 0u;
        // a tree's first published node moves its reduction to a pooled record
        if (lead && sh.gidx[es_slot] < 0) {
          const unsigned long long idx = atomicAdd(&es->agg_next.v, 1ull);
          if (idx < pools.agg_cap) {
            TreeAgg& A = pools.aggs[idx];
            A.coll_key = sh.coll_key[es_slot];
            A.margin_bits = 0x7ff0000000000000ull;
            A.undecided = 0u;
            A.outstanding = 1u;  // this warp's part
            __threadfence();
            sh.gidx[es_slot] = (int)idx;
          }
        }
        __syncwarp();
        const int gi = lane < count ? sh.gidx[es_slot] : -1;
        const unsigned without = __ballot_sync(FULL, gi < 0);  // no record left, or beyond count
        count = without != 0u ? __ffs((int)without) - 1 : count;
        unsigned long long task = 0;
        if (lane == 0 && count > 0) task = atomicAdd(&es->task_reserve.v, (unsigned long long)count);
        task = __shfl_sync(FULL, task, 0);
        mine &= count > 0 ? FULL >> (32 - count) : 0u;
        unsigned gone = 0u;
        if (lead && lane < count) {
          const int given = __popc(mine), left = sh.outstanding[es_slot] - given;
          sh.outstanding[es_slot] = left;
          TreeAgg& A = pools.aggs[gi];
          if (left == 0) {  // nothing of the tree stays: its part goes with one of the nodes
            atomicMin(&A.margin_bits, sh.margin[es_slot]);
            if (sh.undecided[es_slot] != 0) atomicOr(&A.undecided, 1u);
            gone = 1u << es_slot;
          }
          const unsigned more = (unsigned)given - (left == 0 ? 1u : 0u);
          if (more != 0u) atomicAdd(&A.outstanding, more);
        }
        __syncwarp();
        bool lost = false;
        if (lane < count) {
          SubtreeTask* tk = pools.tasks + ((task + (unsigned long long)lane) & (pools.task_cap - 1ull));
          // The taker of the ring's previous lap has long read the entry: the
          // ring holds more than all warps can have published and not taken
          // (certify_shape).  Wait for it all the same, and if the budget ends
          // first fail the launch: a node written over would be lost.
#pragma unroll 1
          for (unsigned spin = 0; volatile_load(&tk->tag) != 0ull && !lost; ++spin) {
            __nanosleep(64);
            lost = (spin & 255u) == 255u && (global_ns() - t_start) > prm.budget_ns;
          }
          if (!lost) {
            tk->path = sh.nkey[e];
            const unsigned long long tag = (((unsigned long long)sh.qidx[es_slot] << 24) |
                                            ((unsigned long long)gi << 8) |
                                            (unsigned long long)(sh.family[es_slot] - 1)) + 1ull;
            __threadfence();  // the leader's record updates come before the tag
            store_release(&tk->tag, tag);
          }
        }
        if (__any_sync(FULL, lost)) {
          ok = false;
          break;
        }
        st.donations += (unsigned)count;
        bottom += (unsigned)count;
        free_mask |= __reduce_or_sync(FULL, gone);
        __syncwarp();
      }
    }
    P2C_PROF_MARK(8)
  }
  P2C_PROF_FLUSH()
  return ok;
}

// The recursion's own walk of one tree, depth-first on one lane, counting its
// nodes, samples and FP64 operations (the census launch).  Returns false when
// the time budget ends first.
__device__ inline bool walk_tree(const Geo& g, int family, double T0, double T1, const CertParams& prm,
                                 unsigned long long t_start, Outcome& out, CensusStats& st) {
  struct Points {
    const Geo& g;
    __device__ __forceinline__ double p0(int k) const { return g.p0[k]; }
    __device__ __forceinline__ double p1(int k) const { return g.p1[k]; }
  };
  const Points pts{g};
  OpCount ops;
  double nrm[4];
  motion_norms(pts, nrm, ops);
  auto sample = [&](double t) {
    st.evals += 1;
    return family == 1 ? distance_at<1>(pts, t, ops) : distance_at<2>(pts, t, ops);
  };
  double st0[kMaxTreeDepth + 1], st1[kMaxTreeDepth + 1];  // pending right siblings
  int sdepth[kMaxTreeDepth + 1], pending = 0;
  double t0 = T0, t1 = T1, margin = INFINITY;
  int depth = 0;
  bool undecided = false;
  out = Outcome{P2C_STATUS_COLLISION, T0, T1, T0, 0.0};
  st.nodes += 1;
  const double d0 = sample(T0);
  double d1 = 0.0;
  bool done = d0 <= prm.eps_space;  // the root collides at t0
  if (!done) d1 = sample(T1);
  for (unsigned k = 0; !done; ++k) {
    if ((k & 63u) == 63u && global_ns() - t_start > prm.budget_ns) return false;
    const double mid = mul(0.5, add(t0, t1));
    ops.add(2);
    if (depth > 0) st.nodes += 1;
    const double d = sample(mid);
    if (d <= prm.eps_space || (depth == 0 && d1 <= prm.eps_space)) {
      out.t0 = t0;
      out.t1 = t1;
      out.toi = d <= prm.eps_space ? mid : t1;
      done = true;
      break;
    }
    const double lb = sub(d, family == 1 ? motion_radius<1>(nrm, t0, t1, ops) : motion_radius<2>(nrm, t0, t1, ops));
    ops.add(1);
    if (lb > prm.eps_space) {
      const double m = max_std(0.0, sub(lb, prm.eps_space));
      ops.add(1);
      if (m < margin) margin = m;
    } else if (depth >= prm.max_depth || sub(t1, t0) <= prm.eps_time) {
      undecided = true;
    } else {
      st0[pending] = mid;
      st1[pending] = t1;
      sdepth[pending++] = ++depth;
      t1 = mid;
      continue;
    }
    if (pending == 0) break;
    --pending;
    t0 = st0[pending];
    t1 = st1[pending];
    depth = sdepth[pending];
  }
  st.ops += ops.n;
  if (!done)
    out = undecided ? Outcome{P2C_STATUS_UNDECIDED, T0, T1, T1, 0.0}
                    : Outcome{P2C_STATUS_SEPARATION, T0, T1, T1, margin};
  return true;
}

}  // namespace p2c
