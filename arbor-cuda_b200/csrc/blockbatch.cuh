// blockbatch.cuh - block-batched primitive tests for forest rays.
//
// The reference tests one candidate primitive at a time inside its BVH loop
// (Arbor.cu:226).  On a GPU that serialises a warp: the rare, long tests
// (the leaf Newton solve, the bark SDF march) run with one or two lanes
// active.  Here each lane traverses on its own (tracer.cuh) and, instead of
// testing a candidate, queues it (up to kQueue per lane); the 256 threads of a CTA
// then run everything that was queued as compacted jobs - leaf clips, Newton
// solves of the clips that pass, wood tests and the rest - one job per thread,
// and each lane applies its own results.
//
// The whole CTA goes through the stages together (advance for at most kSlice
// steps, classify, clip, solve, march, apply; barriers between them).  What
// binds these passes is instruction fetch: the stages together are some
// 100 KB of code, an SM's warps run them from one instruction cache, and with
// warps that moved through the stages on their own (16 per SM, each somewhere
// else) 60 % of the warps' waiting was for instructions.  In step, one fetch
// serves eight warps, and the jobs of eight warps fill the test passes.
//
// Why results do not change: the primitive surfaces lie inside their own
// bounding boxes (the leaf-frame box, petiole, bark relief and ellipsoid are
// built inside boundLow/boundHigh, Arbor.cu:132-133), so a hit t is not below
// the box's entry span.x, and the reference only prunes boxes with span.x >=
// best.  A primitive it prunes then cannot beat its final answer, and the
// answer is the nearest hit over the accepted leaf boxes whatever the order
// of the tests.  Traversing past a queued candidate with the not-yet-updated
// best only adds tests that cannot win; the footprint of each test depends
// only on its own box (Arbor.cu:226).  Between exactly equal t values the
// reference keeps the one it meets first; block_apply decides such ties by the
// reference's visiting order (ref_before).  Where rounding puts a hit before
// its box's entry and another hit between the two, the order decides;
// finish_tree notices and repeats that tree in a fixed order.  The DDA advance
// and tree hand-over wait for all results, so they use the reference's best.
#pragma once
#include "orderbatch.cuh"

namespace arbor {

constexpr int kQueue = 12;       // candidates a lane may queue
constexpr int kOrderedChunk = 16;  // tree_in_order's chunk of the single-image passes
constexpr int kSlice = 4;        // passes of an advance between two rounds of tests ...
constexpr int kTreeRun = 8;      // ... of at most this many tree steps each
constexpr int kMarchRun = 8;     // steps of an SDF march per round

// Per-block shared-memory batch; Ordered: tree_in_order's chunk.
template <int Ordered>
struct BlockBatchOf {
  static constexpr int kQ = kQueue;
  static constexpr int kJobs = kThreads * kQueue;
  static constexpr int kOrdered = Ordered;
  static constexpr int kRun = kTreeRun;
  static constexpr bool kWhole = false;
  float4 rayO[kThreads];           // each lane's local ray: origin and wind time
  float4 rayD[kThreads];           // direction and footprint cone
  float4 rayI[kThreads];           // inverse direction and, during the tests, Ray::lbest
  float nearest[kThreads];         // nearest t so far, the entry of its box, and the second nearest candidate's t
  float entry[kThreads], second[kThreads];
  float slack[kThreads];           // primary rays: by how much a hit may precede its box (enter_tree)
  uint32_t sib[kLeafDepth + 1][3][kThreads];  // deferred nodes (tree_pop)
  LeafSolve solve[kSolves];
  float span[kJobs];               // a candidate's box entry distance (queue place k of thread t: k * kThreads + t)
  float res[kJobs];                // its result; below 0: a march in progress at -res
  short slot[kJobs];               // its leaf slot
  short prim[kJobs];               // its record
  short job[kJobs];                // compacted job lists: leaf clips from the front, the rest from the back
  short solveJob[kSolves];
  int count[2][2];                 // leaf clips and others queued, by parity of the round
  uint8_t steps[kJobs];            // steps its march has taken
  int solves, unit;                // Newton solves queued and units of tests taken in this round
  uint8_t rayS[kThreads];          // scene (forest of several species)
  __device__ __forceinline__ int record(const uint32_t*, int q) const { return prim[q]; }
};
using BlockBatch = BlockBatchOf<kOrderedChunk>;

// The footprint a queued candidate is tested at (Arbor.cu:226).
template <class BB>
__device__ __forceinline__ float candidate_footprint(const BB& b, int q) {
  return fmaxf(0.000005f, b.rayD[q % kThreads].w * fmaxf(0.05f, b.span[q]));
}

// The test of this lane's queue place q: the reference's own test of its box
// in Nodes (Arbor.cu:223) against the nearest t at the tree's entry (best0),
// then its record: 1 a leaf clip, 2 another test (wood, stones, unused records),
// 0 none (box not accepted, or an Order entry past the records, not read).
template <int Ordered>
__device__ __forceinline__ int classify_candidate(const TraceCtx& c, const Ray& r, BlockBatchOf<Ordered>& b, int q, f3 o, f3 inv, float best0) {
  const int slot = b.slot[q] & (kCapacity - 1);  // (a leaf's slot always is one; no load leaves Order whatever it holds)
  const float* nodes = scene_nodes(c, r.species);
  const float4 lo = ldg4(nodes, 2 * (kCapacity + slot)), hi = ldg4(nodes, 2 * (kCapacity + slot) + 1);
  const uint32_t uid = __ldg(scene_order(c, r.species) + slot);
  int cls = 0;
  float spanx;
  if (node_accept(lo, hi, o, inv, best0, spanx) && uid < (uint32_t)kCapacity)
    cls = (int)ldg4(scene_P(c, r.species), (int)uid * 6).w == 1 ? 1 : 2;
  b.prim[q] = (short)uid;
  b.span[q] = spanx;
  return cls;
}
// Resolve this lane's queued leaf slots and append their tests to the block's
// job lists.  `open`: the queue was resolved before and only its unfinished
// marches go on.  The warp's lanes call it together.
template <class BB>
__device__ __forceinline__ void block_classify(const TraceCtx& c, const Ray& r, BB& b, int (&count)[2], int nq, bool open) {
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31;
  const unsigned lt = (1u << lane) - 1u;
  const float4 o = b.rayO[tid], inv = b.rayI[tid];
  const float best0 = nq > 0 ? r.best / r.lsc : 0.0f;
  if (nq > 0) {
    b.rayI[tid].w = r.lbest;
    if (c.species) b.rayS[tid] = (uint8_t)r.species;
  }
  const int most = __reduce_max_sync(full, nq);
  for (int k = 0; k < most; k++) {
    const int q = k * kThreads + tid;
    int cls = 0;  // 1: leaf clip, 2: another test
    if (k < nq && open) {
      if (b.res[q] < 0.0f) cls = 2;
    } else if (k < nq) {
      cls = classify_candidate(c, r, b, q, xyz(o), xyz(inv), best0);
      b.res[q] = kFar;
      if (c.refine) b.steps[q] = 0;
    }
    const unsigned ml = __ballot_sync(full, cls == 1), mo = __ballot_sync(full, cls == 2);
    int base_l = 0, base_o = 0;
    if (lane == 0) {
      if (ml) base_l = atomicAdd(&count[0], __popc(ml));
      if (mo) base_o = atomicAdd(&count[1], __popc(mo));
    }
    base_l = __shfl_sync(full, base_l, 0);
    base_o = __shfl_sync(full, base_o, 0);
    if (cls == 1) b.job[base_l + __popc(ml & lt)] = (short)q;
    if (cls == 2) b.job[BB::kJobs - 1 - (base_o + __popc(mo & lt))] = (short)q;
  }
}

// Newton solve of candidate q, whose clip `ls` passed.
template <class BB>
__device__ __forceinline__ void block_solve(const TraceCtx& c, BB& b, int q, const LeafSolve& ls) {
  const int s = c.species ? b.rayS[q % kThreads] : 0;
  b.res[q] = leaf_newton(ls, leaf_shape(scene_P(c, s), b.record(scene_order(c, s), q)), b.res[q], candidate_footprint(b, q));
}

// Run the block's queued tests: n_leaf leaf clips, n_other others.  Warps take
// units of 32 jobs as they come free, the others (a march of up to kMarchRun
// steps, the longest jobs) first; the clips that pass leave a Newton solve,
// and the solves run compacted after a barrier.  Every thread of the block
// calls it; the results are in place after its last barrier.
template <class BB>
__device__ __forceinline__ void block_tests(const TraceCtx& c, BB& b, int n_leaf, int n_other) {
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int other_units = (n_other + 31) >> 5, units = other_units + ((n_leaf + 31) >> 5);
  for (;;) {
    int u = 0;
    if (lane == 0) u = atomicAdd(&b.unit, 1);
    u = __shfl_sync(full, u, 0);
    if (u >= units) break;
    if (u < other_units) {
      const int j = 32 * u + lane;
      if (j < n_other) {
        const int q = b.job[BB::kJobs - 1 - j], owner = q % kThreads, s = c.species ? b.rayS[owner] : 0;
        const float4 o = b.rayO[owner], d = b.rayD[owner];
        int steps = c.refine ? b.steps[q] : 0;
        b.res[q] = other_t(scene_P(c, s), b.record(scene_order(c, s), q), xyz(o), xyz(d), candidate_footprint(b, q), c.refine,
                           b.rayI[owner].w, -b.res[q], steps, n_other + n_leaf <= 64 ? 64 : kMarchRun);
        if (c.refine) b.steps[q] = (uint8_t)steps;
      }
    } else {
      const int j = 32 * (u - other_units) + lane;
      bool solve = false;
      LeafSolve ls;
      int q = 0;
      if (j < n_leaf) {
        q = b.job[j];
        const int owner = q % kThreads, s = c.species ? b.rayS[owner] : 0;
        const float4 o = b.rayO[owner], d = b.rayD[owner];
        float tube;
        solve = leaf_clip(scene_P(c, s), b.record(scene_order(c, s), q), xyz(o), xyz(d), o.w, c.wind, ls, tube);
        // The solve stays inside its clipped interval: one that begins beyond
        // the owner's lbest can neither beat it nor matter to the order.
        solve = solve && !(ls.spanx > b.rayI[owner].w);
        b.res[q] = tube;  // the result, or the Newton stage's starting best
      }
      const unsigned m = __ballot_sync(full, solve);
      int at = 0;
      if (lane == 0 && m) at = atomicAdd(&b.solves, __popc(m));
      at = __shfl_sync(full, at, 0) + __popc(m & lt);
      if (solve && at < kSolves) {
        b.solve[at] = ls;
        b.solveJob[at] = (short)q;
      } else if (solve) {
        b.job[j] = (short)(q | 0x4000);  // no room: clipped again below
      }
    }
  }
  __syncthreads();
  const int queued = b.solves, solves = min(queued, kSolves);
  for (int i = tid; i < solves; i += kThreads) block_solve(c, b, b.solveJob[i], b.solve[i]);
  if (queued > kSolves) {  // uniform; rare: more clips passed than there is room for
    for (int j = tid; j < n_leaf; j += kThreads) {
      if (!(b.job[j] & 0x4000)) continue;
      const int q = b.job[j] & 0x3fff, owner = q % kThreads, s = c.species ? b.rayS[owner] : 0;
      const float4 o = b.rayO[owner], d = b.rayD[owner];
      LeafSolve ls;
      float tube;
      if (leaf_clip_again(scene_P(c, s), b.record(scene_order(c, s), q), xyz(o), xyz(d), o.w, c.wind, ls, tube)) block_solve(c, b, q, ls);
    }
  }
  __syncthreads();
}
static_assert(kThreads * kQueue <= 0x4000 && kThreads * kMaxChunk <= 0x4000, "a queue place fits 14 bits");

// Apply a lane's results.  A nearer hit replaces the best; an exactly equal
// one replaces it when the reference meets it first, so the kept primitive
// does not depend on the order of visits or tests.  The best hit's box entry
// and the second nearest t tell finish_tree whether the order could matter
// after all; for that every candidate up to the entry is still tested.
template <int Ordered>
__device__ __forceinline__ void block_apply(const TraceCtx& c, Ray& r, BlockBatchOf<Ordered>& b, int nq) {
  const int tid = threadIdx.x;
  float best = b.nearest[tid], second = b.second[tid], entry = b.entry[tid];
  for (int k = 0; k < nq; k++) {
    const int q = k * kThreads + tid;
    const float t = b.res[q];
    const int slot = b.slot[q];
    if (t < best ||
        (t == best && r.lfound >= 0 && ref_before(scene_nodes(c, r.species), xyz(b.rayO[tid]), xyz(b.rayI[tid]), slot, r.lfound))) {
      if (r.lfound >= 0) second = best;
      best = t;
      entry = b.span[q];
      r.lfound = slot;
    } else {
      second = fminf(second, t);
    }
  }
  b.nearest[tid] = best;
  b.second[tid] = second;
  b.entry[tid] = entry;
  r.lbest = fmaxf(best, entry) + (c.refine ? b.slack[tid] : 0.0f);
}

// The pixels of a persistent CTA: the 8x4-pixel blocks blockIdx.x,
// blockIdx.x + gridDim.x, blockIdx.x + 2 gridDim.x, ... of a width x height
// image, handed out one pixel at a time, in block order, from a counter in
// shared memory.
struct PixelPool {
  int* next;  // shared-memory counter of pixels handed out by this CTA
  int width, height, blocks_x, blocks;
};

// Collective (all 32 lanes): hand the next pixels to the lanes in `idle`.
// Returns true for a lane that received a pixel inside the image; `past` is
// set for every lane once the CTA's blocks are used up.
__device__ __forceinline__ bool pool_take(const PixelPool& pool, unsigned idle, int lane, int& x, int& y, bool& past) {
  const unsigned full = 0xffffffffu;
  int base = 0;
  if (lane == 0) base = atomicAdd(pool.next, __popc(idle));
  base = __shfl_sync(full, base, 0);
  bool got = false, beyond = false;
  if (idle & (1u << lane)) {
    const int idx = base + __popc(idle & ((1u << lane) - 1u));
    const int block = (int)blockIdx.x + (idx >> 5) * (int)gridDim.x;
    if (block >= pool.blocks) {
      beyond = true;
    } else {
      const int by = block / pool.blocks_x, bx = block - by * pool.blocks_x;
      x = bx * 8 + (idx & 7);
      y = by * 4 + ((idx >> 3) & 3);
      got = x < pool.width && y < pool.height;
    }
  }
  past = __any_sync(full, beyond);
  return got;
}

// The pixels of one image shared by every CTA that works on it: its 8x4
// blocks 0, 1, 2, ... handed out one pixel at a time from a counter in
// global memory (the batched renderer's per-view pools).
struct ViewPool {
  int* next;  // global counter of pixels handed out for this image
  int width, height, blocks_x, blocks;
};

// ViewPool form of pool_take (same contract).
__device__ __forceinline__ bool pool_take(const ViewPool& pool, unsigned idle, int lane, int& x, int& y, bool& past) {
  const unsigned full = 0xffffffffu;
  int base = 0;
  if (lane == 0) base = atomicAdd(pool.next, __popc(idle));
  base = __shfl_sync(full, base, 0);
  bool got = false, beyond = false;
  if (idle & (1u << lane)) {
    const int idx = base + __popc(idle & ((1u << lane) - 1u));
    const int block = idx >> 5;
    if (block >= pool.blocks) {
      beyond = true;
    } else {
      const int by = block / pool.blocks_x, bx = block - by * pool.blocks_x;
      x = bx * 8 + (idx & 7);
      y = by * 4 + ((idx >> 3) & 3);
      got = x < pool.width && y < pool.height;
    }
  }
  past = __any_sync(full, beyond);
  return got;
}

// Drive a block through a pixel pool: lanes whose rays are finished take the
// next pixels (Policy::start begins a ray, or finishes the pixel at once), so
// no lane waits for the slowest ray of a fixed tile.  Policy::done is called
// for a finished ray and either continues it (a new trace on r) or sets it
// idle.  Every thread of the block calls it; it begins and ends with a
// barrier.
template <class BB, class Policy, class Pool>
__device__ __forceinline__ void block_drive(const TraceCtx& c, Ray& r, BB& b, Policy& policy, const Pool& pool) {
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31;
  int nq = 0;
  bool open = false;     // a march of this lane's queue is unfinished: the lane waits
  bool drained = false;  // uniform in the warp
  r.phase = kPhIdle;
  if (tid < 2) b.count[tid][0] = b.count[tid][1] = 0;
  if (tid == 0) b.solves = b.unit = 0;
  __syncthreads();
  for (int round = 0;; round ^= 1) {
    for (int step = 0; step < kSlice; step++) {
      // Refill once Policy::kRefill lanes are idle (or all are).
      const unsigned idle = __ballot_sync(full, r.phase == kPhIdle);
      if (!drained && (__popc(idle) >= Policy::kRefill || idle == full)) {
        int x = 0, y = 0;
        bool past = false;
        const bool got = pool_take(pool, idle, lane, x, y, past);
        drained = past;
        if (got) policy.start(c, r, x, y);
      } else if (__all_sync(full, open || r.phase == kPhBlocked || (r.phase == kPhTreeEnd && nq > 0) || r.phase == kPhIdle)) {
        break;  // every ray waits for its tests
      }
      // Tree steps a few at a time, so that the cells and tree entries between
      // them, as many instructions each, run for more lanes at once.
      for (int k = 0; k < BB::kRun; k++) {
        const bool go = r.phase == kPhTree && !open;
        if (!__any_sync(full, go)) break;
        if (go) tree_step(c, r, b, tid, nq);
      }
      if (r.phase == kPhTreeEnd && nq == 0) finish_tree(c, r, b, tid);
      if (r.phase == kPhDDA) dda_step(c, r, b, tid);
      if (r.phase == kPhDone) policy.done(r);
    }
    // (in a fixed order a chunk is tested whole)
    const int now = BB::kWhole && r.phase == kPhTree ? 0 : nq;
    block_classify(c, r, b, b.count[round], now, open);
    if (!__syncthreads_or(r.phase != kPhIdle || !drained)) break;
    const int n_leaf = b.count[round][0], n_other = b.count[round][1];
    if (tid < 2) b.count[round ^ 1][tid] = 0;
    block_tests(c, b, n_leaf, n_other);
    if (tid == 0) b.solves = b.unit = 0;
    if (now > 0) {
      open = false;
      if (c.refine)
        for (int k = 0; k < now; k++) open |= b.res[k * kThreads + tid] < 0.0f;
      if (!open) {
        block_apply(c, r, b, now);
        nq = 0;
        if (r.phase == kPhBlocked) tree_pop(r, b, tid, nq);
      }
    }
  }
}
// The same in the fixed order of orderbatch.cuh, out of line: its code and
// registers stay away from the other loop's.
template <class BB, class Policy, class Pool>
__device__ __noinline__ void block_drive_in_order(TraceCtx c, BB* b, Policy policy, Pool pool) {
  policy.bind(&c);
  Ray r;
  block_drive(c, r, *b, policy, pool);
}
template <class BB, class Policy, class Pool>
__device__ __forceinline__ void block_run_pool(const TraceCtx& c, Ray& r, BB& b, Policy& policy, const Pool& pool) {
  if (c.tight.T == nullptr) {  // uniform in the block
    using OB = OrderBatchOf<BB::kOrdered>;
    static_assert(sizeof(OB) <= sizeof(BB) && BB::kOrdered <= kMaxChunk, "in the other batch's memory");
    Policy copy = policy;
    copy.bind(nullptr);  // (c itself must not leave the registers)
    block_drive_in_order(c, reinterpret_cast<OB*>(&b), copy, pool);
    return;
  }
  block_drive(c, r, b, policy, pool);
}

}  // namespace arbor
