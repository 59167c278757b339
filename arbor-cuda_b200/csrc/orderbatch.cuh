// orderbatch.cuh - the block batch (blockbatch.cuh) over the boxes of Nodes in a
// fixed order.
//
// What a scene shows whose Nodes are not what buildBounds makes of P and Order
// (a refitted, padded or emptied box) depends on the order of its traversal,
// and its tight boxes say nothing.  Its rays keep the order of tree_in_order:
// one child at a time, primary rays by the nearer midpoint of the span in front
// of the origin, shadow segments by the nearer entry; candidates in chunks of
// kQ, a box pruned when its entry is not below the nearest t of the chunks
// before.  The lanes of a CTA go through it together and their candidates are
// tested as block_tests runs them, so only the order differs from the other
// pass.  Bound like that one, by the chain of a lane's steps, of two boxes here.
// 960x540 with sun, a box of Nodes moved: 5.3 ms (a lane at a time, each with its
// own tests, 27.5; a warp at a time 6.6); 1920x1080 without, 4.3 (19.8, 6.5).
//
// Ray's fields here: group is the node, inv the inverse direction, on the
// origin, of.x the node's entry.
#pragma once
#include "tracer.cuh"

namespace arbor {

template <int Chunk>
struct OrderBatchOf {
  static constexpr int kQ = Chunk;
  static constexpr int kJobs = kThreads * Chunk;
  static constexpr int kRun = 16;  // tree steps of a pass: twice the other batch's, of half the boxes each
  static constexpr bool kWhole = true;  // a lane's candidates are tested when its queue is full or its tree finished, not before
  float4 rayO[kThreads], rayD[kThreads], rayI[kThreads];  // as BlockBatchOf's
  float sib[15][kThreads];  // deferred siblings' entries, heap levels 1-15
  LeafSolve solve[kSolves];
  float span[kJobs], res[kJobs];
  short slot[kJobs], job[kJobs];
  short solveJob[kSolves];
  int count[2][2];
  uint8_t steps[kJobs];
  int solves, unit;
  uint8_t rayS[kThreads];
  // Record of candidate q, whose scene's Order is `order`.  (There is no room
  // to keep it: two CTAs of the other batch fill an SM.)
  __device__ __forceinline__ int record(const uint32_t* order, int q) const { return (int)__ldg(order + slot[q]); }
};

template <int Q>
__device__ __forceinline__ void order_queue(Ray& r, OrderBatchOf<Q>& b, int lane, int& nq) {
  const int q = nq++ * kThreads + lane;
  b.slot[q] = (short)(r.group - kCapacity);
  b.span[q] = r.of.x;
}
// Pops deferred siblings, deepest first, until one is an inner node to go on
// with, the queue is full or none is left.
template <int Q>
__device__ __forceinline__ void tree_pop(Ray& r, OrderBatchOf<Q>& b, int lane, int& nq) {
  while (r.pending != 0u) {
    const int level = 31 - __clz(r.pending);
    r.pending &= ~(1u << level);
    r.group = (r.group >> (r.depth - level)) ^ 1;
    r.depth = level;
    r.of.x = b.sib[level - 1][lane];
    if (!(r.of.x < r.lbest)) continue;
    if (r.group < kCapacity) {
      r.phase = kPhTree;
      return;
    }
    order_queue(r, b, lane, nq);
    if (nq == Q) {
      r.phase = kPhBlocked;
      return;
    }
  }
  r.phase = kPhTreeEnd;
}
template <int Q>
__device__ __forceinline__ void tree_step(const TraceCtx& c, Ray& r, OrderBatchOf<Q>& b, int lane, int& nq) {
  const float* nodes = scene_nodes(c, r.species);
  const int left = r.group * 2;
  f2 ls, rs;
  const bool lh = node_accept_span(ldg4(nodes, 2 * left), ldg4(nodes, 2 * left + 1), r.on, r.inv, r.lbest, ls);
  const bool rh = node_accept_span(ldg4(nodes, 2 * left + 2), ldg4(nodes, 2 * left + 3), r.on, r.inv, r.lbest, rs);
  if (lh || rh) {
    r.depth++;
    bool l = lh;
    if (lh && rh) {
      l = c.refine ? fmaxf(ls.x, 0.0f) + ls.y < fmaxf(rs.x, 0.0f) + rs.y : ls.x < rs.x;
      r.pending |= 1u << r.depth;
      b.sib[r.depth - 1][lane] = l ? rs.x : ls.x;
    }
    r.group = l ? left : left + 1;
    r.of.x = l ? ls.x : rs.x;
    if (r.group < kCapacity) return;
    order_queue(r, b, lane, nq);
    if (nq == Q) {
      r.phase = kPhBlocked;
      return;
    }
  }
  tree_pop(r, b, lane, nq);
}
template <int Q>
__device__ __forceinline__ void dda_step(const TraceCtx& c, Ray& r, OrderBatchOf<Q>& b, int lane) {
  LocalRay l;
  if (!dda_next(c, r, l)) return;
  r.lfound = -1;
  r.group = 1;
  r.depth = 0;
  r.pending = 0u;
  r.inv = inv3(l.rd);
  r.on = l.ro;
  const float* nodes = scene_nodes(c, r.species);
  if (!node_accept(ldg4(nodes, 2), ldg4(nodes, 3), r.on, r.inv, r.lbest, r.of.x)) {
    fold_tree(c, r);
    return;
  }
  b.rayO[lane] = make_float4(l.ro.x, l.ro.y, l.ro.z, l.time);
  b.rayD[lane] = make_float4(l.rd.x, l.rd.y, l.rd.z, l.cone);
  r.phase = kPhTree;
}
template <int Q>
__device__ __forceinline__ void finish_tree(const TraceCtx& c, Ray& r, OrderBatchOf<Q>&, int) {
  fold_tree(c, r);
}

// The test of this lane's queue place q (queued leaves passed their box): 1 a
// leaf clip, 2 another, 0 none (an Order entry past the records, not read).
template <int Q>
__device__ __forceinline__ int classify_candidate(const TraceCtx& c, const Ray& r, OrderBatchOf<Q>& b, int q, f3, f3, float) {
  const uint32_t uid = __ldg(scene_order(c, r.species) + b.slot[q]);
  if (uid >= (uint32_t)kCapacity) return 0;
  return (int)ldg4(scene_P(c, r.species), (int)uid * 6).w == 1 ? 1 : 2;
}
// Applies a lane's results in the order of its queue.  Of equal hits a primary
// ray keeps the one the reference meets first (ref_before), a shadow segment
// the first.
template <int Q>
__device__ __forceinline__ void block_apply(const TraceCtx& c, Ray& r, OrderBatchOf<Q>& b, int nq) {
  for (int k = 0; k < nq; k++) {
    const int q = k * kThreads + (int)threadIdx.x;
    const float t = b.res[q];
    const int slot = b.slot[q];
    if (t < r.lbest || (c.refine && t == r.lbest && r.lfound >= 0 && ref_before(scene_nodes(c, r.species), r.on, r.inv, slot, r.lfound))) {
      r.lbest = t;
      r.lfound = slot;
    }
  }
}

}  // namespace arbor
