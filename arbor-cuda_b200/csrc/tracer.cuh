// tracer.cuh - forest ray state machine.
//
// One ray per lane, advanced through the phases of the reference's
// traceForest/traceTree (Arbor.cu:220-251):
//
//   DDA   one forest cell: bounding-sphere test, tree entry, cell advance
//   TREE  one BVH step: test the four grandchildren of a node, descend
//         nearest-first, queue accepted leaves (candidate primitives), or
//         pop a deferred node
//   TREE_END  the tree has no accepted node left (finish_tree folds it in)
//   DONE  the ray's result is final
//
// The cells and the accepted leaves are the reference's; the order of visits
// is not.  The traversal runs over the tight boxes of tight.cuh
// two heap levels at a time: nodes 4g .. 4g + 3, the grandchildren of node g,
// are contiguous, and testing them together halves the chain of dependent
// loads and the loop's passes.  Accepted nodes are visited by the nearer
// midpoint of their span (primary rays) or the nearer entry (shadow segments).
// The result is the nearest hit over the accepted leaf boxes whatever the order
// (blockbatch.cuh gives the argument),
// as long as each hit lies inside its primitive's box; between exactly equal
// hit distances (leaves sharing a petiole base, wood segments sharing a
// joint) the one the reference meets first is kept (ref_before).  Where a hit
// does come before its box, and another one between the two, the answer
// depends on the order: such a tree is noticed and traced again one candidate
// queue at a time in a fixed order (tree_in_order).
#pragma once
#include "tight.cuh"

namespace arbor {

enum RayPhase : int { kPhDDA = 0, kPhTree = 1, kPhDone = 3, kPhIdle = 4, kPhBlocked = 5, kPhTreeEnd = 6 };

// No hit found yet in a tree entered with a nearest t above kFar.  The
// reference divides the world's nearest t by the tree's scale (Arbor.cu:247),
// so for a ray that has met nothing (best = kFar) in a tree smaller than 1 the
// tests' "no hit" value kFar is nearer than best, and the first candidate
// that misses becomes the tree's hit, at kFar, unless a surface is hit.  Here
// such a tree is traversed for real hits alone, and finish_tree looks that
// first candidate up (first_leaf) if there was none.
constexpr int kMissCounts = -2;
// A tree that the batch does not traverse: finish_tree traces it in a fixed
// order (tree_in_order).
constexpr int kInOrder = -3;

constexpr int kThreads = 256;  // threads of a block batch (blockbatch.cuh)
constexpr int kSolves = 256;   // Newton solves a block keeps for compaction

// A lane's ray.  The local ray of the tree being traversed (origin,
// direction, its inverse, wind time, footprint cone) is kept in the block
// batch, where the tests read it; here only what the traversal needs.
struct Ray {
  f3 ro, rd;        // world ray
  float best;       // world-space nearest t so far
  float found;      // primitive id of best (as the reference's float), -1
  int foundTree;    // tree of best, -1
  // forest DDA (Arbor.cu:241-248)
  int ix, iz, sx, sz, step;
  float tx, tz, dx, dz, exit;
  // the tree being traversed
  int tree;
  f3 inv, on, of;   // a box plane at grid coordinate q is met at q * inv - on (near side) or - of (far side)
  uint32_t near;    // per axis a bit: the near plane is the box's hi plane
  int boxes;        // the stored boxes in use: 0 the tight ones, kNodeBoxes those of Nodes
  float lbest, lsc; // lbest prunes the traversal: the nearest t so far, or its box entry where that lies beyond it, plus the slack
  int lfound;       // its leaf slot, -1, kMissCounts or kInOrder
  int group, depth; // nodes 4 group .. 4 group + 3 are tested next; depth 0-7 (nodes at heap level 2 depth + 1)
  uint32_t pending; // deferred nodes per depth, 4 bits each
  int phase;
  int species;      // scene of the tree being traversed (forest of several species; 0 otherwise)
};

struct TraceCtx {
  const float* P;
  const float* Nodes;
  const uint32_t* Order;
  const Instance* inst;   // forest instance table (the world-seed registry's, or shared memory)
  TightView tight;        // the boxes the traversal tests; without them it takes those of Nodes (orderbatch.cuh)
  float cone, time, wind;
  bool refine;            // primary rays: wood refined by the SDF march; false for shadow segments
  bool forest;            // false: the single-tree scene (identity instance)
  bool species = false;   // true: a forest of several species, P / Nodes / Order holding one scene
                          // per species back to back, instance t on scene species_of[t] (or
                          // inst[t].species when species_of is null)
  const uint8_t* species_of = nullptr;
};

// The scene of tree `tree` (0 unless the forest has several species).
__device__ __forceinline__ int tree_species(const TraceCtx& c, int tree) {
  if (!c.species || tree < 0) return 0;
  return c.species_of != nullptr ? (int)c.species_of[tree] : c.inst[tree].species;
}

// The records of scene `s` (s = 0 unless the forest has several species).
__device__ __forceinline__ const float* scene_P(const TraceCtx& c, int s) { return c.species ? c.P + (size_t)s * (kCapacity * kPS) : c.P; }
__device__ __forceinline__ const float* scene_nodes(const TraceCtx& c, int s) {
  return c.species ? c.Nodes + (size_t)s * (kNodeCount * 8) : c.Nodes;
}
__device__ __forceinline__ const uint32_t* scene_tight(const TraceCtx& c, int s) {
  return c.species ? c.tight.T + (size_t)s * kTightWords : c.tight.T;
}
__device__ __forceinline__ const uint32_t* scene_order(const TraceCtx& c, int s) { return c.species ? c.Order + (size_t)s * kCapacity : c.Order; }

// The low (lo plane) or high (hi plane) half of a stored pair as the float
// 2^23 + value, by byte permutation.
constexpr uint32_t kHalfLo = 0x7410u, kHalfHi = 0x7432u;
constexpr float kHalfBias = 8388608.0f;
__device__ __forceinline__ float box_half(uint32_t pair, uint32_t sel) { return __uint_as_float(__byte_perm(pair, 0x4B000000u, sel)); }

// Tree entry with the reference's root test (Arbor.cu:221-223) on the local
// ray (lro, lrd); keeps the local ray in the batch.  Returns true when the
// root is accepted and traversal starts (or, with lfound kInOrder, the tree is
// to be traced in order).
template <class WB>
__device__ __forceinline__ bool enter_tree(const TraceCtx& c, Ray& r, WB& b, int lane, f3 lro, f3 lrd, float lcone, float ltime) {
  r.lfound = -1;
  r.group = 0;  // nodes 2 and 3 (0 and 1 are no children)
  r.depth = 0;
  r.pending = 0u;
  const f3 linv = inv3(lrd);
  const float* nodes = scene_nodes(c, r.species);
  const float4 lo = ldg4(nodes, 2), hi = ldg4(nodes, 3);
  float spanx;
  if (!node_accept(lo, hi, lro, linv, r.lbest, spanx)) return false;
  if (r.lbest > kFar) {
    r.lbest = kFar;
    r.lfound = kMissCounts;
  }
  b.nearest[lane] = r.lbest;
  b.entry[lane] = 0.0f;
  b.second[lane] = kFar;
  // The margin of the box tests: tight.cuh's, plus the rounding of the slab
  // distances as one multiply-add each.
  const f3 far = max3(mk(fabsf(lo.x - lro.x), fabsf(lo.y - lro.y), fabsf(lo.z - lro.z)), mk(fabsf(hi.x - lro.x), fabsf(hi.y - lro.y), fabsf(hi.z - lro.z)));
  const float d = length3(far);
  // (a surface beyond kFar would be a hit after all)
  if (r.lfound == kMissCounts && !(d < 0.99f * kFar)) r.lfound = kInOrder;
  float m = c.tight.rel * d + c.tight.abs;
  float slack = 0.0f;
  r.boxes = 0;
  if (c.refine && m > c.tight.most) {  // (a shadow segment is 36 m at most; its pruning has no slack)
    // The boxes are not widened, but a hit may still come before its box by
    // the margin: pruning allows for it.
    slack = m;
    m = 0.0f;
    r.boxes = kNodeBoxes;
  }
  if (c.refine) {
    b.slack[lane] = slack;
    r.lbest += slack;
  }
  m += 1.0e-6f * (d + fabsf(lro.x) + fabsf(lro.y) + fabsf(lro.z));
  const float* grid = reinterpret_cast<const float*>(scene_tight(c, r.species)) + kTightGrid;
  const f3 step = mk(__ldg(grid + 3), __ldg(grid + 4), __ldg(grid + 5));
  const f3 origin = mk(__ldg(grid), __ldg(grid + 1), __ldg(grid + 2)) - step * kHalfBias;
  m += 4.0f * fmaxf(step.x, fmaxf(step.y, step.z));
  // Nodes without primitives (0 and 1 among them, no one's children) are stored
  // inside out over the whole grid, and a margin of half the grid's widest side
  // turns them right side out: accepted, a walk from nodes 0 or 1 ends at slots
  // before Order's first.  Twice that distance is kept, for the rounding of the
  // planes (the margin holds 1e-6 of the distance, so the side is then above
  // 4e-6 of it and one plane is off by less than 3e-7).  What is smaller beside
  // its margin - a pebble of 9 cm at 45 m, a leaf alone in a storm - is a few
  // pixels or a few primitives.  (Also false where the ray is not finite.)
  const f3 side = xyz(hi) - xyz(lo);
  if (!(fmaxf(side.x, fmaxf(side.y, side.z)) > 4.0f * m)) r.lfound = kInOrder;
  const f3 oa = (lro + mk(m, m, m) - origin) * linv, ob = (lro - mk(m, m, m) - origin) * linv;
  const bool px = linv.x >= 0.0f, py = linv.y >= 0.0f, pz = linv.z >= 0.0f;
  r.inv = step * linv;
  r.on = mk(px ? oa.x : ob.x, py ? oa.y : ob.y, pz ? oa.z : ob.z);
  r.of = mk(px ? ob.x : oa.x, py ? ob.y : oa.y, pz ? ob.z : oa.z);
  r.near = (px ? 0u : 1u) | (py ? 0u : 2u) | (pz ? 0u : 4u);
  b.rayO[lane] = make_float4(lro.x, lro.y, lro.z, ltime);
  b.rayD[lane] = make_float4(lrd.x, lrd.y, lrd.z, lcone);
  b.rayI[lane] = make_float4(linv.x, linv.y, linv.z, 0.0f);  // .w: block_classify
  return true;
}

// After a cell's tree: next crossing, exit test, advance (Arbor.cu:248).
__device__ __forceinline__ void dda_advance(Ray& r) {
  float next = r.tx < r.tz ? r.tx : r.tz;
  if (next > r.exit || next > r.best) {
    r.phase = kPhDone;
    return;
  }
  if (r.tx < r.tz) {
    r.ix += r.sx;
    r.tx += r.dx;
  } else {
    r.iz += r.sz;
    r.tz += r.dz;
  }
  r.step++;
  r.phase = kPhDDA;
}

// The first leaf slot the reference's traversal of this tree tests for the
// local ray (ro, inv) when nothing prunes (Arbor.cu:224-227: depth first, the
// child with the smaller entry first), or -1.  The root is accepted.
static __device__ __noinline__ int first_leaf(const float* __restrict__ Nodes, f3 ro, f3 inv) {
  int node = 1, depth = 0;
  uint32_t pending = 0u;
  for (;;) {
    if (node >= kCapacity) return node - kCapacity;
    const int left = node * 2;
    float lx, rx;
    const bool lh = node_accept(ldg4(Nodes, 2 * left), ldg4(Nodes, 2 * left + 1), ro, inv, 2.0f * kFar, lx);
    const bool rh = node_accept(ldg4(Nodes, 2 * left + 2), ldg4(Nodes, 2 * left + 3), ro, inv, 2.0f * kFar, rx);
    if (lh || rh) {
      depth++;
      if (lh && rh) pending |= 1u << depth;
      node = lh && (!rh || lx < rx) ? left : left + 1;
      continue;
    }
    if (pending == 0u) return -1;
    const int level = 31 - __clz(pending);
    pending &= ~(1u << level);
    node = (node >> (depth - level)) ^ 1;
    depth = level;
  }
}

// True when leaf slot a comes before leaf slot b in the reference's visiting
// order of this tree (Arbor.cu:224-225): a depth-first order in which, at
// every node, the child with the smaller entry span.x goes first (the left
// one only when its entry is strictly smaller).  The two leaves part at their
// lowest common ancestor, so the order is that node's decision, made again
// here on the same values (ro, inv: the tree-local ray).  Ties are rare; the
// function stays out of line, away from the traversal's instruction stream.
static __device__ __noinline__ bool ref_before(const float* __restrict__ Nodes, f3 ro, f3 inv, int a, int b) {
  int na = a + kCapacity, nb = b + kCapacity;
  while ((na >> 1) != (nb >> 1)) {
    na >>= 1;
    nb >>= 1;
  }
  const int left = na & ~1;
  const float4 llo = ldg4(Nodes, 2 * left), lhi = ldg4(Nodes, 2 * left + 1);
  const float4 rlo = ldg4(Nodes, 2 * left + 2), rhi = ldg4(Nodes, 2 * left + 3);
  const float lx = box_span_inv(ro, inv, xyz(llo), xyz(lhi)).x;
  const float rx = box_span_inv(ro, inv, xyz(rlo), xyz(rhi)).x;
  return (na == left) == (lx < rx);
}

// One tree for one ray in a fixed order: the boxes of Nodes, one child at a
// time (primary rays by the nearer midpoint of the span, shadow segments by
// the nearer entry), candidates tested `chunk` at a time, a box pruned when its
// entry is not below the nearest t of the chunks before.  For the rays whose
// answer depends on the order (finish_tree); rare, and out of line.
struct TreeResult {
  float t;
  int slot;  // -1: no hit
};
constexpr int kMaxChunk = 16;
static __device__ __noinline__ TreeResult tree_in_order(const float* __restrict__ P, const float* __restrict__ Nodes,
                                                        const uint32_t* __restrict__ Order, float4 o, float4 d, f3 inv, float wind, float best,
                                                        bool refine, int chunk) {
  const f3 ro = xyz(o), rd = xyz(d);
  float sib[16], span[kMaxChunk];
  int queue[kMaxChunk];
  int node = 1, depth = 0, nq = 0, found = -1;
  uint32_t pending = 0u;
  float spanx;
  bool more = node_accept(ldg4(Nodes, 2), ldg4(Nodes, 3), ro, inv, best, spanx);
  while (more || nq > 0) {
    bool pop = false;
    if (more && node < kCapacity) {
      const int left = node * 2;
      f2 ls, rs;
      const bool lh = node_accept_span(ldg4(Nodes, 2 * left), ldg4(Nodes, 2 * left + 1), ro, inv, best, ls);
      const bool rh = node_accept_span(ldg4(Nodes, 2 * left + 2), ldg4(Nodes, 2 * left + 3), ro, inv, best, rs);
      if (lh || rh) {
        depth++;
        bool l = lh;
        if (lh && rh) {
          l = refine ? fmaxf(ls.x, 0.0f) + ls.y < fmaxf(rs.x, 0.0f) + rs.y : ls.x < rs.x;
          pending |= 1u << depth;
          sib[depth] = l ? rs.x : ls.x;
        }
        node = l ? left : left + 1;
        spanx = l ? ls.x : rs.x;
        continue;
      }
      pop = true;
    } else if (more) {
      queue[nq] = node - kCapacity;
      span[nq++] = spanx;
      pop = nq < chunk;
    }
    if (!pop) {  // the chunk is full, or the tree is finished
      for (int k = 0; k < nq; k++) {
        const uint32_t uid = __ldg(Order + queue[k]);
        const float t = uid < (uint32_t)kCapacity
                            ? object_t(P, (int)uid, ro, rd, fmaxf(0.000005f, d.w * fmaxf(0.05f, span[k])), o.w, wind, refine)
                            : kFar;
        if (t < best || (refine && t == best && found >= 0 && ref_before(Nodes, ro, inv, queue[k], found))) {
          best = t;
          found = queue[k];
        }
      }
      nq = 0;
    }
    if (!more) break;
    more = false;
    while (pending != 0u) {
      const int level = 31 - __clz(pending);
      pending &= ~(1u << level);
      node = (node >> (depth - level)) ^ 1;
      depth = level;
      spanx = sib[level];
      if (spanx < best) {
        more = true;
        break;
      }
    }
  }
  return {best, found};
}

// The tree is exhausted: fold its local result into the world result
// (Arbor.cu:247 for the forest; traceTree's return for the single tree).
__device__ __forceinline__ void fold_tree(const TraceCtx& c, Ray& r) {
  const float found = r.lfound >= 0 ? (float)__ldg(scene_order(c, r.species) + r.lfound) : -1.0f;
  if (!c.forest) {
    r.best = r.lbest;
    r.found = found;
    r.phase = kPhDone;
    return;
  }
  if (r.lfound >= 0 && r.lbest * r.lsc < r.best) {
    r.best = r.lbest * r.lsc;
    r.found = found;
    r.foundTree = r.tree;
  }
  dda_advance(r);
}
template <class WB>
__device__ __forceinline__ void finish_tree(const TraceCtx& c, Ray& r, WB& b, int lane) {
  if (r.lfound == kMissCounts) {
    r.lfound = first_leaf(scene_nodes(c, r.species), xyz(b.rayO[lane]), xyz(b.rayI[lane]));
    r.lbest = r.lfound >= 0 ? kFar : r.best / r.lsc;
  } else {
    r.lbest = b.nearest[lane];  // (in place of the traversal's, which holds the slack)
    // The hit comes before its own box, and another one before that box too:
    // which of them a traversal keeps depends on its order.
    if (r.lfound == kInOrder || (r.lfound >= 0 && b.entry[lane] > r.lbest && b.second[lane] <= b.entry[lane])) {
      const TreeResult h = tree_in_order(scene_P(c, r.species), scene_nodes(c, r.species), scene_order(c, r.species), b.rayO[lane], b.rayD[lane],
                                         xyz(b.rayI[lane]), c.wind, r.best / r.lsc, c.refine, WB::kOrdered);
      r.lbest = h.t;
      r.lfound = h.slot;
    }
  }
  fold_tree(c, r);
}

// Begin a trace of (ro, rd) with initial nearest `best` (Arbor.cu:236-244).
// The single tree is entered by the ray's one "cell" (dda_step).
__device__ __forceinline__ void ray_begin(const TraceCtx& c, Ray& r, f3 ro, f3 rd, float best) {
  r.ro = ro;
  r.rd = rd;
  r.best = best;
  r.found = -1.0f;
  r.foundTree = -1;
  r.tree = -1;
  r.species = 0;
  if (!c.forest) {
    r.phase = kPhDDA;
    return;
  }
  const float half = (float)kSide * kSpacing * 0.5f;
  f2 worldSpan = box_span(ro, rd, mk(-half, -1.2f, -half), mk(half, 13.5f, half));
  float enter = fmaxf(0.0f, worldSpan.x);
  r.exit = fminf(best, worldSpan.y);
  if (r.exit < enter) {
    r.phase = kPhDone;
    return;
  }
  f3 pos = ro + rd * (enter + 0.0002f);
  r.ix = (int)floorf(pos.x / kSpacing + (float)kSide * 0.5f + 0.5f);
  r.iz = (int)floorf(pos.z / kSpacing + (float)kSide * 0.5f + 0.5f);
  r.sx = rd.x >= 0.0f ? 1 : -1;
  r.sz = rd.z >= 0.0f ? 1 : -1;
  float invx = inv_safe(rd.x);
  float invz = inv_safe(rd.z);
  float bx = ((float)(r.ix - kSide / 2) + (r.sx > 0 ? 0.5f : -0.5f)) * kSpacing;
  float bz = ((float)(r.iz - kSide / 2) + (r.sz > 0 ? 0.5f : -0.5f)) * kSpacing;
  r.tx = (bx - ro.x) * invx;
  r.tz = (bz - ro.z) * invz;
  r.dx = kSpacing * fabsf(invx);
  r.dz = kSpacing * fabsf(invz);
  r.step = 0;
  r.phase = kPhDDA;
}

// Forest cells (Arbor.cu:245-248) up to the next tree whose bounding sphere
// the ray meets: true, with the ray in that tree's frame.  The single tree is
// entered by the ray's one "cell".
struct LocalRay {
  f3 ro, rd;
  float cone, time;
};
__device__ __forceinline__ bool dda_next(const TraceCtx& c, Ray& r, LocalRay& l) {
  if (!c.forest) {
    r.lbest = r.best;
    r.lsc = 1.0f;
    l = {r.ro, r.rd, c.cone, c.time};
    return true;
  }
  int tree = -1;
  while (r.phase == kPhDDA) {
    if (r.step >= 48 || r.ix < 0 || r.iz < 0 || r.ix >= kSide || r.iz >= kSide) {
      r.phase = kPhDone;
      return false;
    }
    tree = r.iz * kSide + r.ix;
    ARBOR_COUNT(kEvCell);
    const Instance& it = c.inst[tree];
    if (sphere_t(r.ro, r.rd, mk(it.px + 0.0f, 0.0f + it.cy, it.pz + 0.0f), it.rad) < r.best) break;
    dda_advance(r);
  }
  if (r.phase != kPhDDA) return false;
  ARBOR_COUNT(kEvTree);
  const Instance& it = c.inst[tree];
  r.tree = tree;
  r.lbest = r.best / it.sc;
  r.lsc = it.sc;
  if (c.species) r.species = tree_species(c, tree);
  l = {to_local_point(r.ro, it), to_local_dir(r.rd, it), c.cone / it.sc, c.time + it.phase};
  return true;
}
template <class WB>
__device__ __forceinline__ void dda_step(const TraceCtx& c, Ray& r, WB& b, int lane) {
  LocalRay l;
  if (!dda_next(c, r, l)) return;
  if (enter_tree(c, r, b, lane, l.ro, l.rd, l.cone, l.time))
    r.phase = r.lfound == kInOrder ? kPhTreeEnd : kPhTree;
  else
    fold_tree(c, r);  // root rejected: traceTree returns (best, -1)
}
// Deferred nodes of one lane: per depth the nodes of the path's group after
// the first in the order of their visits (visit_key), each as its entry distance
// (rounded down to 30 bits) with its place in the group in the low two bits; rejected
// ones last.  Ray::pending holds four bits per depth: how many are left and,
// above, the next one's index (0 when none is left).  The group itself follows from the current one: the path's
// group at a smaller depth is the current group without the lower levels' bits.
constexpr int kLeafDepth = 7;

// The order of visits among a group's accepted nodes: primary rays by the
// midpoint of the span in front of the origin, which finds near hits sooner
// than the entry does (1080p trace 7.5 -> 6.9 ms), shadow segments by the
// entry.  The node's place in the low two bits.
__device__ __forceinline__ uint32_t visit_key(bool refine, float tn, float tf, int k) {
  return (__float_as_uint(refine ? tn + tf : tn) & ~3u) | (uint32_t)k;
}

// Two sort keys in order.
__device__ __forceinline__ void order2(uint32_t& a, uint32_t& b) {
  const uint32_t lo = min(a, b);
  b = max(a, b);
  a = lo;
}

// Pops deferred nodes until one is an inner node to go on with, the queue is
// full or none is left; leaves popped on the way are queued.  A deferred node
// passed its box test; of that test only entry < best depends on the ray's
// later state, so a pop repeats just that comparison.
template <class WB>
__device__ __forceinline__ void tree_pop(Ray& r, WB& b, int lane, int& nq) {
  for (;;) {
    if (r.pending == 0u) {
      r.phase = kPhTreeEnd;  // the tree's queued tests must come back first
      return;
    }
    const int depth = (31 - __clz(r.pending)) >> 2;
    const uint32_t here = r.pending >> (4 * depth);
    const uint32_t e = b.sib[depth][(here >> 2) - 1][lane];
    // one fewer left, the next index; none left: no bits
    r.pending = (here & 3u) > 1u ? r.pending + (3u << (4 * depth)) : r.pending & ~(15u << (4 * depth));
    r.group >>= 2 * (r.depth - depth);
    r.depth = depth;
    if (__uint_as_float(e & ~3u) < r.lbest) {
      const int node = 4 * r.group + (int)(e & 3u);
      if (depth < kLeafDepth) {
        r.group = node;
        r.depth = depth + 1;
        r.phase = kPhTree;
        return;
      }
      b.slot[nq++ * kThreads + lane] = (short)(node - kCapacity);
      if (nq == WB::kQ) {
        r.phase = kPhBlocked;  // resume with the pop once results are in
        return;
      }
    }
  }
}

// One step of a tree (Arbor.cu:224-227): tests the four nodes of the current
// group.  Inner nodes: descends to the nearest accepted one, the others
// deferred.  Leaves: queued as candidates (their slot) when all of them fit,
// else deferred.  With no inner node to go on with it pops a deferred one.
template <class WB>
__device__ __forceinline__ void tree_step(const TraceCtx& c, Ray& r, WB& b, int lane, int& nq) {
  const int node = 4 * r.group;
  float tn[4];       // entries
  uint32_t key[4];   // sort keys, 0xffffffff: rejected
  const uint4* boxes = reinterpret_cast<const uint4*>(scene_tight(c, r.species) + r.boxes) + 3 * r.group;
  const uint4 w0 = __ldg(boxes), w1 = __ldg(boxes + 1), w2 = __ldg(boxes + 2);
  const uint32_t w[12] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, w2.x, w2.y, w2.z, w2.w};
  const uint32_t nx = r.near & 1u ? kHalfHi : kHalfLo, ny = r.near & 2u ? kHalfHi : kHalfLo, nz = r.near & 4u ? kHalfHi : kHalfLo;
  const uint32_t fx = nx ^ (kHalfLo ^ kHalfHi), fy = ny ^ (kHalfLo ^ kHalfHi), fz = nz ^ (kHalfLo ^ kHalfHi);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float ax = __fmaf_rn(box_half(w[3 * k], nx), r.inv.x, -r.on.x), ay = __fmaf_rn(box_half(w[3 * k + 1], ny), r.inv.y, -r.on.y),
                az = __fmaf_rn(box_half(w[3 * k + 2], nz), r.inv.z, -r.on.z);
    const float bx = __fmaf_rn(box_half(w[3 * k], fx), r.inv.x, -r.of.x), by = __fmaf_rn(box_half(w[3 * k + 1], fy), r.inv.y, -r.of.y),
                bz = __fmaf_rn(box_half(w[3 * k + 2], fz), r.inv.z, -r.of.z);
    const float tf = fminf(bx, fminf(by, bz));
    tn[k] = fmaxf(fmaxf(ax, ay), fmaxf(az, 0.0001f));
    key[k] = tn[k] <= fminf(tf, r.lbest) ? visit_key(c.refine, tn[k], tf, k) : 0xffffffffu;
  }
  order2(key[0], key[1]);
  order2(key[2], key[3]);
  order2(key[0], key[2]);
  order2(key[1], key[3]);
  order2(key[1], key[2]);
  const int count = (key[0] != 0xffffffffu) + (key[1] != 0xffffffffu) + (key[2] != 0xffffffffu) + (key[3] != 0xffffffffu);
  const bool leaves = r.depth == kLeafDepth;
  // Taken now: the nearest inner node; of leaves all, or one when the queue has
  // no room for all of them.  (At most three are left for the two-bit count.)
  const int first = min(count, leaves && nq + count <= WB::kQ ? 4 : 1);
  if (leaves) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k < first) b.slot[(nq + k) * kThreads + lane] = (short)(node + (int)(key[k] & 3u) - kCapacity);
    nq += first;
  }
  if (count > first) {
#pragma unroll
    for (int k = 1; k < 4; k++) {
      const uint32_t w = key[k] & 3u;
      const float e = w < 2u ? (w == 0u ? tn[0] : tn[1]) : (w == 2u ? tn[2] : tn[3]);
      b.sib[r.depth][k - 1][lane] = c.refine ? (__float_as_uint(e) & ~3u) | w : key[k];
    }
    r.pending |= (uint32_t)((count - first) | (first << 2)) << (4 * r.depth);
  }
  if (!leaves && count > 0) {
    r.group = node + (int)(key[0] & 3u);
    r.depth++;
    return;
  }
  if (nq == WB::kQ) {
    r.phase = kPhBlocked;
    return;
  }
  tree_pop(r, b, lane, nq);
}

}  // namespace arbor
