// tight.cuh - tight bounds over the reference's heap BVH, for the batched
// traversal.
//
// A leaf record's bounding box in Nodes (boundLow/boundHigh, Arbor.cu:132-133)
// is the cube of the leaf's whole reach around its stem base.  The leaf itself
// (blade box and petiole) fills a small part of it: on the 1080p forest walk a
// shadow segment tests 547 boxes and 61 leaves to find 5.5 blade boxes.  The
// trace and shade passes therefore traverse a second set of boxes over the
// same heap: leaf records bounded by their oriented blade box, inner nodes by
// the union of their children, everything else as in Nodes.  The boxes are
// made from P, Order and Nodes by one small kernel in front of each pass (64
// CTAs per scene, about 7 MB of traffic) and kept nowhere.
//
// Why no result changes.  A primitive counts only when the ray passes its box
// in Nodes, and that test is still made, exactly, on every candidate
// (classify_candidate).  The tight boxes only drop candidates whose test returns no
// hit.  To be sure of that the traversal widens every tight box by a margin m
// that covers what the FP32 tests can report off the true surface:
//  - the sphere and cone quadratics cancel: their discriminant is off by at
//    most 25 u D^2 (u = 2^-24, D the largest distance from the ray's origin
//    to the tree's box), so a ray that passes a surface within sqrt(25 u) D =
//    1.22e-3 D may be reported to hit it, at a t off by as much.  kTightRel =
//    1.3e-3.
//  - wind turns a leaf about its blade's cross axis by at most 0.155 wind
//    radians (load_leaf), which moves a point of it by at most that times its
//    distance from the stem base (`reach`).
// Pruning is by the widened box's entry, which no reported t can precede.
//
// The margin grows with the distance and the boxes' own size does not: from
// about 80 m on a widened tight box of a grown tree is larger than the box in
// Nodes, whose test needs no margin.  So the boxes of Nodes are stored too, the
// same way, and a primary ray takes, tree by tree, the tight ones up to a margin
// of kTightMost times the largest leaf's reach (0.29 m in a grown scene: 0.10 m)
// and those of Nodes beyond (1080p trace 6.4 -> 5.4 ms, 5.7 with the line at
// 0.05 m and 5.6 at 0.20; small frames that look along the canopy were up to 1.7
// times slower with tight boxes at every distance; a forest of trees a tenth as
// large 2.6 times slower with the line at 0.10 m whatever the leaves).
//
// The boxes are stored 16 bits a coordinate, on a grid over the root's box and
// rounded outward: the four nodes 4g .. 4g + 3 that a traversal step tests
// together are 48 bytes (128 in Nodes), three 16-byte loads a lane.  The loads
// of a step are scattered, one line a lane, and what bounds them is the number
// of load instructions times lanes; the smaller set also stays in what the
// passes leave of L1 (28 KB).
//
// The boxes are used only where Nodes is what buildBounds makes of P and
// Order (every leaf box equal to the record's, every inner node the union of
// its children) and every record's surface lies inside its box
// (tighten_record).  What any other scene shows depends on the order of the
// traversal; it is traversed in a fixed one (orderbatch.cuh).
#pragma once
#include "arbor_scene.cuh"

namespace arbor {

constexpr int kTightParts = 64;                          // CTAs per scene; part k owns the subtree of node 64 + k
constexpr int kTightLeaves = kCapacity / kTightParts;    // 512 leaves each; nodes above the parts keep their box
constexpr int kNodeBoxes = kNodeCount * 3;               // the boxes of Nodes on the same grid, after the tight ones' 3 words each
constexpr int kTightReach = 2 * kNodeBoxes;              // then per part its reach (-1: use Nodes)
constexpr int kTightGrid = kTightReach + kTightParts;    // the grid's origin and step (x, y, z each)
constexpr int kTightWords = kTightGrid + 8;              // words per scene
constexpr size_t kTightBytes = sizeof(uint32_t) * kTightWords;
static_assert(kTightWords % 4 == 0, "16-byte aligned groups in every scene");
constexpr float kTightRel = 1.3e-3f;
constexpr float kTightMost = 0.345f;  // the widest margin at which the tight boxes are the smaller ones, in reaches
constexpr float kTightTaper = 0.25f;  // steepest taper the margin covers (wood the library grows: 0.143, its petioles: 0.02)
constexpr float kSwing = 0.156f;  // wind's largest turn per unit (0.11 + 0.045 radians, rounded up)

struct TightPart {
  float4 lo[kTightLeaves], hi[kTightLeaves];
};

// Leaf record of one Order slot (Arbor.cu:141): {boundLow, active, boundHigh,
// id}.  An id outside the 32768 records (invalid input) is given the bounds
// of an unused record instead of reading out of bounds.
__device__ __forceinline__ void leaf_record(const float* P, uint32_t uid, float4& lo4, float4& hi4) {
  if (uid >= (uint32_t)kCapacity) {
    lo4 = make_float4(kFar, kFar, kFar, 0.0f);
    hi4 = make_float4(-kFar, -kFar, -kFar, (float)(int)uid);
    return;
  }
  int id = (int)uid;
  float4 r0 = ldg4(P, id * 6), r1 = ldg4(P, id * 6 + 1), r2 = ldg4(P, id * 6 + 2), r4 = ldg4(P, id * 6 + 4);
  f3 lo, hi;
  prim_bounds(r0, r1, r1.w, r2.w, r4.x, lo, hi);
  lo4 = make_float4(lo.x, lo.y, lo.z, r0.w >= 0.0f ? 1.0f : 0.0f);
  hi4 = make_float4(hi.x, hi.y, hi.z, (float)id);
}
// Parent = union of the two children (Arbor.cu:142).
__device__ __forceinline__ void merge(float4 alo, float4 ahi, float4 clo, float4 chi, float4& plo, float4& phi) {
  plo = make_float4(fminf(alo.x, clo.x), fminf(alo.y, clo.y), fminf(alo.z, clo.z), alo.w + clo.w);
  phi = make_float4(fmaxf(ahi.x, chi.x), fmaxf(ahi.y, chi.y), fmaxf(ahi.z, chi.z), -1.0f);
}
__device__ __forceinline__ bool same_box(float4 alo, float4 ahi, float4 blo, float4 bhi) {
  return alo.x == blo.x && alo.y == blo.y && alo.z == blo.z && alo.w == blo.w && ahi.x == bhi.x && ahi.y == bhi.y && ahi.z == bhi.z;
}

// Interval [a, b] times component c of an axis.
__device__ __forceinline__ void add_axis(float c, float a, float b, float& lo, float& hi) {
  lo += fminf(a * c, b * c);
  hi += fmaxf(a * c, b * c);
}
// Shrinks the box (lo, hi) in Nodes of a used record `id`, a leaf's to its
// blade and petiole in still air, and returns the leaf's reach (0: not a leaf).
// -1: the surface is not known to lie inside the box - a leaf wider than it is
// long or curled up beyond its cube, a frame that is not orthonormal, a size
// that is negative or not finite, an unknown type, a taper so steep that the
// cone's test goes wrong by more than the margin (its radius and the root's
// terms grow with the taper times the distance).  A ray can then pass the box
// in one place and meet the surface in another, and which hit counts depends on
// the order: the scene is traversed in the fixed one.
__device__ __forceinline__ float tighten_record(const float* P, int id, float4& lo, float4& hi) {
  const float4 r0 = ldg4(P, id * 6), r1 = ldg4(P, id * 6 + 1), r2 = ldg4(P, id * 6 + 2), r3 = ldg4(P, id * 6 + 3), r4 = ldg4(P, id * 6 + 4);
  const int type = (int)r0.w;
  if (!(lo.x <= hi.x && lo.y <= hi.y && lo.z <= hi.z)) return -1.0f;
  if (type == 0) {
    const f3 ab = xyz(r1) - xyz(r0);
    return r1.w >= 0.0f && r2.w >= 0.0f && fabsf(r2.w - r1.w) <= kTightTaper * length3(ab) ? 0.0f : -1.0f;
  }
  if (type != 1) return type == 2 ? 0.0f : -1.0f;
  const f3 o = xyz(r0), u = xyz(r1), v = xyz(r2), n = xyz(r3);
  const float len = r1.w, width = r2.w, stem = r4.x;
  const float g = fmaxf(fmaxf(fabsf(dot3(u, u) - 1.0f), fmaxf(fabsf(dot3(v, v) - 1.0f), fabsf(dot3(n, n) - 1.0f))),
                        fmaxf(fabsf(dot3(u, v)), fmaxf(fabsf(dot3(u, n)), fabsf(dot3(v, n)))));
  const float x1 = stem + len + 0.002f, w = fmaxf(width, 0.002f) + 0.0005f;
  const float reach = sqrtf(x1 * x1 + w * w + 0.0045f);  // 0.067^2 across
  if (!(g < 1.0e-4f) || !(len >= 0.0f) || !(stem >= 0.0f) || !(width >= 0.0f) || !(reach < 1.0e3f)) return -1.0f;
  if (stem > 0.0f && 0.00045f > kTightTaper * stem) return -1.0f;  // (without a stem the petiole is two balls)
  // Across the blade its height (leaf_height for 0 <= q <= 1, |v| <= width: curl,
  // twist, 9 mm of cupping, the 1.2 mm rib, the solve's tolerance) within the
  // clip box's -0.035 .. 0.065, and the petiole's radius.
  const float height = fabsf(r4.y) + 0.62f * fabsf(r4.z) * w + 0.011f;
  const float z0 = -fminf(height, 0.037f), z1 = fminf(height, 0.067f);
  const float oc[3] = {o.x, o.y, o.z}, uc[3] = {u.x, u.y, u.z}, vc[3] = {v.x, v.y, v.z}, nc[3] = {n.x, n.y, n.z};
  float l[3], h[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float slack = 1.0e-3f * reach + 1.0e-6f * fabsf(oc[k]);
    l[k] = oc[k] - slack;
    h[k] = oc[k] + slack;
    add_axis(uc[k], -0.002f, x1, l[k], h[k]);       // blade -0.001 .. len + 0.001 past the stem, petiole radius 0.0011
    add_axis(vc[k], -w, w, l[k], h[k]);
    add_axis(nc[k], z0, z1, l[k], h[k]);
  }
  if (!(l[0] >= lo.x && l[1] >= lo.y && l[2] >= lo.z && h[0] <= hi.x && h[1] <= hi.y && h[2] <= hi.z)) return -1.0f;
  lo.x = l[0], lo.y = l[1], lo.z = l[2];
  hi.x = h[0], hi.y = h[1], hi.z = h[2];
  return reach;
}

// The grid of a scene's stored boxes, over its root box: origin and step.
struct TightGridC {
  f3 origin, step;
};
__device__ __forceinline__ TightGridC tight_grid(const float* Nodes) {
  const f3 lo = xyz(ldg4(Nodes, 2)), hi = xyz(ldg4(Nodes, 3));
  return {lo, (hi - lo) * (1.00001f / 65535.0f)};
}
__device__ __forceinline__ uint32_t grid_pair(float lo, float hi, float origin, float step) {
  const float a = fminf(fmaxf(floorf((lo - origin) / step) - 1.0f, 0.0f), 65535.0f);
  const float b = fminf(fmaxf(ceilf((hi - origin) / step) + 1.0f, 0.0f), 65535.0f);
  return (uint32_t)a | ((uint32_t)b << 16);
}
// Node `node`'s box on the grid: per axis lo | hi << 16.  A box without
// primitives is stored inside out (lo 65535, hi 0).
__device__ __forceinline__ void store_tight(uint32_t* T, int node, const TightGridC& g, float4 lo, float4 hi) {
  uint32_t* t = T + 3 * node;
  const bool some = lo.w > 0.0f;
  t[0] = some ? grid_pair(lo.x, hi.x, g.origin.x, g.step.x) : 65535u;
  t[1] = some ? grid_pair(lo.y, hi.y, g.origin.y, g.step.y) : 65535u;
  t[2] = some ? grid_pair(lo.z, hi.z, g.origin.z, g.step.z) : 65535u;
}

// Part `part` of a scene's tight boxes, by one CTA of 256 threads.
__device__ __forceinline__ void tight_build_part(TightPart& s, const float* __restrict__ P, const uint32_t* __restrict__ Order,
                                                 const float* __restrict__ Nodes, uint32_t* __restrict__ T, int part) {
  const int tid = threadIdx.x;
  const TightGridC g = tight_grid(Nodes);
  // (a grid that is not finite, or has no extent on an axis, holds nothing)
  bool bad = !(g.step.x > 1.0e-20f && g.step.y > 1.0e-20f && g.step.z > 1.0e-20f && fmaxf(g.step.x, fmaxf(g.step.y, g.step.z)) < 1.0f);
  float reach = 0.0f;
  for (int k = tid; k < kTightLeaves; k += blockDim.x) {
    const int slot = part * kTightLeaves + k, node = kCapacity + slot;
    const uint32_t uid = __ldg(Order + slot);
    const float4 nlo = ldg4(Nodes, 2 * node), nhi = ldg4(Nodes, 2 * node + 1);
    float4 lo, hi;
    leaf_record(P, uid, lo, hi);
    bad |= !same_box(lo, hi, nlo, nhi);
    if (lo.w > 0.0f) {
      const float r = tighten_record(P, (int)uid, lo, hi);
      bad |= !(r >= 0.0f);
      reach = fmaxf(reach, r);
    }
    s.lo[k] = lo;
    s.hi[k] = hi;
    store_tight(T, node, g, lo, hi);
    store_tight(T + kNodeBoxes, node, g, nlo, nhi);
  }
  // Nodes' inner nodes: the unions of their children?  (part 0 also looks at
  // the nodes above the parts)
  for (int k = tid; k < kTightLeaves; k += blockDim.x) {
    if (k > 0) {  // the k-th inner node of this part's subtree, k = 1 its root
      const int depth = 31 - __clz(k);
      const int node = ((kTightParts + part) << depth) + (k - (1 << depth));
      float4 plo, phi;
      merge(ldg4(Nodes, 4 * node), ldg4(Nodes, 4 * node + 1), ldg4(Nodes, 4 * node + 2), ldg4(Nodes, 4 * node + 3), plo, phi);
      const float4 nlo = ldg4(Nodes, 2 * node), nhi = ldg4(Nodes, 2 * node + 1);
      bad |= !same_box(plo, phi, nlo, nhi);
      store_tight(T + kNodeBoxes, node, g, nlo, nhi);
    }
  }
  if (part == 0 && tid < kTightParts) {
    const float4 lo = ldg4(Nodes, 2 * tid), hi = ldg4(Nodes, 2 * tid + 1);
    const float4 l = tid > 1 ? lo : make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // 0 and 1 are no one's children: empty
    store_tight(T, tid, g, l, hi);
    store_tight(T + kNodeBoxes, tid, g, l, hi);
    if (tid > 0) {
      float4 plo, phi;
      merge(ldg4(Nodes, 4 * tid), ldg4(Nodes, 4 * tid + 1), ldg4(Nodes, 4 * tid + 2), ldg4(Nodes, 4 * tid + 3), plo, phi);
      bad |= !same_box(plo, phi, lo, hi);
    }
  }
  __syncthreads();
  int first = kCapacity + part * kTightLeaves;
  for (int width = kTightLeaves / 2; width >= 1; width >>= 1) {
    first >>= 1;
    float4 plo, phi;
    if (tid < width) merge(s.lo[2 * tid], s.hi[2 * tid], s.lo[2 * tid + 1], s.hi[2 * tid + 1], plo, phi);
    __syncthreads();
    if (tid < width) {
      s.lo[tid] = plo;
      s.hi[tid] = phi;
      store_tight(T, first + tid, g, plo, phi);
    }
    __syncthreads();
  }
  // the part's reach (non-negative floats order as their bits do)
  __shared__ int part_reach;
  if (tid == 0) part_reach = 0;
  const bool any_bad = __syncthreads_or(bad);
  atomicMax(&part_reach, __float_as_int(reach));
  __syncthreads();
  if (tid == 0) T[kTightReach + part] = any_bad ? __float_as_uint(-1.0f) : (uint32_t)part_reach;
  if (part == 0 && tid == 0) {
    const float v[6] = {g.origin.x, g.origin.y, g.origin.z, g.step.x, g.step.y, g.step.z};
    for (int k = 0; k < 6; k++) T[kTightGrid + k] = __float_as_uint(v[k]);
  }
}
static_assert(kTightLeaves / 2 == 256, "one thread per node of the widest inner level");

// What a pass traverses.
struct TightView {
  const uint32_t* T;  // the boxes of its scene(s), kTightWords each; null: Nodes, in a fixed order (orderbatch.cuh)
  float rel, abs;     // the boxes' margin: rel x D + abs
  float most;         // the widest margin at which primary rays take them
};
// Largest swing of a leaf under `wind` whose reach is `reach`.
__device__ __forceinline__ float swing_margin(float wind, float reach) { return fminf(fabsf(wind) * kSwing, 2.0f) * reach; }

// One warp: the view of one scene's tight boxes.
__device__ __forceinline__ TightView tight_view_warp(const uint32_t* T, float wind) {
  const int lane = threadIdx.x & 31;
  const float a = __uint_as_float(__ldg(T + kTightReach + lane)), b = __uint_as_float(__ldg(T + kTightReach + 32 + lane));
  if (__any_sync(0xffffffffu, !(a >= 0.0f) || !(b >= 0.0f))) return {nullptr, 0.0f, 0.0f, 0.0f};
  const int reach = __reduce_max_sync(0xffffffffu, __float_as_int(fmaxf(a, b)));
  return {T, kTightRel, swing_margin(wind, __int_as_float(reach)), kTightMost * __int_as_float(reach)};
}
// A block: the view of n scenes' boxes T (null: none were made).  Every thread
// calls it.
__device__ __forceinline__ TightView tight_view_block(const uint32_t* T, int n, float wind) {
  __shared__ int reach;
  if (T == nullptr) return {nullptr, 0.0f, 0.0f, 0.0f};
  if (threadIdx.x == 0) reach = 0;
  __syncthreads();
  bool bad = false;
  for (int k = threadIdx.x; k < n * kTightParts; k += blockDim.x) {
    const float r = __uint_as_float(__ldg(T + (size_t)(k / kTightParts) * kTightWords + kTightReach + k % kTightParts));
    bad |= !(r >= 0.0f);
    atomicMax(&reach, __float_as_int(r));
  }
  if (__syncthreads_or(bad)) return {nullptr, 0.0f, 0.0f, 0.0f};
  return {T, kTightRel, swing_margin(wind, __int_as_float(reach)), kTightMost * __int_as_float(reach)};
}

// Primary rays prune with the margin as slack (enter_tree), and where it is a
// good part of a tree's depth nothing is pruned in it: the fixed order, which
// prunes by the nearest t alone, is then the faster one, up to 8 times.  The line
// lies at a margin of kTightShare of the root box's widest side.  Single trees at
// 256x256, tight boxes against fixed order: 0.64 / 0.72 ms at 0.033 (a grown tree
// at 300 m), 0.96 / 1.00 at 0.032, 0.70 / 0.72 at 0.045, 1.16 / 1.13 at 0.055, 0.82
// / 0.70 at 0.064, 2.09 / 0.72 at 0.066.  Forests at 1280x720, judged at kForestFar:
// 2.04 / 2.26 ms at 0.018 (grown trees), 1.55 / 1.97 at 0.035, 1.60 / 1.57 at 0.050,
// 2.02 / 1.32 at 0.087 (a fifth as large), grown trees in a storm (wind 8) 2.48 /
// 2.24 at 0.047.
constexpr float kTightShare = 0.045f;
constexpr float kForestFar = 160.0f;  // a forest's rays meet trees up to a few hundred metres away
// What primary rays traverse that meet trees up to `far` away, of the n scenes
// of view v.
__device__ __forceinline__ TightView primary_view(TightView v, int n, float far) {
  if (v.T == nullptr) return v;
  float side = 0.0f;
  for (int s = 0; s < n; s++) {
    const float* step = reinterpret_cast<const float*>(v.T + (size_t)s * kTightWords) + kTightGrid + 3;
    side = fmaxf(side, 65535.0f * fmaxf(__ldg(step), fmaxf(__ldg(step + 1), __ldg(step + 2))));
  }
  if (v.rel * far + v.abs > kTightShare * side) v.T = nullptr;
  return v;
}
// What shadow segments traverse.  Their margin is the leaves' swing: in wind above
// kShadowWind the widened boxes hold so many neighbours that the fixed order is the
// faster one.  Tight boxes against fixed order, grown forest at 1280x720: 2.62 /
// 4.31 ms at wind 0.6, 4.08 / 4.74 at 2, 4.54 / 4.42 at 2.5, 5.14 / 4.70 at 3, 13.8 /
// 4.64 at 8, 23.3 / 4.86 at 30; the same line for trees a fifth as large (3.61 /
// 3.61 at 2.5).
constexpr float kShadowWind = 2.5f;
__device__ __forceinline__ TightView shadow_view(TightView v, float wind) {
  if (v.abs > 0.0f && !(fabsf(wind) <= kShadowWind)) v.T = nullptr;  // (no leaves: no swing)
  return v;
}
// The farthest point of a view's (one) root box from `eye`.
__device__ __forceinline__ float tree_far(const TightView& v, f3 eye) {
  if (v.T == nullptr) return 0.0f;
  const float* g = reinterpret_cast<const float*>(v.T) + kTightGrid;
  const f3 lo = mk(__ldg(g), __ldg(g + 1), __ldg(g + 2)) - eye, hi = lo + mk(__ldg(g + 3), __ldg(g + 4), __ldg(g + 5)) * 65535.0f;
  return length3(max3(mk(fabsf(lo.x), fabsf(lo.y), fabsf(lo.z)), mk(fabsf(hi.x), fabsf(hi.y), fabsf(hi.z))));
}

}  // namespace arbor
