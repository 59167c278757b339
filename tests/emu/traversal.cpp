// traversal.cpp - the batched traversal (csrc/blockbatch.cuh and below it) and
// the reference's traversal as written (arbor_scene.cuh), on the CPU, for
// tests/test_traversal_cpu.py.
#include "block_emu.h"

#include "blockbatch.cuh"

using namespace arbor;

namespace {

// Rays given one by one in place of an image's pixels: n x {origin, direction,
// nearest t}; results n x {t, record id, tree}.
struct RayPolicy {
  static constexpr int kRefill = 8;
  const float* rays;
  float* out;
  int n, index;
  void bind(const TraceCtx*) {}
  void start(const TraceCtx& c, Ray& r, int x, int y) {
    index = y * 8 + x;
    if (index >= n) return;
    const float* a = rays + 7 * index;
    ray_begin(c, r, mk(a[0], a[1], a[2]), mk(a[3], a[4], a[5]), a[6]);
  }
  void done(Ray& r) {
    out[3 * index] = r.best;
    out[3 * index + 1] = r.found;
    out[3 * index + 2] = (float)r.foundTree;
    r.phase = kPhIdle;
  }
};

}  // namespace

extern "C" {

void emu_leaf_nodes(const float* P, const uint32_t* Order, float* Nodes) {  // arbor_buildBounds
  emu::buffers = {{(const char*)P, (const char*)(P + kCapacity * kPS)}};
  float4* n = reinterpret_cast<float4*>(Nodes);
  n[0] = n[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int k = 0; k < kCapacity; k++) leaf_record(P, Order[k], n[2 * (kCapacity + k)], n[2 * (kCapacity + k) + 1]);
  for (int k = kCapacity - 1; k >= 1; k--) merge(n[4 * k], n[4 * k + 1], n[4 * k + 2], n[4 * k + 3], n[2 * k], n[2 * k + 1]);
}

static long trace_loads;
long emu_loads() { return trace_loads; }  // of the last emu_trace
int emu_words() { return kTightWords; }

// The tight boxes of a scene; returns the loads outside P, Order and Nodes.
long emu_boxes(const float* P, const uint32_t* Order, const float* Nodes, uint32_t* T) {
  emu::buffers = {{(const char*)P, (const char*)(P + kCapacity * kPS)},
                  {(const char*)Order, (const char*)(Order + kCapacity)},
                  {(const char*)Nodes, (const char*)(Nodes + kNodeCount * 8)}};
  emu::bad_loads = 0;
  static TightPart s;
  for (int part = 0; part < kTightParts; part++) emu::run(kThreads, part, kTightParts, [&] { tight_build_part(s, P, Order, Nodes, T, part); });
  return emu::bad_loads;
}

// Traces n rays through the block batch over the boxes T (null: none).  inst:
// a forest of 324 instances, or null for the single tree.  Returns the loads
// outside the buffers; *regular: whether the boxes were used.
long emu_trace(const float* P, const uint32_t* Order, const float* Nodes, const uint32_t* T, const Instance* inst, const float* rays, int n,
               float cone, float time, float wind, int refine, float* out, int* regular) {
  emu::buffers = {{(const char*)P, (const char*)(P + kCapacity * kPS)},
                  {(const char*)Order, (const char*)(Order + kCapacity)},
                  {(const char*)Nodes, (const char*)(Nodes + kNodeCount * 8)}};
  if (T) emu::buffers.push_back({(const char*)T, (const char*)(T + kTightWords)});
  emu::bad_loads = emu::loads = 0;
  static BlockBatch batch;
  static int next;
  next = 0;
  emu::run(kThreads, 0, 1, [&] {
    const TightView tight = tight_view_block(T, 1, wind);
    if (threadIdx.x == 0) *regular = tight.T != nullptr;
    const TraceCtx c{P, Nodes, Order, inst, tight, cone, time, wind, refine != 0, inst != nullptr};
    const int rows = (n + 7) / 8;
    const PixelPool pool{&next, 8, rows, 1, (rows + 3) / 4};
    RayPolicy policy{rays, out, n, 0};
    Ray r;
    block_run_pool(c, r, batch, policy, pool);
  });
  trace_loads = emu::loads;
  return emu::bad_loads;
}

// Whether primary rays of a scene take its boxes (1) or the fixed order (0):
// from `eye` for the single tree, anywhere in a forest without.
int emu_primary_takes_boxes(const uint32_t* T, float wind, const float* eye) {
  emu::buffers = {{(const char*)T, (const char*)(T + kTightWords)}};
  int takes = -1;
  emu::run(kThreads, 0, 1, [&] {
    const TightView boxes = tight_view_block(T, 1, wind);
    const TightView v = primary_view(boxes, 1, eye ? tree_far(boxes, mk(eye[0], eye[1], eye[2])) : kForestFar);
    if (threadIdx.x == 0) takes = v.T != nullptr;
  });
  return takes;
}

// Whether its shadow segments do.
int emu_shadow_takes_boxes(const uint32_t* T, float wind) {
  emu::buffers = {{(const char*)T, (const char*)(T + kTightWords)}};
  int takes = -1;
  emu::run(kThreads, 0, 1, [&] {
    const TightView v = shadow_view(tight_view_block(T, 1, wind), wind);
    if (threadIdx.x == 0) takes = v.T != nullptr;
  });
  return takes;
}

// The same rays one by one, each tree by tree_in_order.
void emu_in_order(const float* P, const uint32_t* Order, const float* Nodes, const Instance* inst, const float* rays, int n, float cone,
                  float time, float wind, int refine, float* out) {
  emu::buffers = {{(const char*)P, (const char*)(P + kCapacity * kPS)},
                  {(const char*)Order, (const char*)(Order + kCapacity)},
                  {(const char*)Nodes, (const char*)(Nodes + kNodeCount * 8)}};
  const TraceCtx c{P, Nodes, Order, inst, {}, cone, time, wind, refine != 0, inst != nullptr};
  for (int k = 0; k < n; k++) {
    const float* a = rays + 7 * k;
    Ray r;
    ray_begin(c, r, mk(a[0], a[1], a[2]), mk(a[3], a[4], a[5]), a[6]);
    while (r.phase != kPhDone) {
      LocalRay l;
      if (!dda_next(c, r, l)) continue;
      const TreeResult h = tree_in_order(P, Nodes, Order, make_float4(l.ro.x, l.ro.y, l.ro.z, l.time),
                                         make_float4(l.rd.x, l.rd.y, l.rd.z, l.cone), inv3(l.rd), wind, r.lbest, c.refine, kOrderedChunk);
      r.lbest = h.t;
      r.lfound = h.slot;
      fold_tree(c, r);
    }
    out[3 * k] = r.best;
    out[3 * k + 1] = r.found;
    out[3 * k + 2] = (float)r.foundTree;
  }
}

// The same rays one by one in the reference's order.
void emu_reference(const float* P, const uint32_t* Order, const float* Nodes, const Instance* inst, const float* rays, int n, float cone,
                   float time, float wind, int refine, float* out) {
  emu::buffers = {{(const char*)P, (const char*)(P + kCapacity * kPS)},
                  {(const char*)Order, (const char*)(Order + kCapacity)},
                  {(const char*)Nodes, (const char*)(Nodes + kNodeCount * 8)}};
  for (int k = 0; k < n; k++) {
    const float* a = rays + 7 * k;
    int tree = -1;
    const f2 h = inst ? trace_forest(P, Nodes, Order, inst, mk(a[0], a[1], a[2]), mk(a[3], a[4], a[5]), cone, time, wind, a[6], &tree, !refine)
                      : trace_tree(P, Nodes, Order, mk(a[0], a[1], a[2]), mk(a[3], a[4], a[5]), cone, time, wind, a[6], -1, !refine);
    out[3 * k] = h.x;
    out[3 * k + 1] = h.y;
    out[3 * k + 2] = (float)tree;
  }
}

void emu_instances(int world_seed, Instance* inst) {
  for (int t = 0; t < kForest; t++) inst[t] = make_instance(t, world_seed);
}
int emu_instance_bytes() { return (int)sizeof(Instance); }

}  // extern "C"
