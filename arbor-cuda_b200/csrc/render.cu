// render.cu - per-frame image passes: tracePixels and shadePixels
// (Arbor.cu:252-289) and their single-tree and species variants, with their
// C-ABI entry points (filter and resolve: filter.cu).
//
// Launch shapes: the trace and the shade's shadow pass are persistent (2
// CTAs per SM, lanes taking pixels of 8x4 blocks as their rays finish); the
// shade's compose pass runs 256-thread blocks over 16x16 pixel tiles.  The
// persistent passes read the 324-entry forest instance table from the
// world-seed registry (pass_instances); the compose blocks build it in shared
// memory once.  Every table entry equals what the reference's forest helpers
// recompute per ray (Arbor.cu:57-69).
#include <algorithm>

#include "abi_util.h"
#include "passes.cuh"
#include "per_device.h"
#include "scratch.h"

namespace arbor {
namespace {

// ---------------------------------------------------------------- kernels --
// Dynamic shared memory of a persistent pass: the block batch and, for a pass
// without scratch, room for an instance table.
struct PassSmem {
  BlockBatch batch;
  Instance table[kForest];
};
constexpr size_t kPassSmem = sizeof(BlockBatch), kPassSmemTable = sizeof(PassSmem);
static_assert(2 * (kPassSmemTable + 1024 + 512) <= 228 * 1024, "two CTAs per SM");
static_assert(kBlock == kThreads, "a block batch is one block's");
// The instance table of a persistent pass: the registry slot's (global
// memory) when the host registered the world seed, else the one in the
// scratch behind n_scenes' tight boxes (tight_kernel), or without scratch one
// built in shared memory.  Every thread of the block calls it.
__device__ __forceinline__ const Instance* pass_instances(const WorldTrig* trig, int ws, const uint32_t* T, int n_scenes, PassSmem& smem) {
  const WorldTrig* slot = world_slot_of(trig, ws);
  if (slot != nullptr) return slot->inst;
  if (T != nullptr) return reinterpret_cast<const Instance*>(T + (size_t)n_scenes * kTightWords);
  for (int t = threadIdx.x; t < kForest; t += blockDim.x) smem.table[t] = make_instance(t, ws);
  __syncthreads();
  return smem.table;
}

// Persistent form of the trace: a grid of (SMs x 2) CTAs, each taking every
// gridDim.x-th 8x4-pixel block of the image, its lanes taking pixels as
// their rays finish (block_run_pool).
template <bool kForestScene>
__global__ void __launch_bounds__(kBlock, 2) trace_pool_kernel(const float* __restrict__ P, const float* __restrict__ Nodes,
                                                               const uint32_t* __restrict__ Order, const float* __restrict__ C,
                                                               const WorldTrig* __restrict__ trig, const uint32_t* __restrict__ T,
                                                               float* __restrict__ Hit, int width, int height) {
  extern __shared__ float4 batch_smem[];
  PassSmem& smem = *reinterpret_cast<PassSmem*>(batch_smem);
  __shared__ Camera cam;
  __shared__ int next;
  if (threadIdx.x == 0) next = 0;
  block_setup(C, cam, nullptr, false, nullptr);
  const Instance* inst = kForestScene ? pass_instances(trig, cam.ws, T, 1, smem) : nullptr;
  const TightView boxes = tight_view_block(T, 1, cam.wind);
  const TightView tight = primary_view(boxes, 1, kForestScene ? kForestFar : tree_far(boxes, cam.ro));
  const TraceCtx c{P, Nodes, Order, inst, tight, cam.c14 / (float)height, cam.time, cam.wind, true, kForestScene};
  const int bx = (width + 7) / 8;
  const PixelPool pool{&next, width, height, bx, bx * ((height + 3) / 4)};
  trace_pool(c, cam, smem.batch, Hit, pool);
}

// shadePixels in two passes.  The shadow pass is persistent like the trace:
// lanes take pixels from a pool and trace their shadow segments, writing the
// visibility into Linear; with sun shadows off it returns at once.  Each CTA
// first stages the shadow rays of its own pixels (stage_shadows: origin into
// Linear, direction into Guide; both are overwritten by the compose pass), so
// the tracer's loop holds no camera or sun-sampling code.
template <bool kForestScene>
__global__ void __launch_bounds__(kBlock, 2) shadow_pool_kernel(const float* __restrict__ P, const float* __restrict__ Nodes,
                                                                const uint32_t* __restrict__ Order, const float* __restrict__ C,
                                                                const WorldTrig* __restrict__ trig, const uint32_t* __restrict__ T,
                                                                const float* __restrict__ Hit, float* Guide, float* Linear, int width, int height) {
  extern __shared__ float4 batch_smem[];
  PassSmem& smem = *reinterpret_cast<PassSmem*>(batch_smem);
  __shared__ Camera cam;
  __shared__ int next;
  if (threadIdx.x == 0) next = 0;
  block_setup(C, cam, nullptr, false, nullptr);
  if (!(cam.shadows > 0.5f)) return;
  const int bx = (width + 7) / 8;
  const PixelPool pool{&next, width, height, bx, bx * ((height + 3) / 4)};
  stage_shadows(cam, Hit, Linear, Guide, pool);
  const Instance* inst = kForestScene ? pass_instances(trig, cam.ws, T, 1, smem) : nullptr;
  const TightView tight = shadow_view(tight_view_block(T, 1, cam.wind), cam.wind);
  const TraceCtx c{P, Nodes, Order, inst, tight, 0.0001f, cam.time, cam.wind, false, kForestScene};
  staged_shadow_pool(c, smem.batch, Guide, Linear, pool);
}

// The tight boxes (tight.cuh) of n_scenes scenes, one part per CTA, and behind
// them, by one more CTA, the instance table of a world seed that the registry
// does not hold.  C: the pass's camera record; with `shadows` the boxes are
// for a shadow pass, and with sun shadows off nothing is made.
__global__ void __launch_bounds__(kBlock) tight_kernel(const float* __restrict__ P, const uint32_t* __restrict__ Order,
                                                       const float* __restrict__ Nodes, uint32_t* __restrict__ T, int n_scenes,
                                                       const float* __restrict__ C, bool shadows, const WorldTrig* __restrict__ trig) {
  __shared__ TightPart s;
  if (shadows && !(C[22] > 0.5f)) return;
  const size_t k = blockIdx.x / kTightParts;
  if ((int)k == n_scenes) {
    const int ws = (int)C[31];
    if (world_slot_of(trig, ws) != nullptr) return;
    Instance* table = reinterpret_cast<Instance*>(T + k * kTightWords);
    for (int t = threadIdx.x; t < kForest; t += blockDim.x) table[t] = make_instance(t, ws);
    return;
  }
  tight_build_part(s, P + k * (kCapacity * kPS), Order + k * kCapacity, Nodes + k * (kNodeCount * 8), T + k * kTightWords,
                   (int)(blockIdx.x % kTightParts));
}

// The compose pass: one pixel per thread, the surface terms and the colour
// with the shadow pass's visibility; 4 CTAs per SM (64 registers) hide its
// memory latency better than 3 (measured 0.557 -> 0.530 ms at 1080p).
template <bool kForestScene>
__global__ void __launch_bounds__(kBlock, 4) shade_compose_kernel(const float* __restrict__ P, const float* __restrict__ C,
                                                                  const WorldTrig* __restrict__ trig, const float* __restrict__ Hit,
                                                                  float* __restrict__ Linear, float* __restrict__ Guide, float* __restrict__ Normal,
                                                                  int width, int height) {
  __shared__ Camera cam;
  __shared__ Instance inst[kForestScene ? kForest : 1];
  block_setup(C, cam, inst, kForestScene, trig);
  int x, y;
  tile_pixel_at(threadIdx.x, blockIdx.x * kTile, blockIdx.y * kTile, kTile, x, y);
  if (x < width && y < height) shade_compose_px<kForestScene>(P, cam, inst, Hit, Linear, Guide, Normal, x, y, width, height);
}

// ------------------------------------------------ forest of several species --
// The reference's 324 instances all share one resident tree (README.md:8,
// docs/ARCHITECTURE.md:5).  These kernels trace and shade a forest whose
// instance t keeps the reference's transform, wind phase and tint but takes
// its geometry (its own records and BVH) from scene of[t]; P, Nodes and Order
// hold the scenes back to back.  The 2D DDA, bounding spheres and every
// per-instance step are the reference's; only the scene a tree's traversal
// and tests read changes.  With every of[t] = 0 the results equal
// arbor_tracePixels / arbor_shadePixels on scene 0.
struct SpeciesMap {
  uint8_t of[kForest];
};
__device__ __forceinline__ void species_setup(Instance* inst, const SpeciesMap& m) {
  for (int t = threadIdx.x; t < kForest; t += blockDim.x) inst[t].species = m.of[t];
  __syncthreads();
}

__global__ void __launch_bounds__(kBlock, 2) trace_species_kernel(const float* __restrict__ P, const float* __restrict__ Nodes,
                                                                  const uint32_t* __restrict__ Order, const float* __restrict__ C,
                                                                  const WorldTrig* __restrict__ trig, const uint32_t* __restrict__ T, int n_scenes,
                                                                  float* __restrict__ Hit, int width, int height, const SpeciesMap map) {
  extern __shared__ float4 batch_smem[];
  PassSmem& smem = *reinterpret_cast<PassSmem*>(batch_smem);
  __shared__ Camera cam;
  __shared__ uint8_t of[kForest];
  __shared__ int next;
  if (threadIdx.x == 0) next = 0;
  for (int t = threadIdx.x; t < kForest; t += blockDim.x) of[t] = map.of[t];
  block_setup(C, cam, nullptr, false, nullptr);
  const Instance* inst = pass_instances(trig, cam.ws, T, n_scenes, smem);
  const TightView tight = primary_view(tight_view_block(T, n_scenes, cam.wind), n_scenes, kForestFar);
  const TraceCtx c{P, Nodes, Order, inst, tight, cam.c14 / (float)height, cam.time, cam.wind, true, true, true, of};
  const int bx = (width + 7) / 8;
  const PixelPool pool{&next, width, height, bx, bx * ((height + 3) / 4)};
  trace_pool(c, cam, smem.batch, Hit, pool);
}

__global__ void __launch_bounds__(kBlock, 2) shadow_species_kernel(const float* __restrict__ P, const float* __restrict__ Nodes,
                                                                   const uint32_t* __restrict__ Order, const float* __restrict__ C,
                                                                   const WorldTrig* __restrict__ trig, const uint32_t* __restrict__ T, int n_scenes,
                                                                   const float* __restrict__ Hit, float* Guide, float* Linear, int width, int height,
                                                                   const SpeciesMap map) {
  extern __shared__ float4 batch_smem[];
  PassSmem& smem = *reinterpret_cast<PassSmem*>(batch_smem);
  __shared__ Camera cam;
  __shared__ uint8_t of[kForest];
  __shared__ int next;
  if (threadIdx.x == 0) next = 0;
  for (int t = threadIdx.x; t < kForest; t += blockDim.x) of[t] = map.of[t];
  block_setup(C, cam, nullptr, false, nullptr);
  if (!(cam.shadows > 0.5f)) return;
  const int bx = (width + 7) / 8;
  const PixelPool pool{&next, width, height, bx, bx * ((height + 3) / 4)};
  stage_shadows(cam, Hit, Linear, Guide, pool);
  const Instance* inst = pass_instances(trig, cam.ws, T, n_scenes, smem);
  const TightView tight = shadow_view(tight_view_block(T, n_scenes, cam.wind), cam.wind);
  const TraceCtx c{P, Nodes, Order, inst, tight, 0.0001f, cam.time, cam.wind, false, true, true, of};
  staged_shadow_pool(c, smem.batch, Guide, Linear, pool);
}

__global__ void __launch_bounds__(kBlock, 4) shade_compose_species_kernel(const float* __restrict__ P, const float* __restrict__ C,
                                                                          const WorldTrig* __restrict__ trig,
                                                                          const float* __restrict__ Hit, float* __restrict__ Linear,
                                                                          float* __restrict__ Guide, int width, int height, const SpeciesMap map) {
  __shared__ Camera cam;
  __shared__ Instance inst[kForest];
  block_setup(C, cam, inst, true, trig);
  species_setup(inst, map);
  int x, y;
  tile_pixel_at(threadIdx.x, blockIdx.x * kTile, blockIdx.y * kTile, kTile, x, y);
  if (x < width && y < height) shade_compose_px<true, true>(P, cam, inst, Hit, Linear, Guide, nullptr, x, y, width, height);
}

// tracePixels and shadePixels with the reference's traversal as written
// (Arbor.cu:220-289): one ray per thread over 16x16-pixel CTAs, candidates
// tested in visiting order, children nearest entry first, no batching.
// Slower forms kept to check that the batched passes' order does not change
// a result (the in-order entry points).
template <bool kForestScene>
__global__ void __launch_bounds__(kBlock) trace_inorder_kernel(const float* __restrict__ P, const float* __restrict__ Nodes,
                                                               const uint32_t* __restrict__ Order, const float* __restrict__ C,
                                                               const WorldTrig* __restrict__ trig,
                                                               float* __restrict__ Hit, int width, int height) {
  __shared__ Camera cam;
  __shared__ Instance inst[kForestScene ? kForest : 1];
  block_setup(C, cam, inst, kForestScene, trig);
  int x, y;
  tile_pixel(threadIdx.x, x, y);
  if (x >= width || y >= height) return;
  const f3 ro = cam.ro;
  const f3 rd = camera_ray(cam, x, y, width, height);
  const float ground = rd.y < -0.00001f ? -ro.y / rd.y : kFar;
  const float cone = cam.c14 / (float)height;
  const float best = ground > 0.0f ? ground : kFar;
  int tree = -1;
  const f2 h = kForestScene ? trace_forest(P, Nodes, Order, inst, ro, rd, cone, cam.time, cam.wind, best, &tree, false)
                            : trace_tree(P, Nodes, Order, ro, rd, cone, cam.time, cam.wind, best, -1, false);
  reinterpret_cast<float4*>(Hit)[y * width + x] = make_float4(h.x, h.y, (float)tree, cam.c14 * h.x / (float)height);
}

template <bool kForestScene>
__global__ void __launch_bounds__(kBlock) shade_inorder_kernel(const float* __restrict__ P, const float* __restrict__ Nodes,
                                                               const uint32_t* __restrict__ Order, const float* __restrict__ C,
                                                               const WorldTrig* __restrict__ trig,
                                                               const float* __restrict__ Hit, float* __restrict__ Linear,
                                                               float* __restrict__ Guide, int width, int height) {
  __shared__ Camera cam;
  __shared__ Instance inst[kForestScene ? kForest : 1];
  block_setup(C, cam, inst, kForestScene, trig);
  int x, y;
  tile_pixel(threadIdx.x, x, y);
  if (x >= width || y >= height) return;
  const int pixel = y * width + x;
  Shading sh;
  shade_pre<kForestScene>(P, cam, inst, __ldg(reinterpret_cast<const float4*>(Hit) + pixel), x, y, width, height, sh);
  f3 vis = mk(1.0f, 1.0f, 1.0f);
  if (!sh.final && sh.shadow) {
    // lightVisibility (Arbor.cu:271-274)
    f3 trans = mk(1.0f, 1.0f, 1.0f);
    f3 o = sh.origin;
    for (int j = 0; j < 4; j++) {
      int tree = -1;
      const f2 h = kForestScene ? trace_forest(P, Nodes, Order, inst, o, sh.light, 0.0001f, cam.time, cam.wind, 36.0f, &tree, true)
                                : trace_tree(P, Nodes, Order, o, sh.light, 0.0001f, cam.time, cam.wind, 36.0f, -1, true);
      const int id = (int)h.y;
      if (id < 0) {
        vis = trans;
        break;
      }
      if (ldg4(P, id * 6).w != 1.0f) {
        vis = mk(0.0f, 0.0f, 0.0f);
        break;
      }
      trans = trans * mk(0.18f, 0.29f, 0.065f);
      o = o + sh.light * (h.x + 0.0018f);
      if (j == 3) vis = trans;
    }
  }
  const f3 col = shade_post(sh, vis);
  reinterpret_cast<float4*>(Linear)[pixel] = make_float4(col.x, col.y, col.z, 1.0f);
  reinterpret_cast<float4*>(Guide)[pixel] = make_float4(sh.guide.x, sh.guide.y, sh.guide.z, 1.0f);
}

template <auto Kernel>
bool pass_smem_ready() {
  return smem_opt_in<Kernel>((int)kPassSmemTable);
}

dim3 pixel_grid(int w, int h) { return dim3((w + kTile - 1) / kTile, (h + kTile - 1) / kTile); }

// Persistent grid: 2 CTAs per SM (the register and shared-memory limit of
// the batched tracer), or one CTA per 8x4 block when the image has fewer.
dim3 pool_grid(int w, int h) {
  const long blocks = (long)((w + 7) / 8) * ((h + 3) / 4);
  return dim3((unsigned)std::min<long>(blocks, 2L * device_sms()));
}
// Checks of tracePixels / shadePixels, shared by the entries and the engine.
int trace_checks(const char* name, const float* P, const float* Nodes, const uint32_t* Order, const float* C, const float* Hit, int width,
                 int height, bool* empty) {
  if (int s = check_image(name, width, height, empty)) return s;
  const Binding b[] = {{P, kP, false, 16, "P"},
                       {Nodes, kNodes, false, 16, "Nodes"},
                       {Order, kKeys, false, 4, "Order"},
                       {C, kC, false, 4, "C"},
                       {Hit, *empty ? 0 : image_bytes(width, height), true, 16, "Hit"}};
  return check_bindings(name, b);
}
int smem_error(const char* name) {
  set_error("%s: cannot reserve %zu bytes of shared memory per CTA", name, kPassSmemTable);
  return ARBOR_ERR_CUDA;
}

}  // namespace

size_t tight_bytes(int n_scenes) { return kTightBytes * (size_t)n_scenes + sizeof(Instance) * kForest; }
int launch_tight(const float* P, const uint32_t* Order, const float* Nodes, int n_scenes, uint32_t* T, const float* C, bool shadows,
                 cudaStream_t stream) {
  tight_kernel<<<kTightParts * n_scenes + 1, kBlock, 0, stream>>>(P, Order, Nodes, T, n_scenes, C, shadows, world_trig());
  count_launch();
  return check_launch("tight_kernel");
}

// tracePixels over the boxes T (tight boxes of the scene, or null: Nodes, in a
// fixed order).
int launch_trace(const char* name, bool forest, const float* P, const float* Nodes, const uint32_t* Order, const uint32_t* T, const float* C,
                 float* Hit, int width, int height, cudaStream_t stream) {
  if (!(forest ? pass_smem_ready<trace_pool_kernel<true>>() : pass_smem_ready<trace_pool_kernel<false>>())) return smem_error(name);
  if (forest)
    trace_pool_kernel<true><<<pool_grid(width, height), kBlock, T ? kPassSmem : kPassSmemTable, stream>>>(P, Nodes, Order, C, world_trig(), T, Hit, width, height);
  else
    trace_pool_kernel<false><<<pool_grid(width, height), kBlock, T ? kPassSmem : kPassSmemTable, stream>>>(P, Nodes, Order, C, world_trig(), T, Hit, width, height);
  count_launch();
  return check_launch(name);
}

// shadePixels over the boxes T: shadow segments in a persistent pass whose
// loop holds only the tracer (its code stays small), then the shading of
// every pixel.
int launch_shade(const char* name, bool forest, const float* P, const float* Nodes, const uint32_t* Order, const uint32_t* T, const float* C,
                 const float* Hit, float* Linear, float* Guide, float* Normal, int width, int height, cudaStream_t stream) {
  if (!(forest ? pass_smem_ready<shadow_pool_kernel<true>>() : pass_smem_ready<shadow_pool_kernel<false>>())) return smem_error(name);
  if (forest) {
    shadow_pool_kernel<true><<<pool_grid(width, height), kBlock, T ? kPassSmem : kPassSmemTable, stream>>>(P, Nodes, Order, C, world_trig(), T, Hit, Guide, Linear,
                                                                                       width, height);
    shade_compose_kernel<true><<<pixel_grid(width, height), kBlock, 0, stream>>>(P, C, world_trig(), Hit, Linear, Guide, Normal, width, height);
  } else {
    shadow_pool_kernel<false><<<pool_grid(width, height), kBlock, T ? kPassSmem : kPassSmemTable, stream>>>(P, Nodes, Order, C, world_trig(), T, Hit, Guide, Linear,
                                                                                        width, height);
    shade_compose_kernel<false><<<pixel_grid(width, height), kBlock, 0, stream>>>(P, C, world_trig(), Hit, Linear, Guide, Normal, width, height);
  }
  count_launch(2);
  return check_launch(name);
}

namespace {

int trace_entry(const char* name, bool forest, const float* P, const float* Nodes, const uint32_t* Order, const float* C, float* Hit, int width,
                int height, cudaStream_t stream) {
  bool empty;
  if (int s = trace_checks(name, P, Nodes, Order, C, Hit, width, height, &empty)) return s;
  if (empty) return ARBOR_OK;
  const TightScratch t(P, Order, Nodes, 1, C, false, stream);
  if (t.status) return t.status;
  return launch_trace(name, forest, P, Nodes, Order, t.boxes, C, Hit, width, height, stream);
}

int shade_entry(const char* name, bool forest, const float* P, const float* Nodes, const uint32_t* Order, const float* C, const float* Hit,
                float* Linear, float* Guide, int width, int height, cudaStream_t stream, float* Normal = nullptr) {
  bool empty;
  if (int s = check_image(name, width, height, &empty)) return s;
  size_t img = empty ? 0 : image_bytes(width, height);
  const Binding b[] = {{P, kP, false, 16, "P"},         {Nodes, kNodes, false, 16, "Nodes"}, {Order, kKeys, false, 4, "Order"},
                       {C, kC, false, 4, "C"},          {Hit, img, false, 16, "Hit"},        {Linear, img, true, 16, "Linear"},
                       {Guide, img, true, 16, "Guide"}};
  if (int s = check_bindings(name, b)) return s;
  if (Normal != nullptr) {
    const Binding g[] = {{P, kP, false, 16, "P"}, {Hit, img, false, 16, "Hit"}, {Linear, img, true, 16, "Linear"},
                         {Guide, img, true, 16, "Guide"}, {Normal, img, true, 16, "Normal"}};
    if (int s = check_bindings(name, g)) return s;
  }
  if (empty) return ARBOR_OK;
  const TightScratch t(P, Order, Nodes, 1, C, true, stream);
  if (t.status) return t.status;
  return launch_shade(name, forest, P, Nodes, Order, t.boxes, C, Hit, Linear, Guide, Normal, width, height, stream);
}

// Checks of a forest-of-species call: 1..256 scenes, every instance on one
// of them.  Fills `map`.
int species_args(const char* name, int n_species, const int* species_of, SpeciesMap& map) {
  if (n_species < 1 || n_species > ARBOR_MAX_SPECIES) {
    set_error("%s: n_species %d outside 1..%d", name, n_species, ARBOR_MAX_SPECIES);
    return ARBOR_ERR_VALUE;
  }
  if (species_of == nullptr) {
    set_error("%s: species_of is NULL", name);
    return ARBOR_ERR_NULL;
  }
  for (int t = 0; t < kForest; t++) {
    if (species_of[t] < 0 || species_of[t] >= n_species) {
      set_error("%s: species_of[%d] = %d outside 0..%d", name, t, species_of[t], n_species - 1);
      return ARBOR_ERR_VALUE;
    }
    map.of[t] = (uint8_t)species_of[t];
  }
  return ARBOR_OK;
}

}  // namespace
}  // namespace arbor

using namespace arbor;

extern "C" int arbor_traceSpeciesPixels(const float* P, const float* Nodes, const uint32_t* Order, int n_species, const int* species_of,
                                        const float* C, float* Hit, int width, int height, arbor_stream stream) {
  const char* name = "arbor_traceSpeciesPixels";
  SpeciesMap map;
  if (int s = species_args(name, n_species, species_of, map)) return s;
  bool empty;
  if (int s = check_image(name, width, height, &empty)) return s;
  const size_t n = (size_t)n_species;
  const Binding b[] = {{P, n * kP, false, 16, "P"},
                       {Nodes, n * kNodes, false, 16, "Nodes"},
                       {Order, n * kKeys, false, 4, "Order"},
                       {C, kC, false, 4, "C"},
                       {Hit, empty ? 0 : image_bytes(width, height), true, 16, "Hit"}};
  if (int s = check_bindings(name, b)) return s;
  if (empty) return ARBOR_OK;
  if (!pass_smem_ready<trace_species_kernel>()) return smem_error(name);
  const TightScratch t(P, Order, Nodes, n_species, C, false, stream);
  if (t.status) return t.status;
  trace_species_kernel<<<pool_grid(width, height), kBlock, t.boxes ? kPassSmem : kPassSmemTable, stream>>>(P, Nodes, Order, C, world_trig(), t.boxes, n_species, Hit, width,
                                                                                 height, map);
  count_launch();
  return check_launch(name);
}
extern "C" int arbor_shadeSpeciesPixels(const float* P, const float* Nodes, const uint32_t* Order, int n_species, const int* species_of,
                                        const float* C, const float* Hit, float* Linear, float* Guide, int width, int height, arbor_stream stream) {
  const char* name = "arbor_shadeSpeciesPixels";
  SpeciesMap map;
  if (int s = species_args(name, n_species, species_of, map)) return s;
  bool empty;
  if (int s = check_image(name, width, height, &empty)) return s;
  const size_t n = (size_t)n_species;
  const size_t img = empty ? 0 : image_bytes(width, height);
  const Binding b[] = {{P, n * kP, false, 16, "P"},  {Nodes, n * kNodes, false, 16, "Nodes"}, {Order, n * kKeys, false, 4, "Order"},
                       {C, kC, false, 4, "C"},      {Hit, img, false, 16, "Hit"},             {Linear, img, true, 16, "Linear"},
                       {Guide, img, true, 16, "Guide"}};
  if (int s = check_bindings(name, b)) return s;
  if (empty) return ARBOR_OK;
  if (!pass_smem_ready<shadow_species_kernel>()) return smem_error(name);
  const TightScratch t(P, Order, Nodes, n_species, C, true, stream);
  if (t.status) return t.status;
  shadow_species_kernel<<<pool_grid(width, height), kBlock, t.boxes ? kPassSmem : kPassSmemTable, stream>>>(P, Nodes, Order, C, world_trig(), t.boxes, n_species, Hit, Guide,
                                                                                  Linear, width, height, map);
  shade_compose_species_kernel<<<pixel_grid(width, height), kBlock, 0, stream>>>(P, C, world_trig(), Hit, Linear, Guide, width, height, map);
  count_launch(2);
  return check_launch(name);
}

extern "C" int arbor_tracePixels(const float* P, const float* Nodes, const uint32_t* Order, const float* C, float* Hit, int width, int height,
                                 arbor_stream stream) {
  return trace_entry("arbor_tracePixels", true, P, Nodes, Order, C, Hit, width, height, stream);
}
extern "C" int arbor_traceTreePixels(const float* P, const float* Nodes, const uint32_t* Order, const float* C, float* Hit, int width, int height,
                                     arbor_stream stream) {
  return trace_entry("arbor_traceTreePixels", false, P, Nodes, Order, C, Hit, width, height, stream);
}
extern "C" int arbor_shadePixels(const float* P, const float* Nodes, const uint32_t* Order, const float* C, const float* Hit, float* Linear,
                                 float* Guide, int width, int height, arbor_stream stream) {
  return shade_entry("arbor_shadePixels", true, P, Nodes, Order, C, Hit, Linear, Guide, width, height, stream);
}
extern "C" int arbor_shadeGBuffer(const float* P, const float* Nodes, const uint32_t* Order, const float* C, const float* Hit, float* Linear,
                                  float* Guide, float* Normal, int width, int height, arbor_stream stream) {
  if (Normal == nullptr && width > 0 && height > 0) {
    set_error("arbor_shadeGBuffer: buffer Normal is NULL");
    return ARBOR_ERR_NULL;
  }
  return shade_entry("arbor_shadeGBuffer", true, P, Nodes, Order, C, Hit, Linear, Guide, width, height, stream, Normal);
}
extern "C" int arbor_shadeTreePixels(const float* P, const float* Nodes, const uint32_t* Order, const float* C, const float* Hit, float* Linear,
                                     float* Guide, int width, int height, arbor_stream stream) {
  return shade_entry("arbor_shadeTreePixels", false, P, Nodes, Order, C, Hit, Linear, Guide, width, height, stream);
}
extern "C" int arbor_tracePixelsInOrder(const float* P, const float* Nodes, const uint32_t* Order, const float* C, float* Hit, int width,
                                        int height, int single_tree, arbor_stream stream) {
  const char* name = "arbor_tracePixelsInOrder";
  bool empty;
  if (int s = check_image(name, width, height, &empty)) return s;
  const Binding b[] = {{P, kP, false, 16, "P"},
                       {Nodes, kNodes, false, 16, "Nodes"},
                       {Order, kKeys, false, 4, "Order"},
                       {C, kC, false, 4, "C"},
                       {Hit, empty ? 0 : image_bytes(width, height), true, 16, "Hit"}};
  if (int s = check_bindings(name, b)) return s;
  if (empty) return ARBOR_OK;
  if (single_tree)
    trace_inorder_kernel<false><<<pixel_grid(width, height), kBlock, 0, stream>>>(P, Nodes, Order, C, world_trig(), Hit, width, height);
  else
    trace_inorder_kernel<true><<<pixel_grid(width, height), kBlock, 0, stream>>>(P, Nodes, Order, C, world_trig(), Hit, width, height);
  count_launch();
  return check_launch(name);
}
extern "C" int arbor_shadePixelsInOrder(const float* P, const float* Nodes, const uint32_t* Order, const float* C, const float* Hit,
                                        float* Linear, float* Guide, int width, int height, int single_tree, arbor_stream stream) {
  const char* name = "arbor_shadePixelsInOrder";
  bool empty;
  if (int s = check_image(name, width, height, &empty)) return s;
  size_t img = empty ? 0 : image_bytes(width, height);
  const Binding b[] = {{P, kP, false, 16, "P"},         {Nodes, kNodes, false, 16, "Nodes"}, {Order, kKeys, false, 4, "Order"},
                       {C, kC, false, 4, "C"},          {Hit, img, false, 16, "Hit"},        {Linear, img, true, 16, "Linear"},
                       {Guide, img, true, 16, "Guide"}};
  if (int s = check_bindings(name, b)) return s;
  if (empty) return ARBOR_OK;
  if (single_tree)
    shade_inorder_kernel<false><<<pixel_grid(width, height), kBlock, 0, stream>>>(P, Nodes, Order, C, world_trig(), Hit, Linear, Guide, width, height);
  else
    shade_inorder_kernel<true><<<pixel_grid(width, height), kBlock, 0, stream>>>(P, Nodes, Order, C, world_trig(), Hit, Linear, Guide, width, height);
  count_launch();
  return check_launch(name);
}
