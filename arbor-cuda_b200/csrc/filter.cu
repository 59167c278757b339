// filter.cu - filterLighting and resolvePixels (Arbor.cu:292-304), apart and
// fused, with their C-ABI entry points.
#include "abi_util.h"
#include "passes.cuh"

namespace arbor {
namespace {

// filterLighting (+ resolvePixels) of one 32x16 tile per CTA, its halo
// staged from global memory; 4 CTAs per SM.
template <bool kResolve>
__global__ void __launch_bounds__(kFX * kFT, 4) filter_kernel(const float* __restrict__ Linear, const float* __restrict__ Guide,
                                                              const float* __restrict__ Hit, float* __restrict__ Filtered,
                                                              float* __restrict__ History, uint32_t* __restrict__ Pixels,
                                                              const float* __restrict__ C, int width, int height) {
  __shared__ FilterTile s;
  filter_tile<kResolve>(s, Linear, Guide, Hit, Filtered, History, Pixels, kResolve ? C[9] : 0.0f, kResolve ? C[10] : 0.0f, C[15],
                        kResolve ? C[20] : 0.0f, width, height, blockIdx.x * kFX, blockIdx.y * kFY);
}

// resolvePixels alone (Arbor.cu:304): 32x8-pixel CTAs, one pixel per thread.
constexpr int kRX = 32, kRY = 8;
__global__ void __launch_bounds__(kRX * kRY) resolve_kernel(const float* __restrict__ Filtered, float* __restrict__ History,
                                                            uint32_t* __restrict__ Pixels, const float* __restrict__ C, int width,
                                                            int height) {
  const int x = blockIdx.x * kRX + threadIdx.x, y = blockIdx.y * kRY + threadIdx.y;
  if (x >= width || y >= height) return;
  float4 f = __ldg(reinterpret_cast<const float4*>(Filtered) + y * width + x);
  const float count = sample_count(C[9], C[10]);
  resolve_px(mk(f.x, f.y, f.z), History, Pixels, count, 1.0f / (count + 1.0f), C[20], vig_coord(x, width), vig_coord(y, height), y * width + x);
}


dim3 filter_grid(int w, int h) { return dim3((w + kFX - 1) / kFX, (h + kFY - 1) / kFY); }

// filterLighting (+ resolvePixels) over width x height: one 32x16 tile per CTA.
int launch_filter(const char* name, bool resolve, const float* Linear, const float* Guide, const float* Hit, float* Filtered, float* History,
                  uint32_t* Pixels, const float* C, int width, int height, cudaStream_t stream) {
  if (resolve)
    filter_kernel<true><<<filter_grid(width, height), dim3(kFX, kFT), 0, stream>>>(Linear, Guide, Hit, Filtered, History, Pixels, C, width, height);
  else
    filter_kernel<false><<<filter_grid(width, height), dim3(kFX, kFT), 0, stream>>>(Linear, Guide, Hit, Filtered, nullptr, nullptr, C, width,
                                                                                    height);
  count_launch();
  return check_launch(name);
}
dim3 resolve_grid(int w, int h) { return dim3((w + kRX - 1) / kRX, (h + kRY - 1) / kRY); }

}  // namespace
}  // namespace arbor

using namespace arbor;

extern "C" int arbor_filterLighting(const float* Linear, const float* Guide, const float* Hit, float* Filtered, const float* C, int width,
                                    int height, arbor_stream stream) {
  const char* name = "arbor_filterLighting";
  bool empty;
  if (int s = check_image(name, width, height, &empty)) return s;
  size_t img = empty ? 0 : image_bytes(width, height);
  const Binding b[] = {{Linear, img, false, 16, "Linear"},
                       {Guide, img, false, 16, "Guide"},
                       {Hit, img, false, 16, "Hit"},
                       {Filtered, img, true, 16, "Filtered"},
                       {C, kC, false, 4, "C"}};
  if (int s = check_bindings(name, b)) return s;
  if (empty) return ARBOR_OK;
  return launch_filter(name, false, Linear, Guide, Hit, Filtered, nullptr, nullptr, C, width, height, stream);
}
extern "C" int arbor_resolvePixels(const float* Filtered, float* History, uint32_t* Pixels, const float* C, int width, int height,
                                   arbor_stream stream) {
  const char* name = "arbor_resolvePixels";
  bool empty;
  if (int s = check_image(name, width, height, &empty)) return s;
  size_t img = empty ? 0 : image_bytes(width, height);
  const Binding b[] = {{Filtered, img, false, 16, "Filtered"},
                       {History, img, true, 16, "History"},
                       {Pixels, empty ? 0 : pixel_bytes(width, height), true, 4, "Pixels"},
                       {C, kC, false, 4, "C"}};
  if (int s = check_bindings(name, b)) return s;
  if (empty) return ARBOR_OK;
  resolve_kernel<<<resolve_grid(width, height), dim3(kRX, kRY), 0, stream>>>(Filtered, History, Pixels, C, width, height);
  count_launch();
  return check_launch(name);
}
extern "C" int arbor_filterResolve(const float* Linear, const float* Guide, const float* Hit, float* Filtered, float* History, uint32_t* Pixels,
                                   const float* C, int width, int height, arbor_stream stream) {
  const char* name = "arbor_filterResolve";
  bool empty;
  if (int s = check_image(name, width, height, &empty)) return s;
  size_t img = empty ? 0 : image_bytes(width, height);
  const Binding b[] = {{Linear, img, false, 16, "Linear"},     {Guide, img, false, 16, "Guide"},
                       {Hit, img, false, 16, "Hit"},           {Filtered, img, true, 16, "Filtered"},
                       {History, img, true, 16, "History"},    {Pixels, empty ? 0 : pixel_bytes(width, height), true, 4, "Pixels"},
                       {C, kC, false, 4, "C"}};
  if (int s = check_bindings(name, b)) return s;
  if (empty) return ARBOR_OK;
  return launch_filter(name, true, Linear, Guide, Hit, Filtered, History, Pixels, C, width, height, stream);
}

