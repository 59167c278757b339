// scratch.cu - the library's scratch pool (scratch.h).
#include "scratch.h"

#include <mutex>

namespace arbor {
namespace {

constexpr int kMaxDevices = 64;

// While one lives, this thread's allocations do not disturb a capture that
// another thread has begun in the global mode (torch's default): a pool that
// has to grow would invalidate it.
struct OtherCaptures {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  OtherCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~OtherCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};

// The current device's pool; null when it cannot be made.
cudaMemPool_t scratch_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mu);
  if (g_pool[dev] != nullptr) return g_pool[dev];
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  uint64_t keep = kScratchKeep;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    pool = nullptr;
  } else if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
    cudaGetLastError();
    cudaMemPoolDestroy(pool);
    pool = nullptr;
  }
  g_pool[dev] = pool;
  return pool;
}

}  // namespace

TightScratch::TightScratch(const float* P, const uint32_t* Order, const float* Nodes, int n_scenes, const float* C, bool shadows, cudaStream_t s)
    : stream(s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (cs != cudaStreamCaptureStatusNone || n_scenes > kTightMaxScenes) return;
  const OtherCaptures undisturbed;
  const cudaMemPool_t pool = scratch_pool();
  void* p = nullptr;
  if (pool == nullptr || cudaMallocFromPoolAsync(&p, tight_bytes(n_scenes), pool, stream) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  boxes = static_cast<uint32_t*>(p);
  status = launch_tight(P, Order, Nodes, n_scenes, boxes, C, shadows, stream);
}

TightScratch::~TightScratch() {
  if (boxes == nullptr) return;
  const OtherCaptures undisturbed;
  if (cudaFreeAsync(boxes, stream) != cudaSuccess) cudaGetLastError();
}

}  // namespace arbor
