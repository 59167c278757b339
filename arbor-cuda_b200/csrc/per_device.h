// per_device.h - facts about a device that are found once per process.
#pragma once
#include <atomic>

namespace arbor {

// A positive int per device.  Threads that ask first each run `find`, which
// must give the same answer to all; what is not positive is not kept, so a
// failure is met again by the next call.
class PerDevice {
  static constexpr int kDevices = 64;
  std::atomic<int> value_[kDevices] = {};

 public:
  template <class F>
  int get(int device, F find) {
    const bool kept = device >= 0 && device < kDevices;
    int v = kept ? value_[device].load(std::memory_order_acquire) : 0;
    if (v > 0) return v;
    v = find();
    if (kept && v > 0) value_[device].store(v, std::memory_order_release);
    return v;
  }
};

}  // namespace arbor

#ifdef __CUDACC__
#include <cuda_runtime.h>

namespace arbor {

// -1: no current device.
inline int current_device() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}
// Multiprocessors of the current device (148 when it cannot be asked).
inline int device_sms() {
  static PerDevice sms;
  const int dev = current_device();
  const int n = sms.get(dev, [&] {
    int v = 0;
    return cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? v : 0;
  });
  return n > 0 ? n : 148;
}
// Opts `Kernel` in to `bytes` of dynamic shared memory on the current device
// (the attribute is the device's).  A kernel is always asked for with the same
// size.
template <auto Kernel>
inline bool smem_opt_in(int bytes) {
  static PerDevice done;
  return done.get(current_device(), [&] {
    return cudaFuncSetAttribute(reinterpret_cast<const void*>(Kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? 1 : 0;
  }) > 0;
}

}  // namespace arbor
#endif
