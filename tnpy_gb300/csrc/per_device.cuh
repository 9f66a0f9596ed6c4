// One-time setup of a kernel, per device.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace tnx {

// Devices on which an idempotent setup has been made; threads may race to it. Devices beyond the 64 that fit are set up
// each time.
class DeviceSet {
  std::atomic<unsigned long long> bits_{0};

 public:
  bool has(int dev) const { return dev >= 0 && dev < 64 && ((bits_.load(std::memory_order_acquire) >> dev) & 1) != 0; }
  void add(int dev) {
    if (dev >= 0 && dev < 64) bits_.fetch_or(1ull << dev, std::memory_order_release);
  }
};

// Lets `kernel` use up to `most` bytes of dynamic shared memory on the current device: the attribute is the device's, and
// has to be the largest that any call needs, since another thread may launch between a call's setting and its launch.
template <typename K>
cudaError_t allow_smem(K kernel, size_t most, DeviceSet& done) {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess || done.has(dev)) return err;
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most));
  if (err == cudaSuccess) done.add(dev);
  return err;
}

}  // namespace tnx
