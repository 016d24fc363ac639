// What a launcher finds out once about its kernel on a device: attributes of a
// kernel (its limit of dynamic shared memory) belong to the device that was
// current when they were set, and so does what the occupancy calls say.
#pragma once

#include <cuda_runtime.h>

#include <array>
#include <atomic>
#include <string>

namespace qfx {

class PerDevice {
 public:
  // The positive number that `find` gives for the current device, kept from
  // the first call there on (`find` may run twice where threads meet).
  template <typename F>
  int operator()(F&& find) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= (int)known_.size()) return find();
    const int v = known_[dev].load(std::memory_order_acquire);
    if (v > 0) return v;
    const int found = find();
    known_[dev].store(found, std::memory_order_release);
    return found;
  }

 private:
  std::array<std::atomic<int>, 64> known_{};
};

// Raises a kernel's limit of dynamic shared memory on the current device.
template <typename K>
void raise_smem_limit(K* kernel, int bytes) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess)
    throw std::string("ERROR (qflex_gb300: CUDA cudaFuncSetAttribute) --> ") + cudaGetErrorString(e);
}

}  // namespace qfx
