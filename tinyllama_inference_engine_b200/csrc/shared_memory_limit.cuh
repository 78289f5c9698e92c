// A kernel that takes more than 48 KB of dynamic shared memory has to be told so, on every device that it runs on: the attribute belongs to the device
// that is current when it is set.
#pragma once

#include <atomic>

#include <cuda_runtime.h>

namespace tlie {

// Sets it once per device.  `devices`: a bit per device that has it, one such word per kernel.
template <typename Kernel>
static inline cudaError_t allow_shared_memory(Kernel* kernel, int bytes, std::atomic<unsigned long long>& devices) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;   // (beyond those it is set every time)
  if (devices.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) devices.fetch_or(bit, std::memory_order_release);
  return e;
}

}  // namespace tlie
