// Settings of a kernel that the runtime keeps per device (a function's shared-memory limit): made once for every device
// the process launches it on.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <stdint.h>

namespace dfccl {

// `f` (its own type per place of use) is called with the current device until it has succeeded there once.
template <typename F>
cudaError_t oncePerDevice(F f) {
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = f();                                               // (two threads may both get here: the setting is the same)
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

// Raises the dynamic shared memory a kernel may be launched with.
template <typename K>
cudaError_t allowSharedMemory(K kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); }

}  // namespace dfccl
