// Host: kernel attributes, which belong to a kernel on one device.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace pb {

constexpr int kMaxDevices = 64;

// Allows `kKernel` to be launched with `kBytes` of dynamic shared memory on the current device.  Asked of the runtime once
// per kernel and device; two threads that come first together ask twice, with the same value.
template <auto kKernel, int kBytes>
cudaError_t allow_smem() {
  static std::atomic<bool> allowed[kMaxDevices];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool known = dev >= 0 && dev < kMaxDevices;
  if (known && allowed[dev].load(std::memory_order_relaxed)) return cudaSuccess;
  e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kKernel), cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e == cudaSuccess && known) allowed[dev].store(true, std::memory_order_relaxed);
  return e;
}

}  // namespace pb
