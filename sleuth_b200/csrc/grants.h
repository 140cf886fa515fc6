// Dynamic shared memory above 48 KB has to be allowed for a kernel, once on every device that runs it.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>

namespace slb {

// Lets `kernel` have `bytes` of dynamic shared memory on the current device; `done`, one word a kernel, remembers by bit the devices
// where it may. Host threads may race: the worst is that a device is asked twice for the same. Every launcher goes through here: a
// flag of a launcher's own would remember a process, and the kernel could be launched on the first device only.
inline cudaError_t allow_shared(const void* kernel, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;      // (a device beyond is asked every time)
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

}  // namespace slb
