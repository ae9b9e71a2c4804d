// The dynamic shared-memory limit of a kernel.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>

namespace hhg {

// Lets `kern` be launched with `bytes` of dynamic shared memory on the current device; false, and no error left, if
// the device refuses.  The limit is one value per function and device and a launch above it fails, while an instance
// may serve solves of several sizes from several host threads: so it is only ever raised.  It is read back on each call,
// as it goes with the context.
template <typename Kernel>
bool allow_shared_memory(Kernel kern, size_t bytes) {
  static std::mutex mu;  // (one per kernel type: between reading the limit and raising it)
  std::lock_guard<std::mutex> lock(mu);
  const void* f = reinterpret_cast<const void*>(kern);
  cudaFuncAttributes a{};
  bool ok = cudaFuncGetAttributes(&a, f) == cudaSuccess;
  if (ok && (size_t)a.maxDynamicSharedSizeBytes < bytes)
    ok = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
  if (!ok) cudaGetLastError();
  return ok;
}

}  // namespace hhg
