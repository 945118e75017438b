// Dynamic shared memory above 48 KB, which a kernel is granted per device.
#pragma once
#include <mutex>
#include <set>
#include <utility>

#include "common.cuh"

namespace drg {

// Lets launches of `kernel` on the current device use up to `bytes`, the most
// that any launch of it asks for.  Asked for once per kernel and device;
// contexts on several devices and host threads call it at the same time.
inline void allow_smem(const void* kernel, size_t bytes) {
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> allowed;
  int device = 0;
  DRG_CUDA(cudaGetDevice(&device));
  std::lock_guard<std::mutex> lock(mu);
  if (allowed.count({device, kernel})) return;
  DRG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  allowed.insert({device, kernel});
}

}  // namespace drg
