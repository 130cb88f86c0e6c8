// sgh_limits.h -- launch limits of kernels that need more than the default.
//
// The dynamic shared-memory limit and the permission for clusters of 16 CTAs
// belong to a kernel (per device), not to a launch: any host thread that lowers a limit
// can make another thread's launch of the same kernel fail, and a limit raised
// on one device says nothing about the next. kernel_limits() therefore only ever
// raises them, once per kernel, device and size, under a lock, and every launch
// calls it first. Callers pass the largest size that the kernel is ever launched
// with, so that the one call to the runtime precedes every launch of the kernel on
// that device and none runs beside it. What a host thread has seen raised it finds
// in a table of its own, without the lock.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#include <map>
#include <mutex>
#include <utility>

namespace sgh {

struct KernelLimits {
  std::mutex lock;
  std::map<std::pair<const void*, int>, std::pair<int, bool>> seen;  // (kernel, device) -> (bytes, 16 CTAs)
};
inline KernelLimits& kernel_limits_table() {
  static KernelLimits* t = new KernelLimits;  // never destroyed: launches may run during exit
  return *t;
}

inline cudaError_t kernel_limits(const void* kernel, int bytes, bool wide_clusters = false) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  struct Own {
    const void* kernel;
    int dev, bytes;
    bool wide;
  };
  static thread_local Own own[64];
  Own& o = own[(reinterpret_cast<uintptr_t>(kernel) >> 4) % 64];
  if (o.kernel == kernel && o.dev == dev && bytes <= o.bytes && (o.wide || !wide_clusters)) return cudaSuccess;
  KernelLimits& t = kernel_limits_table();
  std::lock_guard<std::mutex> hold(t.lock);
  auto& s = t.seen[{kernel, dev}];
  if (bytes > s.first) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    s.first = bytes;
  }
  if (wide_clusters && !s.second) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    s.second = true;
  }
  o = {kernel, dev, s.first, s.second};
  return cudaSuccess;
}

}  // namespace sgh
