// What a process finds out or sets once per device.
#pragma once
#include <cuda_runtime.h>
#include <atomic>

#define TL_DEVICES 64

// The current device's number, or -1 where nothing can be kept for it.
static inline int tl_device() {
  int d = -1;
  return cudaGetDevice(&d) == cudaSuccess && d >= 0 && d < TL_DEVICES ? d : -1;
}

// Lets KERNEL have `bytes` of dynamic shared memory on the current device.  The limit belongs to the device's context, so a
// process that has set it on one device has not on the next.
template <auto KERNEL>
static cudaError_t tl_allow_smem(int bytes) {
  static std::atomic<unsigned long long> done{0};    // bit d: set on device d
  const int d = tl_device();
  if (d >= 0 && (done.load(std::memory_order_acquire) >> d & 1ull)) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute((const void*)KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && d >= 0) done.fetch_or(1ull << d, std::memory_order_release);
  return e;
}
