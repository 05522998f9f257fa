// smem_limit.h -- the dynamic shared-memory limit of a kernel, set so that concurrent callers
// cannot take it from one another.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace ghc {

// Dynamic shared memory that one CTA of the current device may have (227 KB on B200); 0: no device.
inline size_t cta_smem_limit() {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || v <= 0)
    return 0;
  return (size_t)v;
}

// Lets Kernel's launches on the current device use up to cta_smem_limit() bytes; false: refused.
// cudaFuncAttributeMaxDynamicSharedMemorySize belongs to the kernel, not to a launch: a caller that
// set it to its own size before each launch could lower it between another thread's set and launch,
// whose launch is then refused (and a limit that is only raised can still be lowered so, between two
// threads that both found it too low).  Every caller sets the same value here, once per kernel and
// device, so the order does not matter and later launches spare the call.
template <auto Kernel>
bool allow_smem() {
  constexpr int kDevs = 64;
  static std::atomic<bool> allowed[kDevs];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (dev < kDevs && allowed[dev].load(std::memory_order_acquire)) return true;
  const size_t limit = cta_smem_limit();
  if (limit == 0 ||
      cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit) != cudaSuccess)
    return false;
  if (dev < kDevs) allowed[dev].store(true, std::memory_order_release);
  return true;
}

}  // namespace ghc
