// The dynamic shared-memory limit of a kernel whose launches differ in size.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace hfg {

// Raises Kern's limit to the most a block may use on the current device, once
// per device.  The limit belongs to the function, not to the launch: contexts
// on several threads share it, so a launch that set it to its own size could
// lower it between another's setting and launch, which then fails.
template <auto Kern>
cudaError_t raise_smem_limit() {
  constexpr int kMaxDev = 64;
  static std::atomic<bool> raised[kMaxDev];
  int dev = 0, most = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool known = dev >= 0 && dev < kMaxDev;
  if (known && raised[dev].load(std::memory_order_acquire)) return cudaSuccess;
  cudaFuncAttributes fa{};
  if ((e = cudaFuncGetAttributes(&fa, Kern)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  e = cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes);
  if (e == cudaSuccess && known) raised[dev].store(true, std::memory_order_release);
  return e;
}

}  // namespace hfg
