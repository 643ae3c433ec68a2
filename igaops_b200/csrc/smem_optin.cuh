// Opt-in of a kernel to more than 48 KB of dynamic shared memory.
//
// cudaFuncSetAttribute acts on the current device, so what was done is kept per
// device, and the kernel gets its device's whole limit: the calls of two threads with
// different sizes set the same value, and no later size needs another call. (Plain C++:
// tests/test_smem_optin_cpu.py compiles it against a fake runtime of two devices.)
#pragma once

#include <cuda_runtime_api.h>
#include <stdint.h>

#include <atomic>

namespace iga {

class SmemOptIn {  // one static object per kernel
 public:
  cudaError_t allow(const void* kernel, size_t smem) {
    if (smem <= 48 * 1024) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? uint64_t(1) << dev : 0;  // further devices: set on every call
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    int most = 0;
    if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) !=
        cudaSuccess)
      return e;
    cudaFuncAttributes attr;
    if ((e = cudaFuncGetAttributes(&attr, kernel)) != cudaSuccess) return e;
    most -= (int)attr.sharedSizeBytes;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most)) !=
        cudaSuccess)
      return e;
    done_.fetch_or(bit, std::memory_order_release);
    return cudaSuccess;
  }

 private:
  std::atomic<uint64_t> done_{0};  // a bit per device
};

}  // namespace iga
