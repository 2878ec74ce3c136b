// Opt-in to more dynamic shared memory than 48 KB: an attribute of a kernel on one device.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#include <atomic>

namespace ds {

// Lets `kernel` use `bytes` of dynamic shared memory on the current device, asked for
// once per device and kernel (`done`: the kernel's devices, of the first 64).
template <class K>
inline cudaError_t allow_smem(K* kernel, size_t bytes, std::atomic<uint64_t>& done) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && (done.load() >> dev & 1u)) return cudaSuccess;
  e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)bytes);
  if (e == cudaSuccess && dev < 64) done.fetch_or(1ull << dev);
  return e;
}

}  // namespace ds
