// What a kernel is allowed belongs to the device that is current when it is said: a process with several of them says it once on
// each.  Only runtime calls, so that it can be run on the host with others in their place.
#pragma once
#include <cuda_runtime_api.h>
#include <stddef.h>

#include <atomic>

struct CbDeviceAttr {
  std::atomic<unsigned long long> done{0};       // bit d: said on device d; devices from 64 on are told every time
};

// dynamic shared memory of `kernel` on the current device, more than the 48 KB that need no word; `carveout`: and all of an SM's for it
template <typename K> int cb_allow_smem(CbDeviceAttr& attr, K* kernel, size_t bytes, bool carveout = false) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  const unsigned long long bit = device < 64 ? 1ull << device : 0;
  if (attr.done.load(std::memory_order_acquire) & bit) return 0;
  const void* f = reinterpret_cast<const void*>(kernel);
  if (bytes > 48 * 1024) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && carveout)
    e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) attr.done.fetch_or(bit, std::memory_order_release);
  return (int)e;
}
