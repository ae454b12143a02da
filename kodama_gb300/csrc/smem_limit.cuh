// The dynamic shared memory a kernel may be launched with.
#pragma once

#include <cuda_runtime.h>

namespace kgb {

// Allows a kernel all the dynamic shared memory that its static part leaves of an SM's.
// The limit belongs to the kernel, which the host threads of the process share: set to
// every launch's own size, one thread's smaller size could come between another's and
// its launch, which then failed.
template <class... Args>
inline cudaError_t allow_shared_memory(void (*kernel)(Args...)) {
  int device = 0, most = 0;
  cudaFuncAttributes own{};
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&own, kernel);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             most - static_cast<int>(own.sharedSizeBytes));
  return e;
}

}  // namespace kgb
