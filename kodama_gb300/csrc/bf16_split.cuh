// bfloat16 hi + lo split of float rows for the tensor-core distances (knn_tc.cu,
// kmeans.cu): x = hi + lo + r with |r| <= 2^-16 |x|.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace kgb {

// Round to the nearest bfloat16 (ties to even); inf / nan kept.
__device__ __forceinline__ uint32_t bf16_bits(float v) {
  const uint32_t u = __float_as_uint(v);
  if ((u & 0x7f800000u) == 0x7f800000u) return u >> 16;
  return (u + 0x7fffu + ((u >> 16) & 1u)) >> 16;
}

}  // namespace kgb
