// Float32 numbers as sums of three bfloat16 numbers, for products on the tensor cores.
#pragma once

#include "common.cuh"

namespace mlr {

// Two neighbours' next bfloat16 part, taken off them.  Three in turn hold all 24 bits: 8 each, and the remainder of a rounding is exact.
__device__ __forceinline__ uint32_t take_part(float& a, float& b) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(a, b);
  const uint32_t bits = *reinterpret_cast<const uint32_t*>(&pair);
  a -= __uint_as_float(bits << 16);
  b -= __uint_as_float(bits & 0xffff0000u);
  return bits;
}

}  // namespace mlr
