// Products of 32-bit numbers by mma.sync, operands in three bfloat16 parts, six of the nine products of parts (the rest is below 2^-26).
#pragma once

#include "float_parts.cuh"
#include "mma_attention.cuh"

namespace mlr {

// The three parts of a 16 x 16 left operand whose numbers lie as two neighbouring accumulators do.
__device__ __forceinline__ void split_operand(uint32_t (&parts)[3][4], const float (&left)[4], const float (&right)[4]) {
  float v[8] = {left[0], left[1], left[2], left[3], right[0], right[1], right[2], right[3]};
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i) parts[q][i] = take_part(v[2 * i], v[2 * i + 1]);
}

// lead += x0 w0, low += the five smaller products, of 2 * PAIRS neighbouring accumulators, of which the pairs from `begin` on.  from: this
// lane's ldmatrix address in part 0 of the first pair, `step` entries on the next one's.  Product by product over all accumulators: an
// MMA's result is 35 cycles away, the next MMA 8.
template <bool TRANS, int PAIRS>
__device__ __forceinline__ void add_products(float (&lead)[2 * PAIRS][4], float (&low)[2 * PAIRS][4], const uint32_t (&x)[3][4], const bf16* from,
                                             int step, int apart, int begin = 0, int end = PAIRS) {
#pragma unroll
  for (int q = 2; q >= 0; --q) {
    uint32_t w[PAIRS][4];
#pragma unroll
    for (int j = 0; j < PAIRS; ++j)
      if (j >= begin && j < end) {
        if (TRANS) ldmatrix_x4_trans(w[j], from + j * step + q * apart); else ldmatrix_x4(w[j], from + j * step + q * apart);
      }
#pragma unroll
    for (int i = 2 - q; i >= 0; --i)
#pragma unroll
      for (int j = 0; j < PAIRS; ++j)
        if (j >= begin && j < end) {
          mma_bf16(i + q == 0 ? lead[2 * j] : low[2 * j], x[i], w[j][0], w[j][1]);
          mma_bf16(i + q == 0 ? lead[2 * j + 1] : low[2 * j + 1], x[i], w[j][2], w[j][3]);
        }
  }
}
// A tensor core's sum is cut off, not rounded, at every step.  What that took from `lead` is given back on average, as `share` halves of the last
// place's unit (found by errors against 64 bits), with the sum of the small products.
__device__ __forceinline__ float with_dropped(float lead, float low, float share) {
  return fmaf(__uint_as_float(__float_as_uint(lead) & 0xff800000u), share * 5.9604644775390625e-8f, low);      // its sign and power of two
}
template <int N>
__device__ __forceinline__ void clear(float (&x)[N][4]) {
#pragma unroll
  for (int j = 0; j < N; ++j) x[j][0] = x[j][1] = x[j][2] = x[j][3] = 0.f;
}

}  // namespace mlr
