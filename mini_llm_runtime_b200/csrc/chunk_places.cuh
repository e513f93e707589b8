// Chunks of a segment's tokens that a recurrence takes side by side, and where they keep their states.
#pragma once

#include "common.cuh"

namespace mlr {

constexpr int CHUNK = 64;      // tokens of a chunk; chunks start at a segment's first row

// Where a chunk that starts at `row` keeps its state: one place per aligned run of CHUNK rows for a segment's first
// chunk and one for another chunk.  Among segments of several chunks (the only ones with places) no two chunks share one: a
// second first chunk in the run would start more than CHUNK rows after the first, and so would a second later chunk.
__device__ __forceinline__ size_t chunk_place(int row, bool first) { return 2 * (size_t)(row / CHUNK) + (first ? 1 : 0); }

inline long long chunk_places(int rows) { return 2ll * (rows / CHUNK + 1); }

template <int C>
__device__ __forceinline__ void load_columns(float (&v)[C], const float* src) {
  if constexpr (C == 2) {
    const float2 q = *reinterpret_cast<const float2*>(src);
    v[0] = q.x, v[1] = q.y;
  } else {
    const float4 q = *reinterpret_cast<const float4*>(src);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  }
}
template <int C>
__device__ __forceinline__ void store_columns(float* dst, const float (&v)[C]) {
  if constexpr (C == 2)
    *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[1]);
  else
    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
}

}  // namespace mlr
