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

// A step's long segments, those of `least` rows and more, and their chunks are numbered through; a grid has an entry for each number there
// can be.  (An entry per segment and chunk of the longest segment would mostly be empty: 97 % of them with a portion of 4,000 rows
// beside 31 decoded ones.)
struct ChunkAt {
  int seg, chunk, length, start, slot;      // seg < 0: the step has no such chunk; start: the segment's first row
};

// The long segment (CHUNKS: the chunk of a long segment, where segments below `split` rows are one chunk) of number `index`; every warp
// that asks does so as a whole.
template <bool CHUNKS>
__device__ __forceinline__ ChunkAt chunk_at(const int* seg_q_start, const int* seg_q_len, const int* seg_slot, int segments, int least,
                                            int index, int split = 0) {
  const int lane = threadIdx.x & 31;
  for (int base = 0; base < segments; base += 32) {
    const bool in = base + lane < segments;      // all three asked for together: one trip to memory
    const int length = in ? seg_q_len[base + lane] : 0, start = in ? seg_q_start[base + lane] : 0, slot = in ? seg_slot[base + lane] : 0;
    const int own = length < least || length <= 0 ? 0 : CHUNKS && length >= split ? (length + CHUNK - 1) / CHUNK : 1;
    int upto = own;
    if (segments > 1) {
#pragma unroll
      for (int offset = 1; offset < 32; offset <<= 1) {
        const int before = __shfl_up_sync(0xffffffffu, upto, offset);
        if (lane >= offset) upto += before;
      }
    }
    const unsigned behind = __ballot_sync(0xffffffffu, index < upto);
    if (behind != 0) {
      const int at = __ffs(behind) - 1;
      return {base + at, index - __shfl_sync(0xffffffffu, upto - own, at), __shfl_sync(0xffffffffu, length, at),
              __shfl_sync(0xffffffffu, start, at), __shfl_sync(0xffffffffu, slot, at)};
    }
    index -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return {-1, 0, 0, 0, 0};
}

inline long long long_segments(int rows, int segments, int least) {
  const int most = rows / (least > 1 ? least : 1);
  return segments < most ? segments : most;
}
inline long long long_chunks(int rows, int segments, int least) {
  return segments == 1 ? (rows + CHUNK - 1) / CHUNK : rows / CHUNK + long_segments(rows, segments, least);
}

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
