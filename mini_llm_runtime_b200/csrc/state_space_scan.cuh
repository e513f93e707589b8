// The state-space recurrence of a segment, token by token in a fixed order (see state_space.cu): a kernel of its own there, and beside
// the chunks of longer segments in state_space_chunks.cu.
#pragma once

#include "common.cuh"
#include "copy_async.cuh"

namespace mlr {

constexpr int SCAN_NPT = 16;        // state entries of one value channel a thread holds
constexpr int SCAN_TOKENS = 32;     // tokens staged at once, at most
constexpr int SCAN_THREADS = 128;

struct ScanArgs {
  const float *x, *B, *C, *dt_raw;
  long long x_stride, b_stride, c_stride, dt_stride;
  const float *dt_bias, *A_log, *D;
  float* states;
  float* y;
  const int *seg_q_start, *seg_q_len, *seg_slot;
  int heads, vdim, n, groups;
  int longest;      // segments of more rows are another kernel's
};

// SL: threads that share one value channel's state (a power of two; SL * SCAN_NPT >= n).  Lane l of a warp
// holds 16 entries of channel p = l / SL: the pieces of four entries number s, s + SL, s + 2 SL, s + 3 SL with
// s = l % SL (neighbouring threads read neighbouring 16-byte pieces of a staged row: no bank conflicts; with
// 16 entries in a row per thread a quarter warp's reads fell into two banks).
// A block takes a segment, a head and a block of value channels.  The inputs of 32 tokens at a time are staged in shared
// memory by asynchronous copies, the next 32 while these are walked; WIDE: in 16-byte pieces (state size,
// channel block and all row strides multiples of four floats, pointers aligned).
enum ScanPart { ALL_ROWS, FIRST_HALF, SECOND_HALF };      // of a segment's rows, the second behind the first in a later kernel
template <int SL, bool WIDE, int TOKENS = SCAN_TOKENS>
__device__ __forceinline__ void scan_segment(const ScanArgs& a, float* shared, int seg, int head, int part, ScanPart which_rows = ALL_ROWS) {
  constexpr int P_CTA = SCAN_THREADS / SL;
  const int N = a.n, P = a.vdim;
  const int buffer = TOKENS * (2 * N + P_CTA + 1);      // floats of one staging buffer
  float* decay = shared + 2 * buffer + SCAN_NPT;             // [TOKENS]; a last piece may reach past a buffer's end
  float* step = decay + TOKENS;                         // [TOKENS]
  const int group = head / (a.heads / a.groups);
  const int s = threadIdx.x % SL, p_local = threadIdx.x / SL;
  const int p = part * P_CTA + p_local;
  const float rate = expf(a.A_log[head]), bias = a.dt_bias[head], skip = a.D[head];
  pdl_wait();
  const int q_start = a.seg_q_start[seg], all_rows = a.seg_q_len[seg];
  if (all_rows > a.longest) return;
  const int half = (all_rows + 2 * TOKENS - 1) / (2 * TOKENS) * TOKENS;
  const int begin = which_rows == SECOND_HALF ? half : 0, q_len = which_rows == FIRST_HALF ? min(half, all_rows) : all_rows;
  if (which_rows == SECOND_HALF && begin >= q_len) return;

  // rows [t0, t0 + 32) of the segment into buffer `which`: B and C of the head's group, the block's value
  // channels of x, the head's raw step sizes
  auto stage = [&](int t0, int which) {
    float* b_rows = shared + which * buffer;
    float* c_rows = b_rows + TOKENS * N;
    float* x_rows = c_rows + TOKENS * N;
    float* raw = x_rows + TOKENS * P_CTA;
    const int tokens = min(TOKENS, q_len - t0);
    const size_t row0 = (size_t)(q_start + t0);
    if (WIDE) {
      const int per_row = N >> 2;
      for (int idx = threadIdx.x; idx < tokens * per_row; idx += SCAN_THREADS) {
        const int t = idx / per_row, n = (idx - t * per_row) << 2;
        copy_async_16(b_rows + t * N + n, a.B + (row0 + t) * a.b_stride + (size_t)group * N + n);
        copy_async_16(c_rows + t * N + n, a.C + (row0 + t) * a.c_stride + (size_t)group * N + n);
      }
      constexpr int X_PIECES = P_CTA / 4;
      for (int idx = threadIdx.x; idx < tokens * X_PIECES; idx += SCAN_THREADS) {
        const int t = idx / X_PIECES, pl = (idx - t * X_PIECES) << 2;
        const int pp = part * P_CTA + pl;
        if (pp < P) copy_async_16(x_rows + t * P_CTA + pl, a.x + (row0 + t) * a.x_stride + (size_t)head * P + pp);
      }
    } else {
      for (int idx = threadIdx.x; idx < tokens * N; idx += SCAN_THREADS) {
        const int t = idx / N, n = idx - t * N;
        copy_async_4(b_rows + idx, a.B + (row0 + t) * a.b_stride + (size_t)group * N + n);
        copy_async_4(c_rows + idx, a.C + (row0 + t) * a.c_stride + (size_t)group * N + n);
      }
      for (int idx = threadIdx.x; idx < tokens * P_CTA; idx += SCAN_THREADS) {
        const int t = idx / P_CTA, pl = idx - t * P_CTA;
        const int pp = part * P_CTA + pl;
        if (pp < P) copy_async_4(x_rows + idx, a.x + (row0 + t) * a.x_stride + (size_t)head * P + pp);
      }
    }
    if (threadIdx.x < tokens) copy_async_4(raw + threadIdx.x, a.dt_raw + (row0 + threadIdx.x) * a.dt_stride + head);
    copy_async_commit();
  };

  stage(begin, 0);
  float* state = a.states + (((size_t)a.seg_slot[seg] * a.heads + head) * P + (p < P ? p : 0)) * N;
  auto entry = [&](int i) { return (((i >> 2) * SL + s) << 2) + (i & 3); };      // the state entry a thread's i-th number is
  float S[SCAN_NPT];
#pragma unroll
  for (int i = 0; i < SCAN_NPT; ++i) {
    const int n = entry(i);
    S[i] = (p < P && n < N) ? state[n] : 0.f;
  }
  int which = 0;
  for (int t0 = begin; t0 < q_len; t0 += TOKENS, which ^= 1) {
    const int tokens = min(TOKENS, q_len - t0);
    const bool more = t0 + TOKENS < q_len;
    if (more) stage(t0 + TOKENS, which ^ 1);
    if (more) copy_async_wait<1>(); else copy_async_wait<0>();
    __syncthreads();
    const float* b_rows = shared + which * buffer;
    const float* c_rows = b_rows + TOKENS * N;
    const float* x_rows = c_rows + TOKENS * N;
    const float* raw = x_rows + TOKENS * P_CTA;
    if (threadIdx.x < tokens) {
      const float z = raw[threadIdx.x] + bias;
      const float dt = z > 20.f ? z : log1pf(expf(z));
      step[threadIdx.x] = dt;
      decay[threadIdx.x] = expf(-rate * dt);
    }
    __syncthreads();
    // two tokens in flight: the second one's reads and products run under the first one's sums and shuffles
#pragma unroll 2
    for (int t = 0; t < tokens; ++t) {
      const float av = decay[t], xv = p < P ? x_rows[t * P_CTA + p_local] : 0.f;
      const float dx = step[t] * xv;
      const float* bt = b_rows + t * N;
      const float* ct = c_rows + t * N;
      float bv[SCAN_NPT], cv[SCAN_NPT];
      if (WIDE) {
#pragma unroll
        for (int i = 0; i < SCAN_NPT; i += 4) {
          const float4 b4 = *reinterpret_cast<const float4*>(bt + entry(i)), c4 = *reinterpret_cast<const float4*>(ct + entry(i));
          bv[i] = b4.x; bv[i + 1] = b4.y; bv[i + 2] = b4.z; bv[i + 3] = b4.w;
          cv[i] = c4.x; cv[i + 1] = c4.y; cv[i + 2] = c4.z; cv[i + 3] = c4.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < SCAN_NPT; ++i) {
          const bool in = entry(i) < N;
          bv[i] = in ? bt[entry(i)] : 0.f;
          cv[i] = in ? ct[entry(i)] : 0.f;
        }
      }
      float sums[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < SCAN_NPT; ++i) {
        if (entry(i) < N) {
          S[i] = fmaf(av, S[i], bv[i] * dx);
          sums[i & 3] = fmaf(S[i], cv[i], sums[i & 3]);
        }
      }
      float sum = (sums[0] + sums[1]) + (sums[2] + sums[3]);
#pragma unroll
      for (int offset = SL / 2; offset > 0; offset >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, offset);
      if (s == 0 && p < P) a.y[(size_t)(q_start + t0 + t) * a.heads * P + (size_t)head * P + p] = fmaf(skip, xv, sum);
    }
    __syncthreads();      // the next turn of the loop stages into this buffer
  }
  if (p < P) {
#pragma unroll
    for (int i = 0; i < SCAN_NPT; ++i) {
      const int n = entry(i);
      if (n < N) state[n] = S[i];
    }
  }
}

// Shared memory of a block in bytes.
inline size_t scan_shared(int n, int channels, int tokens = SCAN_TOKENS) {
  return sizeof(float) * (2 * (size_t)tokens * (2 * n + channels + 1) + SCAN_NPT + 2 * tokens);
}

}  // namespace mlr
