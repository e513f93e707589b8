// The state-space recurrence (see state_space.cu) of steps with long segments, in chunks of 64 tokens side by side.
//
// With one decay g per head and token, a chunk's outputs are a masked product of its tokens plus a read of the state before it,
//   y_t = sum_{s <= t} (prod_{s < u <= t} g_u) (C_t . B_s) dt_s x_s + (prod_{u <= t} g_u) S^T C_t + D x_t,
// and its end state is the decays' product times S plus sum_s (prod_{u > s} g_u) B_s (dt_s x_s)^T.  Four kernels:
//   pairs    C_t . B_s of a chunk, once for all heads of a group
//   local    per head and chunk: the masked product and what the chunk's own tokens leave behind; a segment's first chunk
//            also reads the request's state; blocks of its own take the step's shorter segments token by token (portions of 1,531, 77, 1
//            and 439 rows, 32 heads: 139 us with all in chunks, 153 with a launch for the shorter ones, 127 so)
//   carry    per state entry, the chunks of a segment in order
//   read     per head and later chunk: the read of the state before it, added to the outputs
// All 32-bit multiply-adds.  Decay products are products of numbers up to one, formed step by step, never differences of
// logarithms (whose sums grow large while the differences stay small) nor quotients, so decays may be zero.
//
// Token by token a block per (request, head) took 0.2 us per token whatever the width: a chain.  In chunks the step is bound by
// its multiply-adds, 2 vdim n + (vdim + n / heads of a group) * 32 per token and head, fed from shared memory.  2,048 tokens of one
// request, B200: 424 -> 63 us (14 heads, states of 64), 639 -> 124 (32 heads, states of 128).
#include "chunk_places.cuh"
#include "copy_async.cuh"
#include "state_space_scan.cuh"

namespace mlr {

constexpr int VD = 64;              // value channels of a head
constexpr int W_PITCH = CHUNK + 4;  // rows of the chunk's token-by-token weights

struct SpaceArgs {
  const float *x, *B, *C, *dt_raw;
  long long x_stride, b_stride, c_stride, dt_stride;
  const float *dt_bias, *A_log, *D;
  float* states;                     // [slots, heads, VD, n]
  float* y;                          // [rows, heads * VD]
  float* pairs;                      // [rows, groups, CHUNK]: C of the row against B of its chunk's tokens
  float* since;                      // [rows, heads]: the decays' product from the chunk's start to the row, the row included
  float* ends;                       // [chunk places, heads, VD, n]: end states, then the states before
  float* decays;                     // [chunk places, heads]: products over the chunk
  const int *seg_q_start, *seg_q_len, *seg_slot;
  int heads, groups;
  int segments, least;               // segments of `least` rows and more go in chunks
  int scans;                         // blocks per head that take the others token by token
};

// `count` rows of N entries into shared rows `pitch` apart; the rows up to CHUNK become zero.
template <int N, int THREADS>
__device__ __forceinline__ void fetch_rows(float* dst, int pitch, const float* src, long long stride, int count) {
  for (int idx = threadIdx.x; idx < CHUNK * (N / 4); idx += THREADS) {
    const int t = idx / (N / 4), i = (idx % (N / 4)) * 4;
    if (t < count)
      copy_async_16(dst + t * pitch + i, src + t * stride + i);
    else
      *reinterpret_cast<float4*>(dst + t * pitch + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// grid: (chunks, groups * 4): 16 of a chunk's rows against its 64 tokens; a thread takes 2 x 4 of them.
template <int N>
__global__ void __launch_bounds__(128)
space_pairs_kernel(SpaceArgs p) {
  constexpr int PITCH = N + 4;
  extern __shared__ __align__(16) float shared[];
  float *s_b = shared, *s_c = shared + CHUNK * PITCH;
  pdl_trigger();
  pdl_wait();
  const int group = blockIdx.y >> 2, part = blockIdx.y & 3;
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.x);
  if (seg < 0) return;
  const int first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK), t0 = part * 16;
  if (t0 >= count) return;
  fetch_rows<N, 128>(s_b, PITCH, p.B + (size_t)first * p.b_stride + (size_t)group * N, p.b_stride, count);
  for (int idx = threadIdx.x; idx < 16 * (N / 4); idx += 128) {
    const int t = idx / (N / 4), i = (idx % (N / 4)) * 4;
    if (t0 + t < count) copy_async_16(s_c + t * PITCH + i, p.C + (size_t)(first + t0 + t) * p.c_stride + (size_t)group * N + i);
  }
  copy_async_commit();
  copy_async_wait<0>();
  __syncthreads();
  const int s = threadIdx.x & 15, t = threadIdx.x >> 4;      // tokens s, s + 16, ..; rows t, t + 8
  float acc[2][4] = {};
  for (int i0 = 0; i0 < N; i0 += 16) {      // sums of 16 entries each, then of those: a single long chain's roundings would show
    float sum[2][4] = {};
#pragma unroll
    for (int i = i0; i < i0 + 16; i += 4) {
      float b[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) load_columns<4>(b[j], s_b + (s + 16 * j) * PITCH + i);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        float c[4];
        load_columns<4>(c, s_c + (t + 8 * k) * PITCH + i);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) sum[k][j] = fmaf(c[e], b[j][e], sum[k][j]);
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[k][j] += sum[k][j];
  }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (t0 + t + 8 * k < count)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        p.pairs[((size_t)(first + t0 + t + 8 * k) * p.groups + group) * CHUNK + s + 16 * j] = acc[k][j];
}

// y += since * (C S^T) for a chunk's rows: rows of C and of S at a pitch of N + 4 in shared memory; thread (j, t) takes rows
// t, t + 8, .. and value channels j, j + 16, ..
template <int N>
__device__ __forceinline__ void read_state(const SpaceArgs& p, const float* s_c, const float* s_s, int first, int count, int head) {
  constexpr int PITCH = N + 4;
  const int j = threadIdx.x & 15, t = threadIdx.x >> 4;
  float acc[8][4] = {};
  for (int i0 = 0; i0 < N; i0 += 16) {      // sums of 16 entries each, then of those
    float sum[8][4] = {};
#pragma unroll 2
    for (int i = i0; i < i0 + 16; i += 4) {
      float s[4][4];
#pragma unroll
      for (int c = 0; c < 4; ++c) load_columns<4>(s[c], s_s + (j + 16 * c) * PITCH + i);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float r[4];
        load_columns<4>(r, s_c + (t + 8 * k) * PITCH + i);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int c = 0; c < 4; ++c) sum[k][c] = fmaf(r[e], s[c][e], sum[k][c]);
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[k][c] += sum[k][c];
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (t + 8 * k >= count) continue;
    const size_t row = (size_t)(first + t + 8 * k) * p.heads + head;
    const float since = p.since[row];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float* at = p.y + row * VD + j + 16 * c;
      *at = fmaf(since, acc[k][c], *at);
    }
  }
}

// grid: (heads, scans + chunks)
template <int N>
__global__ void __launch_bounds__(128, 3)
space_local_kernel(SpaceArgs p) {
  constexpr int PITCH = N + 4;
  extern __shared__ __align__(16) float shared[];
  float* s_w = shared;                         // [CHUNK][W_PITCH]: weight of token s in row t
  float* s_x = s_w + CHUNK * W_PITCH;          // [CHUNK][VD]: dt x
  float* s_b = s_x + CHUNK * VD;               // [CHUNK][N]
  float* s_g = s_b + CHUNK * PITCH;            // [CHUNK] decays
  float* s_dt = s_g + CHUNK;                   // [CHUNK] step sizes
  float* s_to_end = s_dt + CHUNK;              // [CHUNK] decays' product behind a token
  pdl_trigger();
  if ((int)blockIdx.y < p.scans) {
    constexpr int SL = N / SCAN_NPT, PARTS = VD * SL / SCAN_THREADS;
    const ScanArgs scan{p.x, p.B, p.C, p.dt_raw, p.x_stride, p.b_stride, p.c_stride, p.dt_stride, p.dt_bias, p.A_log, p.D, p.states, p.y,
                        p.seg_q_start, p.seg_q_len, p.seg_slot, p.heads, VD, N, p.groups, p.least - 1};
    scan_segment<SL, true>(scan, shared, blockIdx.y / PARTS, blockIdx.x, blockIdx.y % PARTS);
    return;
  }
  const int head = blockIdx.x, tid = threadIdx.x;
  const float rate = expf(p.A_log[head]), bias = p.dt_bias[head], skip = p.D[head];
  pdl_wait();
  const auto [seg, chunk, length, start, slot] =
      chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.y - p.scans);
  if (seg < 0) return;
  const int first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK);
  const int group = head / (p.heads / p.groups);
  const bool whole = length <= CHUNK;
  fetch_rows<N, 128>(s_b, N, p.B + (size_t)first * p.b_stride + (size_t)group * N, p.b_stride, count);
  fetch_rows<VD, 128>(s_x, VD, p.x + (size_t)first * p.x_stride + (size_t)head * VD, p.x_stride, count);
  fetch_rows<CHUNK, 128>(s_w, W_PITCH, p.pairs + ((size_t)first * p.groups + group) * CHUNK, (long long)p.groups * CHUNK, count);
  copy_async_commit();
  if (tid < CHUNK) {
    float dt = 0.f;
    if (tid < count) {
      const float z = p.dt_raw[(size_t)(first + tid) * p.dt_stride + head] + bias;
      dt = z > 20.f ? z : log1pf(expf(z));
    }
    s_dt[tid] = dt;
    s_g[tid] = tid < count ? expf(-rate * dt) : 1.f;
  }
  copy_async_wait<0>();
  __syncthreads();
  {
    // thread (s, half): the weights of token s in the rows of one half, the product of the decays growing along the rows
    const int s = tid & (CHUNK - 1), half = tid / CHUNK;
    float product = 1.f;
    if (half == 1)
      for (int t = s + 1; t < CHUNK / 2; ++t) product *= s_g[t];
#pragma unroll 8
    for (int t = half * (CHUNK / 2); t < (half + 1) * (CHUNK / 2); ++t) {
      if (t > s) product *= s_g[t];
      float& w = s_w[t * W_PITCH + s];
      w = t >= s ? w * product : 0.f;
      if (s == 0 && t < count) p.since[(size_t)(first + t) * p.heads + head] = product * s_g[0];
    }
    if (half == 1) s_to_end[s] = product;
  }
  for (int idx = tid; idx < CHUNK * (VD / 4); idx += 128) {
    float4& v = *reinterpret_cast<float4*>(s_x + idx * 4);
    const float dt = s_dt[idx / (VD / 4)];
    v.x *= dt, v.y *= dt, v.z *= dt, v.w *= dt;
  }
  __syncthreads();
  {
    // outputs of the chunk's own tokens: rows t, t + 8, .., value channels j .. j + 3; rows before a token have no part in it (where a
    // step of k mixes both, the later tokens are left out rather than weighed with zero: an infinity is theirs alone)
    const int j = (tid & 15) * 4, t = tid >> 4;
    float acc[8][4] = {};
#pragma unroll
    for (int block = 0; block < 8; block += 2) {      // sums of 16 tokens each, then of those
      float sum[8][4] = {};
#pragma unroll
      for (int s = 8 * block; s < 8 * block + 16; s += 4) {
        float x[4][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) load_columns<4>(x[e], s_x + (s + e) * VD + j);
#pragma unroll
        for (int k = s / 8; k < 8; ++k) {
          float w[4];
          load_columns<4>(w, s_w + (t + 8 * k) * W_PITCH + s);
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (k > s / 8 || s % 8 + e <= t) {
#pragma unroll
              for (int c = 0; c < 4; ++c) sum[k][c] = fmaf(w[e], x[e][c], sum[k][c]);
            }
        }
      }
#pragma unroll
      for (int k = block; k < 8; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[k][c] += sum[k][c];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int row = t + 8 * k;
      if (row >= count) continue;
      float x[4];
      load_columns<4>(x, p.x + (size_t)(first + row) * p.x_stride + (size_t)head * VD + j);
#pragma unroll
      for (int c = 0; c < 4; ++c) x[c] = fmaf(skip, x[c], acc[k][c]);
      store_columns<4>(p.y + ((size_t)(first + row) * p.heads + head) * VD + j, x);
    }
  }
  // what the chunk's tokens leave behind: value channels j .. j + 7, state entries i .. i + 3 (and 64 further on)
  constexpr int H = N / 64;
  const int i = (tid & 15) * 4, j = (tid >> 4) * 8;
  float end[8][4 * H] = {};
#pragma unroll 4
  for (int s = 0; s < CHUNK; ++s) {
    float b[4 * H], x[8];
    const float behind = s_to_end[s];
    load_columns<4>(reinterpret_cast<float (&)[4]>(x[0]), s_x + s * VD + j);
    load_columns<4>(reinterpret_cast<float (&)[4]>(x[4]), s_x + s * VD + j + 4);
#pragma unroll
    for (int h = 0; h < H; ++h) load_columns<4>(reinterpret_cast<float (&)[4]>(b[4 * h]), s_b + s * N + i + 64 * h);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float weighted = x[r] * behind;
#pragma unroll
      for (int c = 0; c < 4 * H; ++c) end[r][c] = fmaf(weighted, b[c], end[r][c]);
    }
  }
  const float decay = s_to_end[0] * s_g[0];
  float* state = p.states + ((size_t)slot * p.heads + head) * VD * N;
  const size_t place = chunk_place(first, chunk == 0) * p.heads + head;
  if (chunk == 0) {
    // the read of the request's state: its rows and those of C take the place of what is done with
    __syncthreads();
    for (int idx = tid; idx < VD * (N / 4); idx += 128)
      copy_async_16(shared + idx / (N / 4) * PITCH + idx % (N / 4) * 4, state + idx * 4);
    fetch_rows<N, 128>(s_b, PITCH, p.C + (size_t)first * p.c_stride + (size_t)group * N, p.c_stride, count);
    copy_async_commit();
    copy_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int h = 0; h < H; ++h) {
        float before[4];
        load_columns<4>(before, shared + (j + r) * PITCH + i + 64 * h);
#pragma unroll
        for (int c = 0; c < 4; ++c) end[r][4 * h + c] = fmaf(decay, before[c], end[r][4 * h + c]);
      }
  } else if (tid == 0) {
    p.decays[place] = decay;
  }
  float* to = whole ? state : p.ends + place * VD * N;
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int h = 0; h < H; ++h)
      store_columns<4>(to + (size_t)(j + r) * N + i + 64 * h, reinterpret_cast<const float (&)[4]>(end[r][4 * h]));
  if (chunk == 0) read_state<N>(p, s_b, shared, first, count, head);
}

// A thread owns four neighbouring entries and takes the chunks of its segment in order; BATCH chunks are asked for together.
// All launches from a flushed L2, batches of 8 / 16: 32 heads 132.4 / 128.0 us at 2,048 rows, 235 / 223 at 4,000, 128.4 / 126.7 for 1,531 + 77 + 1 + 439; 14
// heads 59.8 / 58.3 and 97.8 / 89.5; segments of few chunks pay for the registers, 512 rows of 14 heads 37.3 / 38.8.
__global__ void __launch_bounds__(256)
space_carry_kernel(SpaceArgs p, int cells) {
  constexpr int BATCH = 16;
  pdl_trigger();
  pdl_wait();
  const auto [seg, which, length, start, slot] = chunk_at<false>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.y);
  if (seg < 0) return;
  const int first = start, chunks = (length + CHUNK - 1) / CHUNK;
  const int at = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (chunks <= 1 || at >= p.heads * cells) return;
  const int head = at / cells, cell = at - head * cells;
  auto place_of = [&](int chunk) { return chunk_place(first + chunk * CHUNK, chunk == 0) * p.heads + head; };
  float4 S = *reinterpret_cast<float4*>(p.ends + place_of(0) * cells + cell);
  for (int c0 = 1; c0 < chunks; c0 += BATCH) {
    float4 own[BATCH];
    float g[BATCH];
#pragma unroll
    for (int k = 0; k < BATCH; ++k)
      if (c0 + k < chunks) {
        own[k] = *reinterpret_cast<float4*>(p.ends + place_of(c0 + k) * cells + cell);
        g[k] = p.decays[place_of(c0 + k)];
      }
#pragma unroll
    for (int k = 0; k < BATCH; ++k)
      if (c0 + k < chunks) {
        *reinterpret_cast<float4*>(p.ends + place_of(c0 + k) * cells + cell) = S;
        S.x = fmaf(g[k], S.x, own[k].x);
        S.y = fmaf(g[k], S.y, own[k].y);
        S.z = fmaf(g[k], S.z, own[k].z);
        S.w = fmaf(g[k], S.w, own[k].w);
      }
  }
  *reinterpret_cast<float4*>(p.states + ((size_t)slot * p.heads + head) * cells + cell) = S;
}

// grid: (heads, chunks), where a segment's first chunks have nothing to do (a single segment's is left out)
template <int N>
__global__ void __launch_bounds__(128, 3)
space_read_kernel(SpaceArgs p) {
  constexpr int PITCH = N + 4;
  extern __shared__ __align__(16) float shared[];
  float *s_s = shared, *s_c = shared + VD * PITCH;
  pdl_trigger();
  pdl_wait();
  const int head = blockIdx.x;
  const auto [seg, chunk, length, start, slot] =
      chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.y + (p.segments == 1 ? 1 : 0));
  if (seg < 0 || chunk == 0) return;
  const int first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK);
  const int group = head / (p.heads / p.groups);
  const float* before = p.ends + (chunk_place(first, false) * p.heads + head) * VD * N;
  for (int idx = threadIdx.x; idx < VD * (N / 4); idx += 128)
    copy_async_16(s_s + idx / (N / 4) * PITCH + idx % (N / 4) * 4, before + idx * 4);
  fetch_rows<N, 128>(s_c, PITCH, p.C + (size_t)first * p.c_stride + (size_t)group * N, p.c_stride, count);
  copy_async_commit();
  copy_async_wait<0>();
  __syncthreads();
  read_state<N>(p, s_c, s_s, first, count, head);
}

template <int N>
int launch_space(const SpaceArgs& a, int rows, int max_q_len, cudaStream_t stream) {
  constexpr size_t pairs_shared = sizeof(float) * (CHUNK + 16) * (N + 4);
  constexpr size_t chunk_shared = sizeof(float) * (CHUNK * (W_PITCH + VD + N + 4) + 3 * CHUNK);
  const size_t segment_shared = scan_shared(N, SCAN_THREADS / (N / SCAN_NPT));
  const size_t local_shared = a.scans > 0 && segment_shared > chunk_shared ? segment_shared : chunk_shared;
  constexpr size_t read_shared = sizeof(float) * (VD + CHUNK) * (N + 4);
  static_assert(VD * (N + 4) <= CHUNK * (W_PITCH + VD), "the state takes the place of weights and inputs");
  const unsigned chunks = (unsigned)long_chunks(rows, a.segments, a.least);
  cudaError_t err = cudaFuncSetAttribute(space_pairs_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pairs_shared);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(space_local_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)local_shared);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(space_read_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)read_shared);
  if (err != cudaSuccess) return (int)err;
  launch_kernel(space_pairs_kernel<N>, dim3(chunks, a.groups * 4), dim3(128), pairs_shared, stream, a);
  int status = launch_status();
  if (status != MLR_OK) return status;
  launch_kernel(space_local_kernel<N>, dim3(a.heads, a.scans + chunks), dim3(128), local_shared, stream, a);
  if ((status = launch_status()) != MLR_OK || max_q_len <= CHUNK) return status;
  launch_kernel(space_carry_kernel, dim3((a.heads * VD * N / 4 + 255) / 256, (unsigned)long_segments(rows, a.segments, a.least)), dim3(256), 0,
                stream, a, VD * N);
  if ((status = launch_status()) != MLR_OK) return status;
  launch_kernel(space_read_kernel<N>, dim3(a.heads, chunks - (a.segments == 1 ? 1 : 0)), dim3(128), read_shared, stream, a);
  return launch_status();
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// float32 scratch of a step, in numbers: end states first (16-byte aligned), then pairs, products along the rows and products
// over the chunks.
MLR_EXPORT long long mlr_state_space_chunk_scratch(int rows, int heads, int n, int groups) {
  return chunk_places(rows) * heads * (VD * (long long)n + 1) + (long long)rows * (groups * CHUNK + heads);
}

// As mlr_state_space_scan, for heads of 64 value channels with states of 64 or 128 entries and x, B, C, states, y and scratch whose
// rows begin on 16-byte boundaries.  rows: the step's rows.  Segments of fewer than least_rows rows
// go token by token as there; others: whether there can be any.
MLR_EXPORT int mlr_state_space_chunks(const float* x, long long x_stride, const float* B, long long b_stride, const float* C,
                                      long long c_stride, const float* dt_raw, long long dt_stride, const float* dt_bias,
                                      const float* A_log, const float* D, float* states, float* y, float* scratch,
                                      const int* seg_q_start, const int* seg_q_len, const int* seg_slot, int segments, int rows,
                                      int max_q_len, int least_rows, int others, int heads, int vdim, int n, int groups, cudaStream_t stream) {
  if (segments == 0) return MLR_OK;
  if (segments < 0 || least_rows <= 0 || rows <= 0 || max_q_len < least_rows || heads <= 0 || groups <= 0 || heads % groups != 0 || scratch == nullptr)
    return MLR_BAD_SIZE;
  if (vdim != VD || (n != 64 && n != 128) || long_chunks(rows, segments, least_rows) + segments * 4ll > 65535 || groups > 65535 / 4) return MLR_TOO_LARGE;
  const uintptr_t pointers = (uintptr_t)x | (uintptr_t)B | (uintptr_t)C | (uintptr_t)states | (uintptr_t)y | (uintptr_t)scratch;
  if (pointers % 16 != 0 || (x_stride | b_stride | c_stride) % 4 != 0) return MLR_BAD_ALIGNMENT;
  SpaceArgs a{x, B, C, dt_raw, x_stride, b_stride, c_stride, dt_stride, dt_bias, A_log, D, states, y,
              nullptr, nullptr, scratch, nullptr, seg_q_start, seg_q_len, seg_slot, heads, groups, segments, least_rows, others ? segments * (VD * (n / SCAN_NPT) / SCAN_THREADS) : 0};
  a.pairs = a.ends + (size_t)chunk_places(rows) * heads * VD * n;
  a.since = a.pairs + (size_t)rows * groups * CHUNK;
  a.decays = a.since + (size_t)rows * heads;
  return n == 64 ? launch_space<64>(a, rows, max_q_len, stream) : launch_space<128>(a, rows, max_q_len, stream);
}
