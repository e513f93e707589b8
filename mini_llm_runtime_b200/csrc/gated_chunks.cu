// The gated linear recurrences (bonus and forget-gate form, see sequence_mix.cu) of steps with long segments, in chunks
// of tokens that are walked side by side.
//
// S_t = diag(a_t) S_{t-1} + b_t v_t^T is linear in S with a diagonal factor, so a chunk's end state is its decays' product
// times the state before it plus what the chunk's own tokens leave behind, and its outputs are those of a walk from zero
// plus (r_t times the decays' running product)^T S.  Three kernels:
//   walk     every chunk of CHUNK tokens at once, token by token from zero (a segment's first chunk, and a segment too short to be
//            cut, from the request's state):
//            outputs without norm, decay-weighted reads, the decays' product, the end state
//   carry    per state entry, the chunks of a segment in order: the state before every chunk, and the request's new state
//   finish   reads times the state before the chunk (a product of CHUNK x dim by dim x vdim), added to the walk's outputs, then
//            root mean square, weight and gate
// Everything is 32-bit multiply-adds; decay products are products of numbers up to one and never divided by, so decays may
// be zero.  Chunks start at a segment's first row.
//
// One CTA used to walk a whole segment of a head (part), 0.4 us per token on 28 of 148 SMs (2,048 tokens, 14 heads of 64 x
// 64): bound by the latency of that chain.  Walked in chunks it is bound by instructions issued: three operations per state
// entry and token in the walk, one in finish.  2,048 tokens of one request, repeated calls, B200: 761 -> 53 us (14 heads of 64), 768 -> 108
// (32 of 64), 608 -> 77 (7 of 128), 709 -> 150 (16 of 128).
#include "chunk_places.cuh"
#include "copy_async.cuh"

namespace mlr {

struct ChunkArgs {
  const float *r, *b, *v, *raw, *gate;           // row-major views, one row per token; rows of whole 16-byte pieces
  long long r_stride, b_stride, v_stride, raw_stride, gate_stride;
  const float *bias, *aux, *weight;              // aux: the bonus (mode 0) or the lower bound (mode 1)
  float eps;
  float* state;                                  // [slots, heads, dim, vdim]
  float* outputs;                                // [rows, heads * vdim]: the walk's outputs
  float* reads;                                  // [rows, heads * dim]: r times the decays since the chunk's start
  float* ends;                                   // [chunk places, heads, dim, vdim]: end states, then the states before
  float* decays;                                 // [chunk places, heads, dim]: products over the chunk
  const int *seg_q_start, *seg_q_len, *seg_slot;
  int heads, weight_per_head;
  int segments, least, split;                    // segments of fewer than `least` rows are another kernel's, below `split` not cut
};

// Thread (lane, warp) walks key channels [16 * slice, +16) of C neighbouring value channels; T tokens at a time are
// staged (16-byte asynchronous copies, the next T under the walk over these) and transformed in place.
template <int MODE, int DIM, int VDIM>
struct WalkShape {
  static constexpr int KD = 16, SLICES = DIM / KD;
  static constexpr int C = VDIM / 32;                    // value channels per thread: a warp spans the head's
  static constexpr int THREADS = SLICES * 32;
  static constexpr int T = 1024 / DIM;                   // tokens staged at once
  static constexpr int STAGE = T * (3 * DIM + VDIM);     // r, a, b, v of T tokens
  static constexpr size_t SHARED = sizeof(float) * (2 * (size_t)STAGE + (size_t)SLICES * T * VDIM + T);
};

template <int MODE, int DIM, int VDIM>
__global__ void __launch_bounds__(WalkShape<MODE, DIM, VDIM>::THREADS)
chunk_walk_kernel(ChunkArgs p) {
  using W = WalkShape<MODE, DIM, VDIM>;
  constexpr int KD = W::KD, C = W::C, T = W::T, THREADS = W::THREADS, SLICES = W::SLICES;
  pdl_wait();
  const int head = blockIdx.x;
  const auto [seg, chunk, length, start, slot] =
      chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.y, p.split);
  if (seg < 0) return;
  extern __shared__ __align__(16) float shared[];
  float* s_o = shared + 2 * W::STAGE;                    // [SLICES][T][VDIM]
  float* s_bonus = s_o + SLICES * T * VDIM;              // [T] sum_i r c b (mode 0)
  const bool whole = length <= CHUNK || length < p.split;      // the segment is this chunk
  const int first = start + chunk * CHUNK, count = whole ? length : min(CHUNK, length - chunk * CHUNK);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, column = lane * C;
  float* state = p.state + ((size_t)slot * p.heads + head) * DIM * VDIM;

  auto fetch = [&](int t0) {
    float* stage = shared + ((t0 / T) & 1) * W::STAGE;
    const int tokens = min(T, count - t0);
    if (tokens > 0) {
      for (int idx = tid; idx < tokens * (DIM / 4); idx += THREADS) {
        const int t = idx / (DIM / 4), i = (idx % (DIM / 4)) * 4;
        const size_t row = (size_t)(first + t0 + t);
        const int at = t * DIM + i, col = head * DIM + i;
        copy_async_16(stage + at, p.r + row * p.r_stride + col);
        copy_async_16(stage + T * DIM + at, p.raw + row * p.raw_stride + col);
        if (MODE == 0) copy_async_16(stage + 2 * T * DIM + at, p.b + row * p.b_stride + col);
      }
      for (int idx = tid; idx < tokens * (VDIM / 4); idx += THREADS) {
        const int t = idx / (VDIM / 4), j = (idx % (VDIM / 4)) * 4;
        copy_async_16(stage + 3 * T * DIM + t * VDIM + j, p.v + (size_t)(first + t0 + t) * p.v_stride + head * VDIM + j);
      }
    }
    copy_async_commit();
  };
  fetch(0);

  float S[KD][C];
#pragma unroll
  for (int i = 0; i < KD; ++i) {
#pragma unroll
    for (int j = 0; j < C; ++j) S[i][j] = 0.f;
    if (chunk == 0) load_columns<C>(S[i], state + (size_t)(warp * KD + i) * VDIM + column);
  }
  float product = 1.f;      // threads below DIM: the decays of their channel since the chunk's start

  for (int t0 = 0; t0 < count; t0 += T) {
    const int tokens = min(T, count - t0);
    float* s_r = shared + ((t0 / T) & 1) * W::STAGE;
    float *s_a = s_r + T * DIM, *s_b = s_a + T * DIM, *s_v = s_b + T * DIM;
    fetch(t0 + T);
    copy_async_wait<1>();
    __syncthreads();
    for (int idx = tid; idx < tokens * DIM; idx += THREADS) {
      const int col = head * DIM + idx % DIM;
      const float z = s_a[idx] + p.bias[col];
      if (MODE == 0) {
        s_a[idx] = expf(-expf(z));
      } else {
        const float lower = p.aux[col], r = s_r[idx];
        const float a = lower + (1.f - lower) * (1.f / (1.f + expf(-z)));
        s_a[idx] = a;
        s_b[idx] = 1.f - a;
        s_r[idx] = r / (1.f + expf(-r));
      }
    }
    __syncthreads();
    if (tid < DIM) {
      for (int t = 0; t < tokens; ++t) {
        const float a = s_a[t * DIM + tid], r = s_r[t * DIM + tid];
        if (MODE == 1) product *= a;
        if (chunk > 0) p.reads[((size_t)(first + t0 + t) * p.heads + head) * DIM + tid] = r * product;
        if (MODE == 0) product *= a;
      }
    }
    if (MODE == 0) {
      for (int t = warp; t < tokens; t += SLICES) {
        float dot = 0.f;
#pragma unroll
        for (int i = lane; i < DIM; i += 32)
          dot = fmaf(s_r[t * DIM + i] * p.aux[head * DIM + i], s_b[t * DIM + i], dot);
        dot = warp_sum(dot);
        if (lane == 0) s_bonus[t] = dot;
      }
    }
    // one token: the thread's key channels against the token's r, a, b (four channels per load)
    auto one_token = [&](int t, float (&o)[C]) {
      float v[C];
      load_columns<C>(v, s_v + t * VDIM + column);
      const float* at = s_r + t * DIM + warp * KD;
#pragma unroll
      for (int j = 0; j < C; ++j) o[j] = 0.f;
#pragma unroll
      for (int i4 = 0; i4 < KD / 4; ++i4) {
        float r[4], a[4], b[4];
        load_columns<4>(r, at + 4 * i4);
        load_columns<4>(a, at + T * DIM + 4 * i4);
        load_columns<4>(b, at + 2 * T * DIM + 4 * i4);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int j = 0; j < C; ++j) {
            float& s = S[4 * i4 + e][j];
            if (MODE == 0) o[j] = fmaf(r[e], s, o[j]);
            s = fmaf(a[e], s, b[e] * v[j]);
            if (MODE == 1) o[j] = fmaf(r[e], s, o[j]);
          }
      }
    };
    // two tokens before their sums are stored, so that the second one's loads may be issued under the first's arithmetic
    for (int t = 0; t < tokens; t += 2) {
      float o[2][C];
      one_token(t, o[0]);
      if (t + 1 < tokens) one_token(t + 1, o[1]);
      store_columns<C>(s_o + (warp * T + t) * VDIM + column, o[0]);
      if (t + 1 < tokens) store_columns<C>(s_o + (warp * T + t + 1) * VDIM + column, o[1]);
    }
    __syncthreads();
    for (int idx = tid; idx < tokens * (VDIM / 4); idx += THREADS) {
      const int t = idx / (VDIM / 4), j = (idx % (VDIM / 4)) * 4;
      float o[4], part[4];
      load_columns<4>(o, s_o + t * VDIM + j);
#pragma unroll
      for (int s = 1; s < SLICES; ++s) {
        load_columns<4>(part, s_o + (s * T + t) * VDIM + j);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] += part[e];
      }
      if (MODE == 0) {
        float v[4];
        load_columns<4>(v, s_v + t * VDIM + j);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = fmaf(v[e], s_bonus[t], o[e]);
      }
      store_columns<4>(p.outputs + ((size_t)(first + t0 + t) * p.heads + head) * VDIM + j, o);
    }
    __syncthreads();      // the stage may be filled again, and s_o and s_bonus written
  }
  const size_t place = chunk_place(first, chunk == 0) * p.heads + head;
  float* end = whole ? state : p.ends + place * DIM * VDIM;
#pragma unroll
  for (int i = 0; i < KD; ++i) store_columns<C>(end + (size_t)(warp * KD + i) * VDIM + column, S[i]);
  if (chunk > 0 && tid < DIM) p.decays[place * DIM + tid] = product;
  // At the end, in all three kernels: blocks of the next that come in while these still fill some SMs land two to an SM beside empty ones, and each of
  // them runs long.  Trigger in front / at the end: 7 heads of 128 x 128, 512 rows 72 / 47 us, 2,048 rows 81 / 77, 16 heads 73 / 48 and 151 / 150; 14 heads of
  // 64 x 64, 300 rows 41 / 28, 512 rows 46 / 29, 2,048 rows 58 / 53, 32 heads, 512 rows 50 / 36.
  pdl_trigger();
}

// A thread owns four neighbouring value channels of one key channel and takes the chunks of its segment in order; BATCH chunks
// are asked for together.  Bound by round trips to the L2, where most of the states lie.  All launches from a flushed L2, batches of
// 8 / 16: 14 heads of 64 66.6 / 65.4 us at 2,048 rows and 116.5 / 112.1 at 4,000, 32 heads 118.4 / 115.9 and 209 / 207, 16 heads of 128 162.9 / 156.8 and
// 291 / 283; segments of few chunks pay for the registers, 200 rows of 32 heads of 64 38.2 / 39.6, 512 rows of 14 39.8 / 40.2.
__global__ void __launch_bounds__(256)
chunk_carry_kernel(ChunkArgs p, int dim, int vdim) {
  constexpr int BATCH = 16;
  pdl_wait();
  const auto [seg, which, length, start, slot] = chunk_at<false>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, max(p.least, p.split), blockIdx.y);
  if (seg < 0) return;
  const int first = start, chunks = (length + CHUNK - 1) / CHUNK, cells = dim * vdim;
  const int at = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (chunks <= 1 || at >= p.heads * cells) return;
  const int head = at / cells, cell = at - head * cells, i = cell / vdim;
  auto end_of = [&](int chunk) {
    return reinterpret_cast<float4*>(p.ends + (chunk_place(first + chunk * CHUNK, chunk == 0) * p.heads + head) * cells + cell);
  };
  float4 S = *end_of(0);
  for (int c0 = 1; c0 < chunks; c0 += BATCH) {
    float4 own[BATCH];
    float a[BATCH];
#pragma unroll
    for (int k = 0; k < BATCH; ++k)
      if (c0 + k < chunks) {
        own[k] = *end_of(c0 + k);
        a[k] = p.decays[(chunk_place(first + (c0 + k) * CHUNK, false) * p.heads + head) * dim + i];
      }
#pragma unroll
    for (int k = 0; k < BATCH; ++k)
      if (c0 + k < chunks) {
        *end_of(c0 + k) = S;
        S.x = fmaf(a[k], S.x, own[k].x);
        S.y = fmaf(a[k], S.y, own[k].y);
        S.z = fmaf(a[k], S.z, own[k].z);
        S.w = fmaf(a[k], S.w, own[k].w);
      }
  }
  *reinterpret_cast<float4*>(p.state + ((size_t)slot * p.heads + head) * cells + cell) = S;
  pdl_trigger();
}

// CTA per (head, chunk, segment): VDIM / 4 threads side by side take a token's value channels, eight groups of them eight
// tokens each (tokens 8 apart).
template <typename T, int MODE, int DIM, int VDIM>
__global__ void __launch_bounds__(2 * VDIM)
chunk_finish_kernel(ChunkArgs p, T* __restrict__ out) {
  constexpr int LANES = VDIM / 4, THREADS = 2 * VDIM, TOKENS = CHUNK / 8, PITCH = DIM + 4;
  pdl_wait();
  const int head = blockIdx.x;
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.y);
  if (seg < 0) return;
  extern __shared__ __align__(16) float shared[];
  float *s_reads = shared, *s_state = shared + CHUNK * PITCH;
  const int first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK);
  const int j = (threadIdx.x % LANES) * 4, group = threadIdx.x / LANES;
  float o[TOKENS][4];
  const bool behind = chunk > 0 && length >= p.split;      // a state before that the walk did not start from
  if (behind) {
    const float* before = p.ends + (chunk_place(first, false) * p.heads + head) * DIM * VDIM;
    for (int idx = threadIdx.x; idx < DIM * VDIM / 4; idx += THREADS) copy_async_16(s_state + idx * 4, before + idx * 4);
    for (int idx = threadIdx.x; idx < count * (DIM / 4); idx += THREADS) {
      const int t = idx / (DIM / 4), i = (idx % (DIM / 4)) * 4;
      copy_async_16(s_reads + t * PITCH + i, p.reads + ((size_t)(first + t) * p.heads + head) * DIM + i);
    }
    copy_async_commit();
  }
#pragma unroll
  for (int k = 0; k < TOKENS; ++k) {
    const int t = group + 8 * k;
    if (t < count) load_columns<4>(o[k], p.outputs + ((size_t)(first + t) * p.heads + head) * VDIM + j);
  }
  if (behind) {
    copy_async_wait<0>();
    __syncthreads();
    float add[TOKENS][4];      // sums of their own: the rest of the output joins last
#pragma unroll
    for (int k = 0; k < TOKENS; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) add[k][e] = 0.f;
    for (int i = 0; i < DIM; i += 4) {
      float s[4][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) load_columns<4>(s[e], s_state + (i + e) * VDIM + j);
#pragma unroll
      for (int k = 0; k < TOKENS; ++k) {
        float r[4];      // rows past the segment's end hold stale numbers whose sums go nowhere
        load_columns<4>(r, s_reads + (group + 8 * k) * PITCH + i);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int c = 0; c < 4; ++c) add[k][c] = fmaf(r[e], s[e][c], add[k][c]);
      }
    }
#pragma unroll
    for (int k = 0; k < TOKENS; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[k][e] += add[k][e];
  }
  float weight[4];
  load_columns<4>(weight, p.weight + (p.weight_per_head ? head * VDIM + j : j));
#pragma unroll
  for (int k = 0; k < TOKENS; ++k) {
    const int t = group + 8 * k;
    float sq = 0.f;
    if (t < count) {
#pragma unroll
      for (int e = 0; e < 4; ++e) sq = fmaf(o[k][e], o[k][e], sq);
    }
#pragma unroll
    for (int m = LANES / 2; m > 0; m >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, m);
    if (t >= count) continue;
    const float factor = 1.f / sqrtf(sq / (float)VDIM + p.eps);
    const size_t row = (size_t)(first + t);
    T y[4];
    float g[4];
    if (MODE == 0) load_columns<4>(g, p.gate + row * p.gate_stride + head * VDIM + j);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float value = o[k][e] * factor * weight[e];
      if (MODE == 0) value *= g[e] / (1.f + expf(-g[e]));
      y[e] = from_float<T>(value);
    }
    T* dst = out + (row * p.heads + head) * VDIM + j;
    if constexpr (sizeof(T) == 4)
      *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(y);
    else
      *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(y);
  }
  pdl_trigger();
}

template <typename T, int MODE, int DIM, int VDIM>
int launch_chunks(const ChunkArgs& args, void* out, int rows, int max_q_len, cudaStream_t stream) {
  using W = WalkShape<MODE, DIM, VDIM>;
  constexpr size_t finish_shared = sizeof(float) * (CHUNK * (DIM + 4) + (size_t)DIM * VDIM);
  const dim3 grid(args.heads, (unsigned)long_chunks(rows, args.segments, args.least));
  auto walk = chunk_walk_kernel<MODE, DIM, VDIM>;
  auto finish = chunk_finish_kernel<T, MODE, DIM, VDIM>;
  cudaError_t err = cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W::SHARED);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)finish_shared);
  if (err != cudaSuccess) return (int)err;
  launch_kernel(walk, grid, dim3(W::THREADS), W::SHARED, stream, args);
  int status = launch_status();
  if (status != MLR_OK) return status;
  if (max_q_len > CHUNK && max_q_len >= args.split) {
    const int least = args.least > args.split ? args.least : args.split;
    launch_kernel(chunk_carry_kernel, dim3((args.heads * DIM * VDIM / 4 + 255) / 256, (unsigned)long_segments(rows, args.segments, least)), dim3(256), 0, stream, args, DIM, VDIM);
    if ((status = launch_status()) != MLR_OK) return status;
  }
  launch_kernel(finish, grid, dim3(2 * VDIM), finish_shared, stream, args, (T*)out);
  return launch_status();
}

template <int MODE>
int launch_chunks(const ChunkArgs& args, void* out, int rows, int max_q_len, int dim, int vdim, int out_dtype,
                  cudaStream_t stream) {
  const bool wide = dim == 128;
  if (dim != vdim || (dim != 64 && dim != 128)) return MLR_TOO_LARGE;
  if (out_dtype == MLR_F32)
    return wide ? launch_chunks<float, MODE, 128, 128>(args, out, rows, max_q_len, stream)
                : launch_chunks<float, MODE, 64, 64>(args, out, rows, max_q_len, stream);
  if (out_dtype == MLR_BF16)
    return wide ? launch_chunks<bf16, MODE, 128, 128>(args, out, rows, max_q_len, stream)
                : launch_chunks<bf16, MODE, 64, 64>(args, out, rows, max_q_len, stream);
  return MLR_BAD_DTYPE;
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// float32 scratch of a step, in numbers: the walk's outputs, its reads, and per chunk place an end
// state and decay products.
MLR_EXPORT long long mlr_gated_chunk_scratch(int rows, int heads, int dim, int vdim) {
  return (long long)heads * ((long long)rows * (dim + vdim) + chunk_places(rows) * dim * (vdim + 1));
}

// As mlr_gated_recurrence, for square heads of 64 or 128 and inputs (state, weights, output and scratch too) whose rows begin
// on 16-byte boundaries.  rows: the step's rows; scratch: mlr_gated_chunk_scratch numbers.  Segments of fewer than least_rows rows are
// left alone, those of fewer than split_rows walked in one piece.
MLR_EXPORT int mlr_gated_recurrence_chunks(int mode, const float* r, long long r_stride, const float* b, long long b_stride,
                                           const float* v, long long v_stride, const float* raw, long long raw_stride,
                                           const float* gate, long long gate_stride, const float* bias, const float* aux,
                                           const float* weight, float eps, float* state, void* out, float* scratch,
                                           const int* seg_q_start, const int* seg_q_len, const int* seg_slot, int segments,
                                           int rows, int max_q_len, int least_rows, int split_rows, int heads, int dim, int vdim, int out_dtype,
                                           cudaStream_t stream) {
  if (segments == 0 || max_q_len < least_rows) return MLR_OK;
  if (segments < 0 || heads <= 0 || rows <= 0 || max_q_len <= 0 || least_rows <= 0 || split_rows < 0 || scratch == nullptr) return MLR_BAD_SIZE;
  if (long_chunks(rows, segments, least_rows) > 65535) return MLR_TOO_LARGE;
  const uintptr_t pointers = (uintptr_t)r | (uintptr_t)b | (uintptr_t)v | (uintptr_t)raw | (uintptr_t)gate | (uintptr_t)weight |
                             (uintptr_t)state | (uintptr_t)out | (uintptr_t)scratch;
  if (pointers % 16 != 0 || (r_stride | b_stride | v_stride | raw_stride | gate_stride) % 4 != 0) return MLR_BAD_ALIGNMENT;
  ChunkArgs args;
  args.r = r; args.b = b; args.v = v; args.raw = raw; args.gate = gate;
  args.r_stride = r_stride; args.b_stride = b_stride; args.v_stride = v_stride;
  args.raw_stride = raw_stride; args.gate_stride = gate_stride;
  args.bias = bias; args.aux = aux; args.weight = weight; args.eps = eps; args.state = state;
  args.outputs = scratch;
  args.reads = args.outputs + (size_t)rows * heads * vdim;
  args.ends = args.reads + (size_t)rows * heads * dim;
  args.decays = args.ends + (size_t)chunk_places(rows) * heads * dim * vdim;
  args.seg_q_start = seg_q_start; args.seg_q_len = seg_q_len; args.seg_slot = seg_slot;
  args.heads = heads; args.weight_per_head = mode == 0 ? 1 : 0; args.segments = segments; args.least = least_rows; args.split = split_rows;
  if (mode == 0) return launch_chunks<0>(args, out, rows, max_q_len, dim, vdim, out_dtype, stream);
  if (mode == 1) return launch_chunks<1>(args, out, rows, max_q_len, dim, vdim, out_dtype, stream);
  return MLR_BAD_SIZE;
}
