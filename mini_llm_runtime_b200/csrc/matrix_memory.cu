// A matrix memory with exponential gates (the mLSTM of xLSTM): per request and head a memory S [dim, vdim] and a
// normaliser n [dim] in 32-bit floats that are carried from token to token,
//
//   i = cap tanh((i_raw + i_bias) / cap),   f = logsigmoid(cap tanh((f_raw + f_bias) / cap))       (logarithms)
//   m_t = max(f + m_{t-1}, i)
//   S_t = e^(f + m_{t-1} - m_t) S_{t-1} + e^(i - m_t) k_t v_t^T,      n_t likewise with k_t alone
//   o_t = S_t^T q_t / (max(|n_t . q_t|, e^(-m_t)) + guard),           q = q_raw * dim^-1/2
//   out = o / rms(o) * weight * sigmoid(gate)                          (rms over a head's channels)
//
// The state is kept transposed with n as one more value channel (whose value is 1): [vdim + 1, dim].
//
// matrix_memory_decode_kernel   steps of single rows: everything above in one launch, a block per (request, head).
// matrix_memory_gates_kernel    per token and head [keep, write, e^(-m)]: the running maximum is an associative scan of
//                               maps m -> max(a + m, b).  Wherever m appears the same rounded m_t is used, so what m's
//                               own rounding does to S cancels out.
// matrix_memory_scan_kernel     the recurrence of longer segments, token after token, value channels over blocks.
// matrix_memory_finish_kernel   normaliser, head norm, weight and gate of the scan's rows.
//
// In bfloat16, prompts take chunks of 64 tokens through the tensor cores instead of the token-by-token scan.  q, k and
// v are projections and enter rounded to bfloat16; everything else stays 32-bit: products of a 32-bit operand are
// taken of its three bfloat16 parts (24 bits), sums are 32-bit.  With K_t the product of the keeps of a chunk's tokens up to
// t and D_ts = write_s times the keeps of s + 1 .. t (products of numbers up to one, no differences of logarithms),
//
//   S^T q_t (of token t) = K_t S_before^T q_t + sum_{s <= t} A_ts v_s    with  A_ts = D_ts (k_s . q_t)
//   S_behind = K_last S_before + sum_s k_s (D_last,s v_s)^T
//
// Chunks side by side (value heads of up to 128, portions of more than two chunks), which is linear in S as well:
// memory_ends_kernel            per chunk and head: what its own tokens leave behind, sum_s k_s (D_last,s v_s)^T.
// memory_carry_kernel           per state entry, the chunks of a segment in order: the state before each.
// memory_outputs_kernel         per chunk and head: A, both products, normaliser, head norm, weight and gate.
// One behind the other:
// matrix_memory_pairs_kernel    all chunks at once: A, D_last and K of every chunk, q, k and v as bfloat16.
// matrix_memory_chunks_kernel   the chunks of a (request, head) one after the other, value channels over blocks; the
//                               state stays in registers as accumulators.
#include "chunk_places.cuh"
#include "part_products.cuh"
#include "copy_async.cuh"
#include "lane_sums.cuh"

namespace mlr {

struct MemoryArgs {
  const float *q, *k, *v, *i_raw, *f_raw, *gate;      // row-major views, one row per token
  long long q_stride, k_stride, v_stride, i_stride, f_stride, gate_stride;
  const float *i_bias, *f_bias;         // [heads]
  const float* weight;                  // [heads * vdim]
  float4* coef;                         // [rows, heads]: keep, write, e^(-m), unused
  float* reads;                         // [rows, heads, vdim]: S^T q before the normaliser
  float* norms;                         // [rows, heads]: n . q
  float* pairs;                         // chunks: [rows, heads, 64], A
  float2* factors;                      // chunks: [rows, heads]: D_last and K
  bf16 *q16, *k16, *v16;                // chunks: [rows, heads * dim], the same, [rows, heads * vdim]
  float* states;                        // [slots, heads, vdim + 1, dim]
  float* maxima;                        // [slots, heads]
  float* ends;                          // chunks side by side: [chunks, heads, vdim + 1, dim], what a chunk's tokens leave, then the state before it
  float* spans;                         // [chunks, heads]: product of a chunk's keeps
  const int *seg_q_start, *seg_q_len, *seg_slot;
  int segments, least, heads, dim, vdim;      // least: rows of a segment that goes in chunks side by side; 2: single rows go as decoded ones
  float cap, guard, eps, q_scale;
};

__device__ __forceinline__ float capped(float raw, float cap) { return cap * tanhf(raw / cap); }
__device__ __forceinline__ float log_sigmoid(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float sigmoid(float z) { return 1.f / (1.f + expf(-z)); }

// ------------------------------------------------------------------ single rows
constexpr int DECODE_THREADS = 256;
constexpr int DECODE_WARPS = DECODE_THREADS / 32;

__device__ __forceinline__ void round16(float4& x) {
  x = make_float4(__bfloat162float(__float2bfloat16_rn(x.x)), __bfloat162float(__float2bfloat16_rn(x.y)), __bfloat162float(__float2bfloat16_rn(x.z)),
                  __bfloat162float(__float2bfloat16_rn(x.w)));
}

// A block's row of a segment and head.  PIECES: 16-byte pieces of a state row per lane (dim <= 128 * PIECES, rows and pointers aligned), or 0: any
// size, number by number.  shared: [vdim + 1] reads.  BESIDE: a step of longer segments, whose q, k and v enter in bfloat16; others than single rows are left to them.
template <typename T, int PIECES, bool BESIDE>
__device__ __forceinline__ void decode_row(const MemoryArgs& p, T* out, float* shared, int seg, int head) {
  __shared__ float scratch[32];
  const int D = p.dim, V = p.vdim;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t slot_head = (size_t)p.seg_slot[seg] * p.heads + head;
  const size_t row = p.seg_q_start[seg];
  float* state = p.states + slot_head * (size_t)(V + 1) * D;
  const float i_bias = p.i_bias[head], f_bias = p.f_bias[head];
  pdl_wait();
  if (BESIDE && p.seg_q_len[seg] != 1) return;
  const float i_raw = __ldcg(p.i_raw + row * p.i_stride + head), f_raw = __ldcg(p.f_raw + row * p.f_stride + head);
  const float m_old = __ldcg(p.maxima + slot_head);
  const float* q = p.q + row * p.q_stride + (size_t)head * D;
  const float* k = p.k + row * p.k_stride + (size_t)head * D;
  const float* v = p.v + row * p.v_stride + (size_t)head * V;
  float m_new = 0.f, keep = 0.f, write = 0.f;
  auto gates = [&]() {
    const float log_in = capped(i_raw + i_bias, p.cap), log_forget = log_sigmoid(capped(f_raw + f_bias, p.cap));
    m_new = fmaxf(log_forget + m_old, log_in);
    keep = expf(log_forget + m_old - m_new);
    write = expf(log_in - m_new);
  };
  if (PIECES > 0) {
    constexpr int N = PIECES > 0 ? PIECES : 1, ROWS = N >= 4 ? 2 : 8 / N;      // state rows in flight per warp
    float4 q4[N], k4[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const int d = (n * 32 + lane) << 2;
      q4[n] = k4[n] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (d < D) {
        q4[n] = __ldcg(reinterpret_cast<const float4*>(q + d));
        k4[n] = __ldcg(reinterpret_cast<const float4*>(k + d));
        if (BESIDE) round16(q4[n]), round16(k4[n]);
      }
    }
    bool first = true;
    for (int v0 = warp; v0 <= V; v0 += DECODE_WARPS * ROWS) {
      float4 s[ROWS][N];
      float value[ROWS], sum[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int c = v0 + r * DECODE_WARPS;
        value[r] = c < V ? __ldcg(v + c) : 1.f;
        if (BESIDE) value[r] = __bfloat162float(__float2bfloat16_rn(value[r]));
#pragma unroll
        for (int n = 0; n < N; ++n) {
          const int d = (n * 32 + lane) << 2;
          s[r][n] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (c <= V && d < D) s[r][n] = __ldcg(reinterpret_cast<const float4*>(state + (size_t)c * D + d));
        }
      }
      if (first) gates();      // while the state is on its way
      first = false;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int c = v0 + r * DECODE_WARPS;
        const float u = write * value[r];
        sum[r] = 0.f;
#pragma unroll
        for (int n = 0; n < N; ++n) {
          const int d = (n * 32 + lane) << 2;
          float4& x = s[r][n];
          x.x = fmaf(k4[n].x, u, keep * x.x); x.y = fmaf(k4[n].y, u, keep * x.y);
          x.z = fmaf(k4[n].z, u, keep * x.z); x.w = fmaf(k4[n].w, u, keep * x.w);
          sum[r] = fmaf(q4[n].x, x.x, sum[r]); sum[r] = fmaf(q4[n].y, x.y, sum[r]);
          sum[r] = fmaf(q4[n].z, x.z, sum[r]); sum[r] = fmaf(q4[n].w, x.w, sum[r]);
          if (c <= V && d < D) *reinterpret_cast<float4*>(state + (size_t)c * D + d) = x;
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) sum[r] = warp_sum(sum[r]);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int c = v0 + r * DECODE_WARPS;
        if (lane == 0 && c <= V) shared[c] = sum[r] * p.q_scale;
      }
    }
    if (first) gates();        // a warp without a row of its own
  } else {
    gates();
    for (int c = warp; c <= V; c += DECODE_WARPS) {
      const float u = write * (c < V ? __ldcg(v + c) : 1.f);
      float sum = 0.f;
      for (int d = lane; d < D; d += 32) {
        float* s = state + (size_t)c * D + d;
        const float x = fmaf(__ldcg(k + d), u, keep * __ldcg(s));
        *s = x;
        sum = fmaf(__ldcg(q + d), x, sum);
      }
      sum = warp_sum(sum);
      if (lane == 0) shared[c] = sum * p.q_scale;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) p.maxima[slot_head] = m_new;      // every thread read the old one before the barrier
  const float inverse = 1.f / (fmaxf(fabsf(shared[V]), expf(-m_new)) + p.guard);
  float sq = 0.f;
  for (int c = threadIdx.x; c < V; c += DECODE_THREADS) {
    const float o = shared[c] * inverse;
    sq = fmaf(o, o, sq);
  }
  const float factor = inverse / sqrtf(block_sum(sq, scratch) / (float)V + p.eps);
  for (int c = threadIdx.x; c < V; c += DECODE_THREADS) {
    const float g = __ldcg(p.gate + row * p.gate_stride + (size_t)head * V + c);
    out[row * p.heads * V + (size_t)head * V + c] = from_float<T>(shared[c] * factor * p.weight[head * V + c] * sigmoid(g));
  }
}

// grid: (segments, heads)
template <typename T, int PIECES>
__global__ void __launch_bounds__(DECODE_THREADS)
matrix_memory_decode_kernel(MemoryArgs p, T* __restrict__ out) {
  pdl_trigger();
  extern __shared__ __align__(16) float shared[];
  decode_row<T, PIECES, false>(p, out, shared, blockIdx.x, blockIdx.y);
}

// ------------------------------------------------------------------ gates of longer segments
constexpr int GATE_THREADS = 1024;
constexpr int GATE_WARPS = GATE_THREADS / 32;

// grid: (segments, heads).  1,024 tokens per turn.
__global__ void __launch_bounds__(GATE_THREADS)
matrix_memory_gates_kernel(MemoryArgs p) {
  __shared__ float total_a[GATE_WARPS], total_b[GATE_WARPS], last[GATE_WARPS];
  const int seg = blockIdx.x, head = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t slot_head = (size_t)p.seg_slot[seg] * p.heads + head;
  const size_t row0 = p.seg_q_start[seg];
  const int q_len = p.seg_q_len[seg];
  const float i_bias = p.i_bias[head], f_bias = p.f_bias[head];
  // The recurrence behind this kernel is few blocks that run long: brought in while the product in front of this
  // kernel still fills the SMs, they would land several to an SM.  So the trigger comes after the wait.
  pdl_wait();
  pdl_trigger();
  if (q_len < p.least) return;
  float before = __ldcg(p.maxima + slot_head);       // m ahead of this turn's tokens
  float i_next = 0.f, f_next = 0.f;
  auto ask = [&](int t) {
    if (t < q_len) {
      i_next = __ldcg(p.i_raw + (row0 + t) * p.i_stride + head);
      f_next = __ldcg(p.f_raw + (row0 + t) * p.f_stride + head);
    }
  };
  ask(threadIdx.x);
  for (int t0 = 0; t0 < q_len; t0 += GATE_THREADS) {
    const int t = t0 + threadIdx.x;
    float log_in = -INFINITY, log_forget = 0.f;      // a place without a token changes nothing
    if (t < q_len) {
      log_in = capped(i_next + i_bias, p.cap);
      log_forget = log_sigmoid(capped(f_next + f_bias, p.cap));
    }
    ask(t + GATE_THREADS);
    // inclusive scan of the maps m -> max(a + m, b), earlier tokens first
    float a = log_forget, b = log_in;
#pragma unroll
    for (int step = 1; step < 32; step <<= 1) {
      const float a_up = __shfl_up_sync(0xffffffffu, a, step), b_up = __shfl_up_sync(0xffffffffu, b, step);
      if (lane >= step) {
        b = fmaxf(b_up + a, b);
        a += a_up;
      }
    }
    if (lane == 31) {
      total_a[warp] = a;
      total_b[warp] = b;
    }
    __syncthreads();
    float carried = before;
    for (int w = 0; w < warp; ++w) carried = fmaxf(total_a[w] + carried, total_b[w]);
    const float m = fmaxf(a + carried, b);
    if (lane == 31) last[warp] = m;
    __syncthreads();
    float m_before = __shfl_up_sync(0xffffffffu, m, 1);
    if (lane == 0) m_before = warp > 0 ? last[warp - 1] : before;
    if (t < q_len)
      p.coef[(row0 + t) * p.heads + head] = make_float4(expf(log_forget + m_before - m), expf(log_in - m), expf(-m), 0.f);
    before = last[GATE_WARPS - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) p.maxima[slot_head] = before;
}

// ------------------------------------------------------------------ the recurrence of longer segments
// grid: (segments, heads, blocks of state rows).  A group of SL lanes holds C rows of the head's transposed state
// (value channels, the last one the normaliser's), each lane E key channels of them in interleaved pieces of four.
// Reads are summed over the lanes for TB tokens at once; the updates need no sum.  WIDE: rows are staged in 16-byte
// pieces (sizes and strides multiples of four floats, pointers aligned).
template <int E, int SL, int C, bool WIDE, int THREADS>
__global__ void __launch_bounds__(THREADS)
matrix_memory_scan_kernel(MemoryArgs p) {
  pdl_trigger();
  extern __shared__ __align__(16) float shared[];
  constexpr int TB = 4, GROUPS = THREADS / SL, COLS = GROUPS * C, N = TB * C;
  constexpr int TOKENS = SL == 32 ? 16 : 32;      // tokens staged at once
  constexpr int pitch = E * SL;                   // staged rows of keys and queries, filled up with zeros
  constexpr int COEF = 4;
  constexpr int buffer = TOKENS * (2 * pitch + COLS + COEF);
  const int D = p.dim, V = p.vdim;
  const int seg = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * COLS;
  const int lane = threadIdx.x & 31, s = threadIdx.x % SL, group = threadIdx.x / SL;
  const int q_start = p.seg_q_start[seg], q_len = p.seg_q_len[seg];
  float* state = p.states + ((size_t)p.seg_slot[seg] * p.heads + head) * (size_t)(V + 1) * D;

  // what no copy overwrites: zeros behind the rows' D entries, the normaliser's value of one, zeros behind it
  if (D < pitch) {
    for (int idx = threadIdx.x; idx < 4 * TOKENS * (pitch - D); idx += THREADS) {
      const int r = idx / (pitch - D), d = D + idx - r * (pitch - D);
      shared[(r / (2 * TOKENS)) * buffer + (r % (2 * TOKENS)) * pitch + d] = 0.f;
    }
  }
  if (col0 + COLS > V) {
    for (int idx = threadIdx.x; idx < 2 * TOKENS * COLS; idx += THREADS) {
      const int which = idx / (TOKENS * COLS), at = idx - which * TOKENS * COLS, c = at % COLS;
      if (col0 + c >= V) shared[which * buffer + 2 * TOKENS * pitch + at] = col0 + c == V ? 1.f : 0.f;
    }
  }
  pdl_wait();
  auto stage = [&](int t0, int which) {
    float* k_rows = shared + which * buffer;
    float* q_rows = k_rows + TOKENS * pitch;
    float* v_rows = q_rows + TOKENS * pitch;
    float* coef = v_rows + TOKENS * COLS;
    const int tokens = min(TOKENS, q_len - t0);
    const size_t row0 = (size_t)(q_start + t0);
    if (WIDE) {
      const int per_row = D >> 2;
      for (int idx = threadIdx.x; idx < tokens * per_row; idx += THREADS) {
        const int t = idx / per_row, d = (idx - t * per_row) << 2;
        copy_async_16(k_rows + t * pitch + d, p.k + (row0 + t) * p.k_stride + (size_t)head * D + d);
        copy_async_16(q_rows + t * pitch + d, p.q + (row0 + t) * p.q_stride + (size_t)head * D + d);
      }
      constexpr int V_PIECES = (COLS + 3) / 4;
      for (int idx = threadIdx.x; idx < tokens * V_PIECES; idx += THREADS) {
        const int t = idx / V_PIECES, c = (idx - t * V_PIECES) << 2;
        if (col0 + c < V) copy_async_16(v_rows + t * COLS + c, p.v + (row0 + t) * p.v_stride + (size_t)head * V + col0 + c);
      }
    } else {
      for (int idx = threadIdx.x; idx < tokens * D; idx += THREADS) {
        const int t = idx / D, d = idx - t * D;
        copy_async_4(k_rows + t * pitch + d, p.k + (row0 + t) * p.k_stride + (size_t)head * D + d);
        copy_async_4(q_rows + t * pitch + d, p.q + (row0 + t) * p.q_stride + (size_t)head * D + d);
      }
      for (int idx = threadIdx.x; idx < tokens * COLS; idx += THREADS) {
        const int t = idx / COLS, c = idx - t * COLS;
        if (col0 + c < V) copy_async_4(v_rows + idx, p.v + (row0 + t) * p.v_stride + (size_t)head * V + col0 + c);
      }
    }
    if (threadIdx.x < tokens)
      copy_async_16(coef + threadIdx.x * COEF, reinterpret_cast<const float*>(p.coef + (row0 + threadIdx.x) * p.heads + head));
    copy_async_commit();
    if (tokens % TB != 0) {      // the rest of the last block of tokens: kept as it is, nothing written
      const int fill = TB - tokens % TB;
      for (int idx = threadIdx.x; idx < fill * pitch; idx += THREADS) k_rows[tokens * pitch + idx] = q_rows[tokens * pitch + idx] = 0.f;
      for (int idx = threadIdx.x; idx < fill * COLS; idx += THREADS) v_rows[tokens * COLS + idx] = 0.f;
      for (int idx = threadIdx.x; idx < fill * COEF; idx += THREADS) coef[tokens * COEF + idx] = idx % COEF == 0 ? 1.f : 0.f;
    }
  };
  stage(0, 0);
  auto entry = [&](int i) { return (((i >> 2) * SL + s) << 2) + (i & 3); };      // key channel of a lane's i-th number
  float S[C][E];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int column = col0 + group * C + c;
    const bool mine = column <= V;
    const float* src = state + (size_t)(mine ? column : 0) * D;
    if (WIDE) {
#pragma unroll
      for (int i = 0; i < E; i += 4) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (mine && entry(i) < D) x = __ldcg(reinterpret_cast<const float4*>(src + entry(i)));
        S[c][i] = x.x; S[c][i + 1] = x.y; S[c][i + 2] = x.z; S[c][i + 3] = x.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i) S[c][i] = mine && entry(i) < D ? __ldcg(src + entry(i)) : 0.f;
    }
  }
  int which = 0;
  for (int t0 = 0; t0 < q_len; t0 += TOKENS, which ^= 1) {
    const int tokens = min(TOKENS, q_len - t0);
    const bool more = t0 + TOKENS < q_len;
    if (more) stage(t0 + TOKENS, which ^ 1);
    if (more) copy_async_wait<1>(); else copy_async_wait<0>();
    __syncthreads();
    const float* k_rows = shared + which * buffer;
    const float* q_rows = k_rows + TOKENS * pitch;
    const float* v_rows = q_rows + TOKENS * pitch;
    const float* coef = v_rows + TOKENS * COLS;
    for (int t = 0; t < tokens; t += TB) {
      float read[N];
#pragma unroll
      for (int n = 0; n < TB; ++n) {
        const float2 gate = *reinterpret_cast<const float2*>(coef + (t + n) * COEF);      // keep, write
        float u[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          u[c] = gate.y * v_rows[(t + n) * COLS + group * C + c];
          read[n * C + c] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < E; i += 4) {
          const float4 k4 = *reinterpret_cast<const float4*>(k_rows + (t + n) * pitch + entry(i));
          const float4 q4 = *reinterpret_cast<const float4*>(q_rows + (t + n) * pitch + entry(i));
#pragma unroll
          for (int c = 0; c < C; ++c) {
            float sum = read[n * C + c];
            S[c][i] = fmaf(k4.x, u[c], gate.x * S[c][i]);
            sum = fmaf(q4.x, S[c][i], sum);
            S[c][i + 1] = fmaf(k4.y, u[c], gate.x * S[c][i + 1]);
            sum = fmaf(q4.y, S[c][i + 1], sum);
            S[c][i + 2] = fmaf(k4.z, u[c], gate.x * S[c][i + 2]);
            sum = fmaf(q4.z, S[c][i + 2], sum);
            S[c][i + 3] = fmaf(k4.w, u[c], gate.x * S[c][i + 3]);
            read[n * C + c] = fmaf(q4.w, S[c][i + 3], sum);
          }
        }
      }
      const int first = spread_sums<N, SL>(read, lane);
      constexpr int HELD = N > SL ? N / SL : 1;
      if (N >= SL || (s & (SL / N - 1)) == 0) {
#pragma unroll
        for (int i = 0; i < HELD; ++i) {
          const int number = first + i, n = number / C, column = col0 + group * C + number % C;
          if (t + n < tokens && column <= V) {
            const size_t row_head = (size_t)(q_start + t0 + t + n) * p.heads + head;
            if (column < V) p.reads[row_head * V + column] = read[i] * p.q_scale;
            else p.norms[row_head] = read[i] * p.q_scale;
          }
        }
      }
    }
    __syncthreads();      // the next turn of the loop stages into this buffer
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int column = col0 + group * C + c;
    if (column > V) continue;
    float* dst = state + (size_t)column * D;
    if (WIDE) {
#pragma unroll
      for (int i = 0; i < E; i += 4)
        if (entry(i) < D) *reinterpret_cast<float4*>(dst + entry(i)) = make_float4(S[c][i], S[c][i + 1], S[c][i + 2], S[c][i + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i)
        if (entry(i) < D) dst[entry(i)] = S[c][i];
    }
  }
}

template <int E, int SL, int C, bool WIDE, int THREADS = 128>
static int launch_scan(const MemoryArgs& p, int segments, cudaStream_t stream) {
  constexpr int COLS = THREADS / SL * C, TOKENS = SL == 32 ? 16 : 32;
  constexpr size_t shared = sizeof(float) * 2 * (size_t)TOKENS * (2 * E * SL + COLS + 4);
  static_assert(shared <= 227 * 1024, "staging buffers");
  auto kernel = matrix_memory_scan_kernel<E, SL, C, WIDE, THREADS>;
  if (shared > 48 * 1024) {
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (err != cudaSuccess) return (int)err;
  }
  launch_kernel(kernel, dim3(segments, p.heads, (p.vdim + 1 + COLS - 1) / COLS), dim3(THREADS), shared, stream, p);
  return launch_status();
}

// ------------------------------------------------------------------ chunks on the tensor cores
constexpr int CHUNK_COLS = 16;    // value channels of a block of the sequential kernel
constexpr int CHUNK_PITCH = CHUNK_COLS + 8;

__device__ __forceinline__ uint2 pack4(float4 x) { return make_uint2(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w)); }

// grid: (chunks, heads, segments)
template <int D>
__global__ void __launch_bounds__(128)
matrix_memory_pairs_kernel(MemoryArgs p) {
  constexpr int PITCH = D + 8;
  extern __shared__ __align__(16) uint8_t raw[];
  bf16* q_tile = reinterpret_cast<bf16*>(raw);               // [64][PITCH]
  bf16* k_tile = q_tile + CHUNK * PITCH;
  float (*decay)[CHUNK + 1] = reinterpret_cast<float (*)[CHUNK + 1]>(k_tile + CHUNK * PITCH);
  __shared__ float keep[CHUNK], write[CHUNK];
  const int head = blockIdx.y, seg = blockIdx.z, V = p.vdim;
  const int t0 = blockIdx.x * CHUNK, count = min(CHUNK, p.seg_q_len[seg] - t0);
  if (count <= 0) return;
  const size_t row0 = (size_t)p.seg_q_start[seg] + t0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_wait();
  if (threadIdx.x < CHUNK) {      // a place without a token keeps everything and writes nothing
    float2 gate = make_float2(1.f, 0.f);
    if (threadIdx.x < count) gate = __ldcg(reinterpret_cast<const float2*>(p.coef + (row0 + threadIdx.x) * p.heads + head));
    keep[threadIdx.x] = gate.x;
    write[threadIdx.x] = gate.y;
  }
  for (int idx = threadIdx.x; idx < CHUNK * (D / 4); idx += 128) {
    const int r = idx / (D / 4), d = (idx - r * (D / 4)) << 2;
    uint2 q2 = make_uint2(0u, 0u), k2 = q2;
    if (r < count) {
      const size_t at = (row0 + r) * p.heads * D + (size_t)head * D + d;
      q2 = pack4(__ldcg(reinterpret_cast<const float4*>(p.q + (row0 + r) * p.q_stride + (size_t)head * D + d)));
      k2 = pack4(__ldcg(reinterpret_cast<const float4*>(p.k + (row0 + r) * p.k_stride + (size_t)head * D + d)));
      *reinterpret_cast<uint2*>(p.q16 + at) = q2;
      *reinterpret_cast<uint2*>(p.k16 + at) = k2;
    }
    *reinterpret_cast<uint2*>(q_tile + r * PITCH + d) = q2;
    *reinterpret_cast<uint2*>(k_tile + r * PITCH + d) = k2;
  }
  for (int idx = threadIdx.x; idx < count * (V / 4); idx += 128) {
    const int r = idx / (V / 4), c = (idx - r * (V / 4)) << 2;
    *reinterpret_cast<uint2*>(p.v16 + (row0 + r) * p.heads * V + (size_t)head * V + c) =
        pack4(__ldcg(reinterpret_cast<const float4*>(p.v + (row0 + r) * p.v_stride + (size_t)head * V + c)));
  }
  __syncthreads();
  // a thread per column of D: its writing token's share at every later token
  if (threadIdx.x < CHUNK) {
    const int s = threadIdx.x;
    float x = write[s];
    for (int t = 0; t < CHUNK; ++t) {
      if (t > s) x *= keep[t];
      decay[t][s] = t >= s ? x : 0.f;
    }
    if (s < count) p.factors[(row0 + s) * p.heads + head].x = x;      // places behind the last token keep it
  } else if (threadIdx.x == CHUNK) {
    float x = 1.f;
    for (int t = 0; t < count; ++t) {
      x *= keep[t];
      p.factors[(row0 + t) * p.heads + head].y = x;
    }
  }
  uint32_t q_frag[D / 16][4];
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks)
    ldmatrix_x4(q_frag[ks], q_tile + (warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * PITCH + (ks * 2 + (lane >> 4)) * 8);
  float s[CHUNK / 8][4];
  padded_qk<D, CHUNK / 8>(s, q_frag, k_tile, lane);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = warp * 16 + (lane >> 2) + 8 * i;
    if (t >= count) continue;
    float* dst = p.pairs + ((row0 + t) * p.heads + head) * CHUNK;
#pragma unroll
    for (int j = 0; j < CHUNK / 8; ++j) {
      const int c = j * 8 + (lane & 3) * 2;
      *reinterpret_cast<float2*>(dst + c) = make_float2(s[j][2 * i] * decay[t][c], s[j][2 * i + 1] * decay[t][c + 1]);
    }
  }
}

// the three bfloat16 parts of a pair of numbers
__device__ __forceinline__ void split_pair(float x, float y, uint32_t* part) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 rounded = __floats2bfloat162_rn(x, y);
    part[i] = *reinterpret_cast<const uint32_t*>(&rounded);
    const float2 back = __bfloat1622float2(rounded);
    x -= back.x;
    y -= back.y;
  }
}

// c[0 .. 3] (four blocks of 8 columns) += a * tile, tile: 16 rows from `row` of a [..][CHUNK_PITCH] tile
__device__ __forceinline__ void mma_cols(float (*c)[4], const uint32_t* a, const bf16* tile, int row, int lane) {
#pragma unroll
  for (int dp = 0; dp < CHUNK_COLS / 16; ++dp) {
    uint32_t b[4];
    ldmatrix_x4_trans(b, tile + (row + (lane & 7) + (((lane >> 3) & 1) << 3)) * CHUNK_PITCH + (dp * 2 + (lane >> 4)) * 8);
    mma_bf16(c[2 * dp], a, b[0], b[1]);
    mma_bf16(c[2 * dp + 1], a, b[2], b[3]);
  }
}

// grid: (segments, heads, blocks of 16 state rows).  Warp w keeps the key channels w D / 4 .. of the state.
template <int D>
__global__ void __launch_bounds__(128)
matrix_memory_chunks_kernel(MemoryArgs p) {
  pdl_trigger();
  constexpr int PITCH = D + 8, MT = D / 64, NT = CHUNK_COLS / 8, PIECES = D / 8;
  extern __shared__ __align__(16) uint8_t raw[];
  bf16* qk_tiles = reinterpret_cast<bf16*>(raw);                       // 2 x (queries, keys) [64][PITCH]
  bf16* v_tiles = qk_tiles + 4 * CHUNK * PITCH;                         // 2 x [64][CHUNK_PITCH]
  bf16* s_parts = v_tiles + 2 * CHUNK * CHUNK_PITCH;                    // 3 x [D][CHUNK_PITCH]
  bf16* w_parts = s_parts + 3 * D * CHUNK_PITCH;                        // 3 x [64][CHUNK_PITCH]
  float2* factors = reinterpret_cast<float2*>(w_parts + 3 * CHUNK * CHUNK_PITCH);      // 2 x [64]
  const int seg = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * CHUNK_COLS, V = p.vdim;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q_start = p.seg_q_start[seg], q_len = p.seg_q_len[seg];
  float* state = p.states + ((size_t)p.seg_slot[seg] * p.heads + head) * (size_t)(V + 1) * D;
  // value channels beyond the last: the normaliser's is one, the others zero; no copy overwrites them
  for (int idx = threadIdx.x; idx < 2 * CHUNK * CHUNK_COLS; idx += 128) {
    const int r = idx / CHUNK_COLS, c = idx - r * CHUNK_COLS;
    if (col0 + c >= V) v_tiles[r * CHUNK_PITCH + c] = __float2bfloat16_rn(col0 + c == V ? 1.f : 0.f);
  }
  pdl_wait();
  auto stage = [&](int t0, int which) {
    const int count = min(CHUNK, q_len - t0);
    const size_t row0 = (size_t)q_start + t0;
    bf16* q_tile = qk_tiles + which * 2 * CHUNK * PITCH;
    bf16* k_tile = q_tile + CHUNK * PITCH;
    for (int idx = threadIdx.x; idx < CHUNK * PIECES; idx += 128) {
      const int r = idx / PIECES, c = (idx - r * PIECES) * 8;
      const bool valid = r < count;
      const size_t at = valid ? (row0 + r) * p.heads * D + (size_t)head * D + c : 0;
      cp_async_16(q_tile + r * PITCH + c, p.q16 + at, valid);
      cp_async_16(k_tile + r * PITCH + c, p.k16 + at, valid);
    }
    for (int idx = threadIdx.x; idx < CHUNK * (CHUNK_COLS / 8); idx += 128) {
      const int r = idx / (CHUNK_COLS / 8), c = (idx - r * (CHUNK_COLS / 8)) * 8;
      if (col0 + c >= V) continue;
      const bool valid = r < count;
      cp_async_16(v_tiles + (which * CHUNK + r) * CHUNK_PITCH + c,
                  p.v16 + (valid ? (row0 + r) * p.heads * V + (size_t)head * V + col0 + c : 0), valid);
    }
    if (threadIdx.x < CHUNK) {      // a place without a token writes nothing
      const bool valid = threadIdx.x < count;
      copy_async_8(factors + which * CHUNK + threadIdx.x, p.factors + (valid ? (row0 + threadIdx.x) * p.heads + head : 0), valid);
    }
    cp_async_commit();
  };
  stage(0, 0);
  float S[MT][NT][4];      // accumulators: key channel (row) lane / 4 + 8 (e / 2), value channel (column) 2 (lane % 4) + e % 2
  auto place = [&](int mt, int nt, int e, int* d, int* c) {
    *d = warp * (D / 4) + mt * 16 + (lane >> 2) + 8 * (e >> 1);
    *c = col0 + nt * 8 + (lane & 3) * 2 + (e & 1);
  };
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        int d, c;
        place(mt, nt, e, &d, &c);
        S[mt][nt][e] = c <= V ? __ldcg(state + (size_t)c * D + d) : 0.f;
      }
  int which = 0;
  for (int t0 = 0; t0 < q_len; t0 += CHUNK, which ^= 1) {
    const int count = min(CHUNK, q_len - t0);
    const size_t row0 = (size_t)q_start + t0;
    cp_async_wait<0>();
    __syncthreads();      // this chunk is here, and everybody is done with the one before
    if (t0 + CHUNK < q_len) stage(t0 + CHUNK, which ^ 1);
    const bf16* q_tile = qk_tiles + which * 2 * CHUNK * PITCH;
    const bf16* k_tile = q_tile + CHUNK * PITCH;
    const bf16* v_tile = v_tiles + which * CHUNK * CHUNK_PITCH;
    const float2* factor = factors + which * CHUNK;
    // this warp's rows of A, asked for early: keys up to the rows' own chunk part only
    const int r0 = warp * 16 + (lane >> 2);
    const float* a_row[2] = {p.pairs + ((row0 + r0) * p.heads + head) * CHUNK + (lane & 3) * 2,
                             p.pairs + ((row0 + r0 + 8) * p.heads + head) * CHUNK + (lane & 3) * 2};
    float2 a_pair[CHUNK / 16][4];
#pragma unroll
    for (int ks = 0; ks < CHUNK / 16; ++ks)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a_pair[ks][e] = make_float2(0.f, 0.f);
        if (ks <= warp && r0 + 8 * (e & 1) < count)
          a_pair[ks][e] = __ldcg(reinterpret_cast<const float2*>(a_row[e & 1] + ks * 16 + 8 * (e >> 1)));
      }
    // the state and the weighed values in parts
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          uint32_t part[3];
          split_pair(S[mt][nt][2 * i], S[mt][nt][2 * i + 1], part);
          int d, c;
          place(mt, nt, 2 * i, &d, &c);
#pragma unroll
          for (int n = 0; n < 3; ++n)
            *reinterpret_cast<uint32_t*>(s_parts + (n * D + d) * CHUNK_PITCH + (c - col0)) = part[n];
        }
    for (int idx = threadIdx.x; idx < CHUNK * (CHUNK_COLS / 2); idx += 128) {
      const int r = idx / (CHUNK_COLS / 2), c = (idx - r * (CHUNK_COLS / 2)) * 2;
      const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(v_tile + r * CHUNK_PITCH + c));
      const float weight = factor[r].x;
      uint32_t part[3];
      split_pair(weight * v.x, weight * v.y, part);
#pragma unroll
      for (int n = 0; n < 3; ++n) *reinterpret_cast<uint32_t*>(w_parts + (n * CHUNK + r) * CHUNK_PITCH + c) = part[n];
    }
    __syncthreads();
    // reads: of the state before the chunk, then of the chunk's own tokens; a sum per part (short chains of products)
    float o[3][NT][4];
#pragma unroll
    for (int n = 0; n < 3; ++n)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) o[n][nt][0] = o[n][nt][1] = o[n][nt][2] = o[n][nt][3] = 0.f;
    if (warp * 16 < count) {
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t a[4];
        ldmatrix_x4(a, q_tile + (warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * PITCH + (ks * 2 + (lane >> 4)) * 8);
#pragma unroll
        for (int n = 0; n < 3; ++n) mma_cols(o[n], a, s_parts + n * D * CHUNK_PITCH, ks * 16, lane);
      }
      const float before[2] = {factor[r0].y, factor[r0 + 8].y};
#pragma unroll
      for (int n = 0; n < 3; ++n)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[n][nt][e] *= before[e >> 1];
#pragma unroll
      for (int ks = 0; ks < CHUNK / 16; ++ks) {
        if (ks > warp) continue;
        uint32_t part[4][3];
#pragma unroll
        for (int e = 0; e < 4; ++e) split_pair(a_pair[ks][e].x, a_pair[ks][e].y, part[e]);
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          const uint32_t a[4] = {part[0][n], part[1][n], part[2][n], part[3][n]};
          mma_cols(o[n], a, v_tile, ks * 16, lane);
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[0][nt][e] += o[1][nt][e] + o[2][nt][e];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (r0 + 8 * i >= count) continue;
        const size_t row_head = (row0 + r0 + 8 * i) * p.heads + head;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const int c = col0 + nt * 8 + (lane & 3) * 2;
          if (c < V)
            *reinterpret_cast<float2*>(p.reads + row_head * V + c) = make_float2(o[0][nt][2 * i] * p.q_scale, o[0][nt][2 * i + 1] * p.q_scale);
          else if (c == V)
            p.norms[row_head] = o[0][nt][2 * i] * p.q_scale;
        }
      }
    }
    // the state behind the chunk
    const float kept = factor[count - 1].y;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[mt][nt][e] *= kept;
#pragma unroll
      for (int ks = 0; ks < CHUNK / 16; ++ks) {
        uint32_t a[4];      // keys transposed: channels are the product's rows
        ldmatrix_x4_trans(a, k_tile + (ks * 16 + ((lane >> 4) << 3) + (lane & 7)) * PITCH + warp * (D / 4) + mt * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int n = 2; n >= 0; --n) mma_cols(S[mt], a, w_parts + n * CHUNK * CHUNK_PITCH, ks * 16, lane);
      }
    }
  }
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        int d, c;
        place(mt, nt, e, &d, &c);
        if (c <= V) state[(size_t)c * D + d] = S[mt][nt][e];
      }
}

template <int D>
static int launch_chunks(const MemoryArgs& p, int segments, int max_q_len, cudaStream_t stream) {
  constexpr size_t shared = sizeof(bf16) * (size_t)(4 * CHUNK * (D + 8) + (2 * CHUNK + 3 * D + 3 * CHUNK) * CHUNK_PITCH) +
                            sizeof(float2) * 2 * CHUNK;
  static_assert(shared <= 227 * 1024, "tiles");
  constexpr size_t pairs_shared = sizeof(bf16) * (size_t)(2 * CHUNK * (D + 8)) + sizeof(float) * CHUNK * (CHUNK + 1);
  cudaError_t err = cudaFuncSetAttribute(matrix_memory_chunks_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute(matrix_memory_pairs_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pairs_shared);
  if (err != cudaSuccess) return (int)err;
  launch_kernel(matrix_memory_pairs_kernel<D>, dim3((max_q_len + CHUNK - 1) / CHUNK, p.heads, segments), dim3(128), pairs_shared,
                stream, p);
  const int status = launch_status();
  if (status != MLR_OK) return status;
  launch_kernel(matrix_memory_chunks_kernel<D>, dim3(segments, p.heads, (p.vdim + CHUNK_COLS) / CHUNK_COLS), dim3(128), shared, stream, p);
  return launch_status();
}

// ------------------------------------------------------------------ chunks side by side
// Bound by the tensor cores' rate for three products of parts with a warp's instructions between them: a block of the outputs took some 23,000
// cycles alone on an SM (before the leading products had a sum of their own, 2 us of a call), of which 8,500 were the products with the state before (loads, split
// and products of a part after another), 3,000 the chunk's own tokens and 6,500 normaliser, norm and gate; the ends 10,000, 4,100 of them products.  The carry moves
// the states of all chunks through L2.
// 16 warps of half the columns each were slower (splits and fragments of A twice: 56 -> 61 us at the time), a branch around a pair that a warp does not have cost
// 10 % of the products, and rows one after the other with their divisions and roots 4,500 cycles.  Repeated calls, chunks one behind the other (2,048 and 4,000 rows
// in parts of four and more, which these kernels replace) / side by side, 7 heads of 128 x 128: 1,300 and 748 rows 90 / 48 us, 2,048 rows 83 / 49, 4,000 rows 154 / 81,
// 512 rows 41 / 28; 16 heads: 2,048 rows 149 / 91; from a flushed L2 8 of 200 rows 112 / 94.
constexpr int SIDE_THREADS = 256;
constexpr int SIDE_V = 128;               // value channels at most
constexpr int SIDE_PAIRS = SIDE_V / 16 + 1;      // pairs of eight columns, the normaliser's among them
constexpr int SIDE_PITCH = 16 * SIDE_PAIRS + 8;  // rows of value columns: an odd number of 16-byte pieces

// Column pairs of a head: its value channels, the normaliser and zeros.
__host__ __device__ __forceinline__ int side_pairs(int V) { return (V / 8 + 2) / 2; }
// A token's gates: keep and write; a place without a token keeps everything and writes nothing.
__device__ __forceinline__ void side_gates(const MemoryArgs& p, float* keep, float* write, float* floor_of, size_t row0, int count, int head) {
  const int t = threadIdx.x;
  if (t >= CHUNK) return;
  float4 gate = make_float4(1.f, 0.f, 0.f, 0.f);
  if (t < count) gate = __ldcg(p.coef + (row0 + t) * p.heads + head);
  keep[t] = gate.x;
  write[t] = gate.y;
  if (floor_of != nullptr) floor_of[t] = gate.z;
}

// A chunk's rows of float32 numbers, asked for with all loads in flight together and kept as bfloat16: COLUMNS pieces of four, `used` of them
// (and `rows` of the rows) are there, PER of them a thread's.
template <int COLUMNS, int THREADS>
struct SideRows {
  static constexpr int PER = (CHUNK * COLUMNS + THREADS - 1) / THREADS;
  float4 piece[PER];
  __device__ __forceinline__ void ask(const float* from, long long stride, int rows, int used) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int idx = threadIdx.x + i * THREADS, r = idx / COLUMNS, c = idx % COLUMNS;
      piece[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && c < used) piece[i] = __ldcg(reinterpret_cast<const float4*>(from + r * stride) + c);
    }
  }
  template <typename F>
  __device__ __forceinline__ void each(F&& f) {      // f(row, first column, numbers)
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int idx = threadIdx.x + i * THREADS;
      if (idx < CHUNK * COLUMNS) f(idx / COLUMNS, idx % COLUMNS * 4, piece[i]);
    }
  }
};

// A warp takes 16 key channels and its share of the column pairs.  SINGLES: behind the chunks' blocks come those of single rows, which keep the state in device
// memory: as chunks of one row each of their states went through memory four times instead of two, and took a state's scratch.  (A kernel of its own: where no
// block goes there, the branch alone cost 7 heads, 600 rows and four of 64, 42 -> 49 us.)  grid: (heads, chunks [+ segments])
template <int D, int PAIRS, bool SINGLES>
__global__ void __launch_bounds__(SIDE_THREADS, 2)
memory_ends_kernel(MemoryArgs p, bf16* out, int chunks) {
  constexpr int PITCH = D + 8, W_APART = CHUNK * SIDE_PITCH, KEY_TILES = D / 16;
  constexpr int GROUPS = SIDE_THREADS / 32 / KEY_TILES, MOST = (PAIRS + GROUPS - 1) / GROUPS;      // of column pairs, and pairs of a group
  extern __shared__ __align__(16) uint8_t raw[];
  bf16 *k_tile = reinterpret_cast<bf16*>(raw), *w_parts = k_tile + CHUNK * PITCH;      // [64][PITCH], 3 x [64][SIDE_PITCH]
  __shared__ float keep[CHUNK], write[CHUNK], share[CHUNK], kept;
  if (SINGLES && (int)blockIdx.y >= chunks) {
    static_assert(SIDE_THREADS == DECODE_THREADS, "single rows");
    decode_row<bf16, 1, true>(p, out, reinterpret_cast<float*>(raw), blockIdx.y - chunks, blockIdx.x);
    return;
  }
  pdl_wait();
  const int head = blockIdx.x, V = p.vdim, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.y);
  if (seg < 0) return;
  const int count = min(CHUNK, length - chunk * CHUNK);
  const size_t row0 = (size_t)start + chunk * CHUNK;
  side_gates(p, keep, write, nullptr, row0, count, head);
  SideRows<D / 4, SIDE_THREADS> keys;
  keys.ask(p.k + row0 * p.k_stride + (size_t)head * D, p.k_stride, count, D / 4);
  SideRows<4 * PAIRS, SIDE_THREADS> values;
  values.ask(p.v + row0 * p.v_stride + (size_t)head * V, p.v_stride, count, V / 4);
  __syncthreads();
  if (warp == 0) {      // what the chunk's last token has of each, two to a lane: places behind the last token keep it
    const float near = keep[2 * lane], far = keep[2 * lane + 1];
    float all = near * far;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const float later = __shfl_down_sync(0xffffffffu, all, offset);
      if (lane + offset < 32) all *= later;
    }
    float behind = __shfl_down_sync(0xffffffffu, all, 1);
    if (lane == 31) behind = 1.f;
    share[2 * lane + 1] = write[2 * lane + 1] * behind;
    share[2 * lane] = write[2 * lane] * (far * behind);
    if (lane == 0) p.spans[(size_t)blockIdx.y * p.heads + head] = kept = all;
  }
  keys.each([&](int r, int d, const float4& x) { *reinterpret_cast<uint2*>(k_tile + r * PITCH + d) = pack4(x); });
  __syncthreads();
  values.each([&](int r, int c, const float4& x) {
    const float weight = share[r];
    const uint2 rounded = pack4(x);
    float4 v = make_float4(weight * __uint_as_float(rounded.x << 16), weight * __uint_as_float(rounded.x & 0xffff0000u),
                           weight * __uint_as_float(rounded.y << 16), weight * __uint_as_float(rounded.y & 0xffff0000u));
    if (c >= V) v = make_float4(c == V ? weight : 0.f, 0.f, 0.f, 0.f);
    uint32_t low[3], high[3];
    split_pair(v.x, v.y, low);
    split_pair(v.z, v.w, high);
#pragma unroll
    for (int n = 0; n < 3; ++n) *reinterpret_cast<uint2*>(w_parts + n * W_APART + r * SIDE_PITCH + c) = make_uint2(low[n], high[n]);
  });
  __syncthreads();
  float E[2 * MOST][4];
#pragma unroll
  for (int j = 0; j < 2 * MOST; ++j) E[j][0] = E[j][1] = E[j][2] = E[j][3] = 0.f;
  const int tile = warp % KEY_TILES, all_pairs = side_pairs(V), share_of = (all_pairs + GROUPS - 1) / GROUPS;
  const int pair0 = warp / KEY_TILES * share_of, pairs = min(share_of, all_pairs - pair0);
#pragma unroll
  for (int ks = 0; ks < CHUNK / 16; ++ks) {
    if (ks * 16 >= count) break;
    uint32_t a[4];      // keys transposed: channels are the product's rows
    ldmatrix_x4_trans(a, k_tile + (ks * 16 + ((lane >> 4) << 3) + (lane & 7)) * PITCH + tile * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
    for (int n = 2; n >= 0; --n)
#pragma unroll
      for (int j = 0; j < MOST; ++j) {      // a pair beyond the last is multiplied and dropped: a branch here would keep loads and products apart
        uint32_t b[4];
        ldmatrix_x4_trans(b, w_parts + n * W_APART + (ks * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * SIDE_PITCH +
                                 (min(pair0 + j, PAIRS - 1) * 2 + (lane >> 4)) * 8);
        mma_bf16(E[2 * j], a, b[0], b[1]);
        mma_bf16(E[2 * j + 1], a, b[2], b[3]);
      }
  }
  const int c0 = pair0 * 16 + (lane & 3) * 2;
  const size_t mine = (size_t)c0 * D + tile * 16 + (lane >> 2);
  float* to = p.ends + ((size_t)blockIdx.y * p.heads + head) * (size_t)(V + 1) * D + mine;
  float* state = p.states + ((size_t)slot * p.heads + head) * (size_t)(V + 1) * D + mine;
  auto entry = [&](int j, int e) { return (j * 8 + (e & 1)) * D + 8 * (e >> 1); };
  auto there = [&](int j, int e) { return j < 2 * pairs && c0 + j * 8 + (e & 1) <= V; };
  if (length > CHUNK) {
#pragma unroll
    for (int j = 0; j < 2 * MOST; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (there(j, e)) to[entry(j, e)] = E[j][e];
    pdl_trigger();      // late, as in the kernel behind
    return;
  }
  // the segment's only chunk: nothing is left for the carry
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float before[MOST][4];
#pragma unroll
    for (int j = 0; j < MOST; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (there(half * MOST + j, e)) before[j][e] = __ldcg(state + entry(half * MOST + j, e));
#pragma unroll
    for (int j = 0; j < MOST; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (there(half * MOST + j, e)) {
          to[entry(half * MOST + j, e)] = before[j][e];
          state[entry(half * MOST + j, e)] = fmaf(kept, before[j][e], E[half * MOST + j][e]);
        }
  }
}

// A thread owns four neighbouring entries and takes the chunks of its segment in order, BATCH of them asked for together.  Leaves the state before
// every chunk where what its tokens left behind was.  grid: (entries, segments)
__global__ void __launch_bounds__(256)
memory_carry_kernel(MemoryArgs p, int cells) {
  constexpr int BATCH = 8;
  pdl_wait();
  const int seg = blockIdx.y, length = p.seg_q_len[seg], at = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (length <= CHUNK) return;
  int first = 0;
  for (int i = threadIdx.x & 31; i < seg; i += 32) first += p.seg_q_len[i] < p.least ? 0 : (p.seg_q_len[i] + CHUNK - 1) / CHUNK;
  first = __reduce_add_sync(0xffffffffu, first);
  if (at >= p.heads * cells) return;
  const int head = at / cells, cell = at - head * cells, chunks = (length + CHUNK - 1) / CHUNK;
  float4* state = reinterpret_cast<float4*>(p.states + ((size_t)p.seg_slot[seg] * p.heads + head) * cells + cell);
  float4 S = *state;
  const size_t step = (size_t)p.heads * cells / 4;
  float4* end = reinterpret_cast<float4*>(p.ends + ((size_t)first * p.heads + head) * cells + cell);
  const float* span = p.spans + (size_t)first * p.heads + head;
  for (int c0 = 0; c0 < chunks; c0 += BATCH, end += BATCH * step, span += BATCH * p.heads) {
    float4 own[BATCH];
    float g[BATCH];
#pragma unroll
    for (int k = 0; k < BATCH; ++k)
      if (c0 + k < chunks) {
        own[k] = end[k * step];
        g[k] = span[k * p.heads];
      }
#pragma unroll
    for (int k = 0; k < BATCH; ++k)
      if (c0 + k < chunks) {
        end[k * step] = S;
        S.x = fmaf(g[k], S.x, own[k].x);
        S.y = fmaf(g[k], S.y, own[k].y);
        S.z = fmaf(g[k], S.z, own[k].z);
        S.w = fmaf(g[k], S.w, own[k].w);
      }
  }
  *state = S;
  // The outputs' blocks, brought in while these still fill some SMs, would land two to an SM beside empty ones: a step of 512 rows, 7 heads, takes
  // 34.8 us with the trigger in front, 26.6 so, and one of 2,048 rows 50.4 and (with that of the ends) 45.6.
  pdl_trigger();
}

constexpr int SIDE_D = 32;                // key channels of the state taken at a time
constexpr int SIDE_D_PITCH = SIDE_D + 8;
constexpr int SIDE_A_PITCH = CHUNK + 8;
// Sums of the outputs: the leading part's products in an accumulator of their own; the smaller ones' sums of 32 key channels (16 tokens) are added with
// what the leading sum's steps dropped on average (with_dropped).  Sums that cancel to some 2^-18 of their products, heads of 128 (64), errors with one chunk
// behind the other / all in one accumulator / so: reads of the state 1.23e-2 (0.66e-2) / 5.9e-2 (3.5e-2) / 0.99e-2 (0.66e-2), with tokens 3.1e-2 (2.3e-2) /
// 13.5e-2 (10.2e-2) / 2.8e-2 (2.1e-2); 0.0 and 0.0 give 1.39e-2 (0.80e-2) and 3.3e-2 (2.7e-2).  1,300 and 748 rows of 7
// heads: 48.3 us in one accumulator, 50.4 so.
constexpr float STATE_DROPPED = 0.6f, TOKENS_DROPPED = 0.25f;
constexpr int SIDE_LOW = 2;               // column pairs whose smaller products are summed at a time
constexpr int SIDE_SUMS = SIDE_V + 8;     // float32 sums of a row, the normaliser among them

template <int D>
struct SideShape {
  static constexpr int QK_PITCH = D + 8, S_APART = 16 * SIDE_PAIRS * SIDE_D_PITCH;
  static constexpr size_t Q = CHUNK * QK_PITCH * sizeof(bf16), VALUES = CHUNK * SIDE_PITCH * sizeof(bf16), A = CHUNK * SIDE_A_PITCH * sizeof(float);
  static constexpr size_t S = 3 * S_APART * sizeof(bf16);      // keys before
  static_assert(S >= Q && A + S >= CHUNK * SIDE_SUMS * sizeof(float), "keys, sums");
  static constexpr size_t SHARED = Q + VALUES + A + S;
  static constexpr size_t ENDS = Q + 3 * CHUNK * SIDE_PITCH * sizeof(bf16);
};

// Warps 4 i .. 4 i + 3 take 16 rows each with the i-th share of the column pairs (of the tokens for A).  grid: (heads, chunks)
template <int D, int PAIRS>
__global__ void __launch_bounds__(SIDE_THREADS, 2)
memory_outputs_kernel(MemoryArgs p, bf16* __restrict__ out) {
  using Shape = SideShape<D>;
  constexpr int PITCH = Shape::QK_PITCH, SIDES = SIDE_THREADS / 128, MOST = (PAIRS + SIDES - 1) / SIDES;      // column pairs of a warp
  extern __shared__ __align__(16) uint8_t raw[];
  bf16 *q_tile = reinterpret_cast<bf16*>(raw), *v_tile = q_tile + CHUNK * PITCH;
  float* A = reinterpret_cast<float*>(raw + Shape::Q + Shape::VALUES);                      // [64][SIDE_A_PITCH]
  bf16* s_parts = reinterpret_cast<bf16*>(raw + Shape::Q + Shape::VALUES + Shape::A);      // 3 x [columns][SIDE_D_PITCH]; keys before
  bf16* k_tile = s_parts;
  __shared__ __align__(16) float keep[CHUNK];
  __shared__ float write[CHUNK], floor_of[CHUNK], since[CHUNK];
  pdl_wait();
  const int head = blockIdx.x, V = p.vdim, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.y);
  if (seg < 0) return;
  const int count = min(CHUNK, length - chunk * CHUNK);
  const size_t row0 = (size_t)start + chunk * CHUNK;
  side_gates(p, keep, write, floor_of, row0, count, head);
  {
    SideRows<D / 4, SIDE_THREADS> queries, keys;
    queries.ask(p.q + row0 * p.q_stride + (size_t)head * D, p.q_stride, count, D / 4);
    keys.ask(p.k + row0 * p.k_stride + (size_t)head * D, p.k_stride, count, D / 4);
    queries.each([&](int r, int d, const float4& x) { *reinterpret_cast<uint2*>(q_tile + r * PITCH + d) = pack4(x); });
    keys.each([&](int r, int d, const float4& x) { *reinterpret_cast<uint2*>(k_tile + r * PITCH + d) = pack4(x); });
  }
  SideRows<4 * PAIRS, SIDE_THREADS> values;      // on their way until the products of queries and keys are done
  values.ask(p.v + row0 * p.v_stride + (size_t)head * V, p.v_stride, count, V / 4);
  const int all_pairs = side_pairs(V);
  // a part of the state before the chunk
  const float* before = p.ends + ((size_t)blockIdx.y * p.heads + head) * (size_t)(V + 1) * D;
  constexpr int S_PIECES = (16 * PAIRS * (SIDE_D / 4) + SIDE_THREADS - 1) / SIDE_THREADS;
  float4 piece[S_PIECES];
  auto ask = [&](int d0) {
#pragma unroll
    for (int k = 0; k < S_PIECES; ++k) {
      const int idx = threadIdx.x + k * SIDE_THREADS, c = idx / (SIDE_D / 4), d = idx % (SIDE_D / 4) * 4;
      piece[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c <= V) piece[k] = __ldcg(reinterpret_cast<const float4*>(before + (size_t)c * D + d0 + d));
    }
  };
  ask(0);
  __syncthreads();
  {      // thread (s, quarter): token s's share at the quarter's rows
    constexpr int ROWS = CHUNK * CHUNK / SIDE_THREADS;
    const int s = threadIdx.x & (CHUNK - 1), t0 = threadIdx.x / CHUNK * ROWS;
    float x = write[s], all = 1.f;
    auto four = [&](int t, auto&& at) {
      const float4 k4 = *reinterpret_cast<const float4*>(keep + t);
      const float own[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (t + i > s) x *= own[i];
        all *= own[i];
        at(t + i);
      }
    };
#pragma unroll 4
    for (int t = 0; t < t0; t += 4) four(t, [](int) {});
#pragma unroll
    for (int t = 0; t < ROWS; t += 4)
      four(t0 + t, [&](int row) {
        A[row * SIDE_A_PITCH + s] = row >= s ? x : 0.f;
        if (s == 0) since[row] = all;
      });
  }
  const int tile = warp & 3, side = warp >> 2, r = lane >> 2, c2 = (lane & 3) * 2;
  const bf16* q_at = q_tile + (tile * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * PITCH + (lane >> 4) * 8;
  constexpr int BLOCKS = 4 / SIDES;      // blocks of 16 tokens of a warp; those behind its rows are not seen
  float s[BLOCKS][2][4];
#pragma unroll
  for (int n = 0; n < BLOCKS; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[n][0][e] = s[n][1][e] = 0.f;
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    uint32_t a[4];
    ldmatrix_x4(a, q_at + ks * 16);
#pragma unroll
    for (int n = 0; n < BLOCKS; ++n)
      {
        uint32_t b[4];
        ldmatrix_x4(b, k_tile + ((n * SIDES + side) * 16 + (lane & 7) + ((lane >> 4) << 3)) * PITCH + ks * 16 + ((lane >> 3) & 1) * 8);
        mma_bf16(s[n][0], a, b[0], b[1]);
        mma_bf16(s[n][1], a, b[2], b[3]);
      }
  }
  __syncthreads();      // the shares are there, the keys have been read
#pragma unroll
  for (int n = 0; n < BLOCKS; ++n)
    if (n * SIDES + side <= tile) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int row = tile * 16 + r + 8 * i, token = (n * SIDES + side) * 16 + j * 8 + c2;      // later tokens are not seen, whatever numbers they hold
          float2* at = reinterpret_cast<float2*>(A + row * SIDE_A_PITCH + token);
          const float2 d = *at;
          *at = make_float2(token <= row ? s[n][j][2 * i] * d.x : 0.f, token < row ? s[n][j][2 * i + 1] * d.y : 0.f);
        }
    }
  values.each([&](int row, int c, const float4& x) {
    *reinterpret_cast<uint2*>(v_tile + row * SIDE_PITCH + c) = c < V ? pack4(x) : make_uint2(c == V ? 0x3f80u : 0u, 0u);      // the normaliser's value is one
  });
  const int share_of = (all_pairs + SIDES - 1) / SIDES, pair0 = side * share_of, pairs = min(share_of, all_pairs - pair0);
  float o[2 * MOST][4];
#pragma unroll
  for (int j = 0; j < 2 * MOST; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
#pragma unroll 1
  for (int d0 = 0; d0 < D; d0 += SIDE_D) {
    if (d0 > 0) __syncthreads();      // the part before has been read
#pragma unroll
    for (int k = 0; k < S_PIECES; ++k) {
      const int idx = threadIdx.x + k * SIDE_THREADS, c = idx / (SIDE_D / 4), d = idx % (SIDE_D / 4) * 4;
      if (c >= 16 * PAIRS) continue;
      uint32_t first[3], second[3];
      split_pair(piece[k].x, piece[k].y, first);
      split_pair(piece[k].z, piece[k].w, second);
#pragma unroll
      for (int n = 0; n < 3; ++n) *reinterpret_cast<uint2*>(s_parts + n * Shape::S_APART + c * SIDE_D_PITCH + d) = make_uint2(first[n], second[n]);
    }
    __syncthreads();
    if (d0 + SIDE_D < D) ask(d0 + SIDE_D);
    if (tile * 16 < count) {
      uint32_t a[SIDE_D / 16][4];
#pragma unroll
      for (int ks = 0; ks < SIDE_D / 16; ++ks) ldmatrix_x4(a[ks], q_at + d0 + ks * 16);
#pragma unroll
      for (int j0 = 0; j0 < MOST; j0 += SIDE_LOW) {
        float low[2 * SIDE_LOW][4] = {};
#pragma unroll
        for (int ks = 0; ks < SIDE_D / 16; ++ks)
#pragma unroll
          for (int n = 2; n >= 0; --n)
#pragma unroll
            for (int j = j0; j < j0 + SIDE_LOW && j < MOST; ++j) {
              uint32_t b[4];
              ldmatrix_x4(b, s_parts + n * Shape::S_APART + (min(pair0 + j, PAIRS - 1) * 16 + (lane & 7) + ((lane >> 4) << 3)) * SIDE_D_PITCH + ks * 16 +
                                 ((lane >> 3) & 1) * 8);
              float (*sum)[4] = n > 0 ? low + 2 * (j - j0) : o + 2 * j;
              mma_bf16(sum[0], a[ks], b[0], b[1]);
              mma_bf16(sum[1], a[ks], b[2], b[3]);
            }
#pragma unroll
        for (int i = 0; i < 2 * SIDE_LOW && 2 * j0 + i < 2 * MOST; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[2 * j0 + i][e] += with_dropped(o[2 * j0 + i][e], low[i][e], STATE_DROPPED);
      }
    }
  }
  const float kept[2] = {since[tile * 16 + r], since[tile * 16 + r + 8]};
#pragma unroll
  for (int j = 0; j < 2 * MOST; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] *= kept[e >> 1];
  if (tile * 16 < count) {
#pragma unroll 1
    for (int ks = 0; ks <= tile; ++ks) {      // the chunk's own tokens; later ones are not seen
      uint32_t part[4][3];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = *reinterpret_cast<const float2*>(A + (tile * 16 + r + 8 * (e & 1)) * SIDE_A_PITCH + ks * 16 + 8 * (e >> 1) + c2);
        split_pair(x.x, x.y, part[e]);
      }
#pragma unroll
      for (int j0 = 0; j0 < MOST; j0 += SIDE_LOW) {
        float low[2 * SIDE_LOW][4] = {};
        uint32_t b[SIDE_LOW][4];
#pragma unroll
        for (int n = 2; n >= 0; --n)
#pragma unroll
          for (int j = j0; j < j0 + SIDE_LOW && j < MOST; ++j) {
            if (n == 2)
              ldmatrix_x4_trans(b[j - j0], v_tile + (ks * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * SIDE_PITCH + (min(pair0 + j, PAIRS - 1) * 2 + (lane >> 4)) * 8);
            const uint32_t a[4] = {part[0][n], part[1][n], part[2][n], part[3][n]};
            float (*sum)[4] = n > 0 ? low + 2 * (j - j0) : o + 2 * j;
            mma_bf16(sum[0], a, b[j - j0][0], b[j - j0][1]);
            mma_bf16(sum[1], a, b[j - j0][2], b[j - j0][3]);
          }
#pragma unroll
        for (int i = 0; i < 2 * SIDE_LOW && 2 * j0 + i < 2 * MOST; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[2 * j0 + i][e] += with_dropped(o[2 * j0 + i][e], low[i][e], TOKENS_DROPPED);
      }
    }
  }
  // Normaliser, head norm, weight and gate: a warp takes ROWS rows, its lanes the channels; what a row needs once, a lane works out for each row.
  // No branches between the rows (those behind the last are dropped when they are stored), or each waits for the one before.
  __syncthreads();      // A has been read
  float* sums = A;      // [64][SIDE_SUMS]
#pragma unroll
  for (int j = 0; j < 2 * MOST; ++j) {
    const int c = pair0 * 16 + j * 8 + c2;
    if (j < 2 * pairs && c <= V) {
#pragma unroll
      for (int i = 0; i < 2; ++i) *reinterpret_cast<float2*>(sums + (tile * 16 + r + 8 * i) * SIDE_SUMS + c) = make_float2(o[j][2 * i], o[j][2 * i + 1]);
    }
  }
  constexpr int ROWS = CHUNK / (SIDE_THREADS / 32), COLUMNS = SIDE_V / 32;      // rows of a warp, channels of a lane
  const int first = warp * ROWS;
  const bool full = V == SIDE_V && first + ROWS <= count;
  const float* gate_at = p.gate + (row0 + first) * p.gate_stride + (size_t)head * V + lane;
  float gate[ROWS][COLUMNS], weight[COLUMNS], x[ROWS][COLUMNS], sq[ROWS];
#pragma unroll
  for (int j = 0; j < COLUMNS; ++j) weight[j] = lane + 32 * j < V ? p.weight[(size_t)head * V + lane + 32 * j] : 0.f;
#pragma unroll
  for (int i = 0; i < ROWS; ++i)
#pragma unroll
    for (int j = 0; j < COLUMNS; ++j) gate[i][j] = full || (first + i < count && lane + 32 * j < V) ? __ldcg(gate_at + i * p.gate_stride + 32 * j) : 0.f;
  __syncthreads();
  const int own_row = first + (lane & (ROWS - 1));
  const float own_scale = p.q_scale / (fmaxf(fabsf(sums[own_row * SIDE_SUMS + V] * p.q_scale), floor_of[own_row]) + p.guard);
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const float scale = __shfl_sync(0xffffffffu, own_scale, i);
    sq[i] = 0.f;
#pragma unroll
    for (int j = 0; j < COLUMNS; ++j) {
      x[i][j] = lane + 32 * j < V ? sums[(first + i) * SIDE_SUMS + lane + 32 * j] * scale : 0.f;
      sq[i] = fmaf(x[i][j], x[i][j], sq[i]);
    }
  }
  float own_sq = 0.f;
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1)
#pragma unroll
    for (int i = 0; i < ROWS; ++i) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], offset);
#pragma unroll
  for (int i = 0; i < ROWS; ++i)
    if ((lane & (ROWS - 1)) == i) own_sq = sq[i];
  const float own_factor = 1.f / sqrtf(own_sq / (float)V + p.eps);
  bf16* dst = out + ((row0 + first) * p.heads + head) * V + lane;
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const float factor = __shfl_sync(0xffffffffu, own_factor, i);
#pragma unroll
    for (int j = 0; j < COLUMNS; ++j) {
      const bf16 y = __float2bfloat16(x[i][j] * factor * weight[j] * sigmoid(gate[i][j]));
      if (full || (first + i < count && lane + 32 * j < V)) dst[(size_t)i * p.heads * V + 32 * j] = y;
    }
  }
  pdl_trigger();
}

template <int D, int PAIRS>
static int launch_side(const MemoryArgs& p, bf16* out, int chunks, int segments, cudaStream_t stream) {
  const int cells = (p.vdim + 1) * D;
  auto ends = p.least > 1 ? memory_ends_kernel<D, PAIRS, true> : memory_ends_kernel<D, PAIRS, false>;
  static OncePerDevice once;
  const cudaError_t err = once([] {
    cudaError_t err = cudaFuncSetAttribute(memory_outputs_kernel<D, PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SideShape<D>::SHARED);
    for (auto kernel : {memory_ends_kernel<D, PAIRS, true>, memory_ends_kernel<D, PAIRS, false>})
      if (err == cudaSuccess) err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SideShape<D>::ENDS);
    return err;
  });
  if (err != cudaSuccess) return (int)err;
  launch_kernel(ends, dim3(p.heads, chunks + (p.least > 1 ? segments : 0)), dim3(SIDE_THREADS), SideShape<D>::ENDS, stream, p, out, chunks);
  int status = launch_status();
  if (status != MLR_OK) return status;
  launch_kernel(memory_carry_kernel, dim3((p.heads * cells / 4 + 255) / 256, segments), dim3(256), 0, stream, p, cells);
  if ((status = launch_status()) != MLR_OK) return status;
  launch_kernel(memory_outputs_kernel<D, PAIRS>, dim3(p.heads, chunks), dim3(SIDE_THREADS), SideShape<D>::SHARED, stream, p, out);
  return launch_status();
}

// ------------------------------------------------------------------ normaliser, head norm, weight, gate
__device__ __forceinline__ void store4(float* dst, float4 y) { *reinterpret_cast<float4*>(dst) = y; }
__device__ __forceinline__ void store4(bf16* dst, float4 y) { *reinterpret_cast<uint2*>(dst) = pack4(y); }

// A warp per (row, head).  WIDE: at most 256 channels, in pieces of four (sizes, strides and pointers allow it).
template <typename T, bool WIDE>
__global__ void __launch_bounds__(128)
matrix_memory_finish_kernel(MemoryArgs p, T* __restrict__ out, long long items) {
  pdl_trigger();
  pdl_wait();
  const long long item = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= items) return;
  const int lane = threadIdx.x & 31, V = p.vdim;
  const long long row = item / p.heads;
  const int head = (int)(item - row * p.heads);
  const float* reads = p.reads + item * V;
  const float* gate = p.gate + row * p.gate_stride + (size_t)head * V;
  const float* weight = p.weight + (size_t)head * V;
  const float inverse = 1.f / (fmaxf(fabsf(__ldcg(p.norms + item)), __ldcg(&p.coef[item].z)) + p.guard);
  if (WIDE) {
    float4 o[2], g[2];
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = (lane + 32 * j) * 4;
      o[j] = g[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < V) {
        o[j] = __ldcg(reinterpret_cast<const float4*>(reads + c));
        g[j] = __ldcg(reinterpret_cast<const float4*>(gate + c));
      }
      o[j].x *= inverse; o[j].y *= inverse; o[j].z *= inverse; o[j].w *= inverse;
      sq += fmaf(o[j].x, o[j].x, o[j].y * o[j].y) + fmaf(o[j].z, o[j].z, o[j].w * o[j].w);
    }
    const float factor = 1.f / sqrtf(warp_sum(sq) / (float)V + p.eps);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = (lane + 32 * j) * 4;
      if (c >= V) continue;
      const float4 w = *reinterpret_cast<const float4*>(weight + c);
      store4(out + item * V + c, make_float4(o[j].x * factor * w.x * sigmoid(g[j].x), o[j].y * factor * w.y * sigmoid(g[j].y),
                                             o[j].z * factor * w.z * sigmoid(g[j].z), o[j].w * factor * w.w * sigmoid(g[j].w)));
    }
    return;
  }
  constexpr int HELD = 8;      // channels a lane keeps in registers
  float o[HELD], g[HELD], sq = 0.f;
#pragma unroll
  for (int j = 0; j < HELD; ++j) {
    const int c = lane + 32 * j;
    o[j] = c < V ? __ldcg(reads + c) * inverse : 0.f;
    g[j] = c < V ? __ldcg(gate + c) : 0.f;
    sq = fmaf(o[j], o[j], sq);
  }
  for (int c = lane + 32 * HELD; c < V; c += 32) {
    const float x = __ldcg(reads + c) * inverse;
    sq = fmaf(x, x, sq);
  }
  const float factor = 1.f / sqrtf(warp_sum(sq) / (float)V + p.eps);
  T* dst = out + item * V;
#pragma unroll
  for (int j = 0; j < HELD; ++j) {
    const int c = lane + 32 * j;
    if (c < V) dst[c] = from_float<T>(o[j] * factor * weight[c] * sigmoid(g[j]));
  }
  for (int c = lane + 32 * HELD; c < V; c += 32)
    dst[c] = from_float<T>(__ldcg(reads + c) * inverse * factor * weight[c] * sigmoid(__ldcg(gate + c)));
}

static bool side_fits(int dim, int vdim) { return (dim == 64 || dim == 128) && vdim % 8 == 0 && vdim <= SIDE_V; }
static bool chunks_fit(int dim, int vdim) { return (dim == 64 || dim == 128) && vdim % 8 == 0; }

template <typename T>
static int launch_memory(const MemoryArgs& p, T* out, int rows, int chunks, int segments, int max_q_len, bool wide, cudaStream_t stream) {
  const int D = p.dim;
  if (max_q_len == 1) {
    const dim3 grid(segments, p.heads);
    const size_t shared = sizeof(float) * (size_t)(p.vdim + 1);
    if (!wide) launch_kernel(matrix_memory_decode_kernel<T, 0>, grid, dim3(DECODE_THREADS), shared, stream, p, out);
    else if (D <= 128) launch_kernel(matrix_memory_decode_kernel<T, 1>, grid, dim3(DECODE_THREADS), shared, stream, p, out);
    else if (D <= 256) launch_kernel(matrix_memory_decode_kernel<T, 2>, grid, dim3(DECODE_THREADS), shared, stream, p, out);
    else launch_kernel(matrix_memory_decode_kernel<T, 4>, grid, dim3(DECODE_THREADS), shared, stream, p, out);
    return launch_status();
  }
  if (p.coef == nullptr || (p.ends == nullptr && (p.reads == nullptr || p.norms == nullptr))) return MLR_BAD_SIZE;
  launch_kernel(matrix_memory_gates_kernel, dim3(segments, p.heads), dim3(GATE_THREADS), 0, stream, p);
  int status = launch_status();
  if (status != MLR_OK) return status;
  if (p.ends != nullptr) {
    if constexpr (sizeof(T) == 2) {
      if (!wide || !side_fits(D, p.vdim) || chunks <= 0 || (long long)chunks + segments > 65535) return MLR_BAD_SIZE;
      if (side_pairs(p.vdim) <= 6)
        return D == 64 ? launch_side<64, 6>(p, out, chunks, segments, stream) : launch_side<128, 6>(p, out, chunks, segments, stream);
      return D == 64 ? launch_side<64, SIDE_PAIRS>(p, out, chunks, segments, stream) : launch_side<128, SIDE_PAIRS>(p, out, chunks, segments, stream);
    }
    return MLR_BAD_DTYPE;
  }
  if (p.pairs != nullptr) {
    if (!wide || !chunks_fit(D, p.vdim)) return MLR_BAD_SIZE;
    status = D == 64 ? launch_chunks<64>(p, segments, max_q_len, stream) : launch_chunks<128>(p, segments, max_q_len, stream);
  } else if (wide) {
    if (D <= 32) status = launch_scan<4, 8, 1, true>(p, segments, stream);
    else if (D <= 64) status = launch_scan<4, 16, 1, true>(p, segments, stream);
    else if (D <= 128) status = launch_scan<8, 16, 2, true>(p, segments, stream);
    else if (D <= 256) status = launch_scan<8, 32, 2, true>(p, segments, stream);
    else status = launch_scan<16, 32, 2, true>(p, segments, stream);
  } else {
    if (D <= 32) status = launch_scan<4, 8, 1, false>(p, segments, stream);
    else if (D <= 128) status = launch_scan<16, 8, 1, false>(p, segments, stream);
    else status = launch_scan<16, 32, 1, false>(p, segments, stream);
  }
  if (status != MLR_OK) return status;
  const long long items = (long long)rows * p.heads;
  auto aligned = [](const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0; };
  const bool pieces = p.vdim % 4 == 0 && p.vdim <= 256 && p.gate_stride % 4 == 0 && aligned(p.gate) && aligned(p.reads) &&
                      aligned(p.weight) && aligned(out);
  launch_kernel(pieces ? matrix_memory_finish_kernel<T, true> : matrix_memory_finish_kernel<T, false>,
                dim3((unsigned)((items + 3) / 4)), dim3(128), 0, stream, p, out, items);
  return launch_status();
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// Whether prompts of these head sizes can go through the tensor cores in chunks (with `pairs`).
MLR_EXPORT int mlr_matrix_memory_chunks_fit(int dim, int vdim) { return chunks_fit(dim, vdim); }

// 1 where a step's chunks go side by side, 0 where a segment's go one behind the other: where no portion has more than two.  One behind the other / side by
// side, repeated calls: 65 rows of 7 heads 21.5 / 24.4 us, 128 rows 22.5 / 24.4, 129 rows 24.9 / 24.8, 192 rows 25.5 / 24.9, 16 heads of 129 rows 25.2 / 25.2; from a
// flushed L2 129 rows 42 / 34, 192 rows 44 / 36, four of 129 rows 48 / 36, of 16 heads 63 / 54.
MLR_EXPORT int mlr_matrix_memory_side_by_side(int chunks, int segments, int max_q_len, int vdim) {
  return side_fits(64, vdim) && max_q_len > 2 * CHUNK && (long long)chunks + segments <= 65535 ? 1 : 0;
}
// .. and the float32 numbers of scratch that side by side needs.
MLR_EXPORT long long mlr_matrix_memory_side_scratch(int chunks, int heads, int dim, int vdim) { return (long long)chunks * heads * ((long long)(vdim + 1) * dim + 1); }

// q, k: float32 rows of heads * dim entries; v, gate: rows of heads * vdim; i_raw, f_raw: rows of `heads` entries (each
// with its own row stride); i_bias, f_bias: float32 [heads]; weight: float32 [heads * vdim]; coef: float32 scratch
// [rows, heads, 4], reads: [rows, heads, vdim], norms: [rows, heads] (all three null for steps of single rows); pairs:
// float32 scratch [rows, heads, 64 + 2] and packed: bfloat16 scratch [rows, heads, 2 dim + vdim] (both or neither: chunks
// on the tensor cores, or the token-by-token scan; 16-byte aligned); ends: null, or the scratch of chunks side by side (as the two
// functions above say, for bfloat16 results; reads, norms, pairs and packed are then not asked for) with chunks: those of all segments of `least` rows (1, or 2
// where there may be single rows) and more, or the most there can be; states:
// float32 [slots, heads, vdim + 1, dim], maxima: float32 [slots, heads]; out: [rows, heads * vdim] in `dtype`.
// max_q_len: the longest segment of the step.
MLR_EXPORT int mlr_matrix_memory(const float* q, long long q_stride, const float* k, long long k_stride, const float* v,
                                 long long v_stride, const float* i_raw, long long i_stride, const float* f_raw,
                                 long long f_stride, const float* gate, long long gate_stride, const float* i_bias,
                                 const float* f_bias, const float* weight, float* coef, float* reads, float* norms,
                                 float* pairs, void* packed, float* ends, int chunks, int least, float* states, float* maxima, void* out, const int* seg_q_start, const int* seg_q_len,
                                 const int* seg_slot, int rows, int segments, int max_q_len, int heads, int dim, int vdim,
                                 float cap, float guard, float eps, float q_scale, int dtype, cudaStream_t stream) {
  if (segments == 0 || rows == 0) return MLR_OK;
  if (segments < 0 || rows < 0 || max_q_len <= 0 || heads <= 0 || dim <= 0 || vdim <= 0 || !(cap > 0.f)) return MLR_BAD_SIZE;
  if (dim > 512 || vdim > 4096 || heads > 65535 || segments > 65535) return MLR_TOO_LARGE;
  bf16* q16 = (bf16*)packed;
  bf16* k16 = q16 == nullptr ? nullptr : q16 + (size_t)rows * heads * dim;
  bf16* v16 = q16 == nullptr ? nullptr : k16 + (size_t)rows * heads * dim;
  if ((pairs == nullptr) != (packed == nullptr) || least < 1 || least > 2 || (least > 1 && ends == nullptr)) return MLR_BAD_SIZE;
  MemoryArgs p{q, k, v, i_raw, f_raw, gate, q_stride, k_stride, v_stride, i_stride, f_stride, gate_stride, i_bias, f_bias,
               weight, reinterpret_cast<float4*>(coef), reads, norms, pairs,
               pairs == nullptr ? nullptr : reinterpret_cast<float2*>(pairs + (size_t)rows * heads * CHUNK), q16, k16, v16, states, maxima, ends,
               ends == nullptr ? nullptr : ends + (size_t)chunks * heads * (vdim + 1) * dim, seg_q_start, seg_q_len, seg_slot,
               segments, least, heads, dim, vdim, cap, guard, eps, q_scale};
  auto multiple = [](long long n) { return n % 4 == 0; };
  auto aligned = [](const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0; };
  if (!aligned(coef) || !aligned(pairs) || !aligned(packed) || !aligned(ends)) return MLR_BAD_ALIGNMENT;
  const bool wide = multiple(dim) && multiple(vdim) && multiple(q_stride) && multiple(k_stride) && multiple(v_stride) &&
                    aligned(q) && aligned(k) && aligned(v) && aligned(states);
  if (dtype == MLR_F32) return launch_memory(p, (float*)out, rows, chunks, segments, max_q_len, wide, stream);
  if (dtype == MLR_BF16) return launch_memory(p, (bf16*)out, rows, chunks, segments, max_q_len, wide, stream);
  return MLR_BAD_DTYPE;
}
