// The gated delta rule of delta_rule.cu with long segments in chunks of 64 tokens.  Within a chunk that starts from the state S
// [dim, vdim] (G_t the decays of its tokens up to t, D(t, s) those of s + 1 .. t, keys and queries with their norms folded into factors),
//
//   A_ts = beta_t D(t, s) k_t . k_s  (s < t),   T = (1 + A)^-1,   P_ts = D(t, s) q_t . k_s  (s <= t)
//   R_t = beta_t (v_t - G_t S^T k_t),   u = T R,   o_t = G_t S^T q_t + sum_s P_ts u_s,   S' = G_last S + sum_s D(last, s) k_s u_s^T
//
// delta_solve_kernel   all chunks at once: T, P and the factors of every chunk and head, on the CUDA cores
// delta_chain_kernel   the chunks of a (segment, head) one after the other, 16 value channels per CTA; leaves every chunk's S and u
// delta_read_kernel    all chunks at once: o
//
// Products run on the tensor cores (mma.sync) in 32 bits: operands in three bfloat16 parts, six of the nine products (the rest is below
// 2^-26), the leading product and the small ones in sums of their own, at most 64 k long (the tensor cores' sums drop bits at every
// step: with_dropped), added in float32.  Decays are products throughout: nothing divides, they may be zero.
//
// Roundings that every output sees are saved: norms, decays and P are computed in 64 bits and rounded once, beta v - G .. and u's share of
// the state are each one rounding.  Error against 64 bits (2-norm, outputs / states, means of four inputs), token by token, here without and
// with all that, in 1e-7: 2,048 rows of 32 heads of 128 x 64 1.21 / 1.24, 1.65 / 1.25, 1.09 / 1.11; 14 heads of 64 x 64 1.29 / 1.27, 1.84 / 1.49,
// 1.11 / 1.12.  It costs 12 us of 2,048 rows of the 32 heads, 6 of the 14.
//
// Measured (B200), token by token / in chunks: 2,048 rows of 32 heads of 128 x 64 340 / 191 us, from a flushed L2 347 / 206 (first kernel
// 71, second 83, third 48), of 14 heads of 64 x 64 214 / 105 (23, 62, 16).  The first kernel waits for shared memory (chains of reads of
// triangles and decays) and for its code, the chain is the latency of its steps, 4,800 cycles per chunk, of which the tensor pipe is busy for
// 1,900, the last waits for its loads.
//
// The first two kernels do not bring in the next one early: its waiting CTAs slow them down (512 rows of 14 heads of 64 x 64: the first
// kernel 17 -> 25 us, all three 46 -> 56; of 32 heads of 128 x 64 71 -> 77).
//
// In the chain four warps issue MMAs, each with 16 channels x a quarter of dim of the state in its registers (as accumulators, whose
// layout is that of the next product's left operand), while four fetch the next chunk's keys and T, whose parts the first kernel left.
#include "chunk_places.cuh"
#include "part_products.cuh"
#include "tma.cuh"

namespace mlr {

constexpr int DC_COLS = 16;                     // value channels of a chain's CTA
constexpr int DC_SQUARE = CHUNK * CHUNK;
constexpr int DC_FACTORS = 4 * CHUNK;           // of a chunk and head: beta G rk | beta | D(last, .) rk | G rq;  rk, rq: one over the norms
constexpr int DC_PITCH = CHUNK + 8;             // shared rows of 64 numbers: float pairs and ldmatrix without bank conflicts

struct DeltaChunkArgs {
  const float *q, *k, *v, *a, *b;       // row-major views, one row per token
  long long q_stride, k_stride, v_stride, a_stride, b_stride;
  const float *dt_bias, *A_log;         // [heads]
  float* states;                        // [slots, heads, vdim, dim]
  float* y;                             // [rows, heads * vdim]
  bf16* key_parts;                      // [chunks, kv heads, 3, 64, dim + 8]: the keys, rows spaced as in the chain's shared memory
  bf16* T;                              // [chunks, heads, 3, 64, DC_PITCH], likewise
  float* P;                             // [chunks, heads, 64, 64]
  float* factors;                       // [chunks, heads, DC_FACTORS]
  float* decays;                        // [chunks, heads]: G_last
  float* u;                             // [chunks, heads, vdim, 64]
  float* before;                        // [chunks, heads, vdim, dim]: S
  const int *seg_q_start, *seg_q_len, *seg_slot;
  int segments, least, heads, kv_heads, vdim;
  int first_chunk, chunks;              // of this round; scratch is indexed from the first on
  int beside;                           // the launch just before is the recurrence of the short segments, which runs beside the first kernel
  float unit_eps, q_scale;
  int* error_word;
};

// Chunks of the long segments before segment `seg`.
__device__ __forceinline__ int chunks_before(const int* seg_q_len, int seg, int least) {
  int count = 0;
  for (int i = threadIdx.x & 31; i < seg; i += 32) {
    const int length = seg_q_len[i];
    if (length >= least) count += (length + CHUNK - 1) / CHUNK;
  }
  return __reduce_add_sync(0xffffffffu, count);
}

// ---------------------------------------------------------------- products in parts
// Four neighbouring numbers of a row as parts into three tiles `apart` entries apart.
__device__ __forceinline__ void store_parts(bf16* dst, int apart, float4 v) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const uint32_t low = take_part(v.x, v.y), high = take_part(v.z, v.w);
    *reinterpret_cast<uint2*>(dst + q * apart) = make_uint2(low, high);
  }
}

// Of a left operand whose columns are tokens from t0 on: numbers whose parts are not finite become zeros, else a zero weight would carry them
// to the tokens before; first: the earliest of them, in this lane's two rows.  That is infinities, NaN and what rounds to an infinite part.
__device__ __forceinline__ bool take_out(float (&v)[2][4], int t0, int (&first)[2]) {
  constexpr float LIMIT = 3.39617752923046e38f;      // half a last place above the largest bfloat16 number
  bool any = false;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) any |= !(fabsf(v[j][e]) < LIMIT);
  if (!__any_sync(0xffffffffu, any)) return false;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (!(fabsf(v[j][e]) < LIMIT)) {
        first[e >> 1] = min(first[e >> 1], t0 + j * 8 + (e & 1));
        v[j][e] = 0.f;
      }
  return true;
}
__device__ __forceinline__ void earliest_of_row(int (&first)[2]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    first[i] = min(first[i], __shfl_xor_sync(0xffffffffu, first[i], 1));
    first[i] = min(first[i], __shfl_xor_sync(0xffffffffu, first[i], 2));
  }
}

// ---------------------------------------------------------------- T, P and factors
template <int D>
struct SolveShape {
  static constexpr int KEY_PITCH = D + 8, KEY_APART = CHUNK * KEY_PITCH, QUERY_PITCH = D + 8, SQUARE_PITCH = CHUNK + 4;
  static constexpr size_t INPUTS = 3 * KEY_APART * sizeof(bf16) + CHUNK * QUERY_PITCH * sizeof(float);      // until the products are there
  static constexpr size_t SQUARES = 4 * CHUNK * SQUARE_PITCH * sizeof(float);                               // kk, qk, A of two heads
  static constexpr size_t SHARED = INPUTS > SQUARES ? INPUTS : SQUARES;
};

// A CTA per chunk and key/value head: the products k_t . k_s and q_t . k_s of s <= t on the tensor cores, then its heads two at a time.
// T is a triangular inverse: the two triangles of 32 rows at once, a thread per column, then T_21 = -T_22 A_21 T_11.  Bound by
// shared-memory reads; on the CUDA cores the products alone took 24,000 cycles of a CTA, and 64 rows one behind the other 19,000.
// Behind delta_scan_kernel, which triggers its successor only once all that came before it is complete, it starts without a wait: the two
// share nothing.  One thread waits at the end, so that whoever waits for this kernel has waited for that one as well.
// grid: (chunks, kv heads)
template <int D>
__global__ void __launch_bounds__(256, 2)
delta_solve_kernel(DeltaChunkArgs p) {
  using Shape = SolveShape<D>;
  constexpr int SQUARE_PITCH = Shape::SQUARE_PITCH, HALF = CHUNK / 2, ROW_LANES = D / 4;
  extern __shared__ __align__(128) uint8_t solve_shared[];
  bf16* keys = reinterpret_cast<bf16*>(solve_shared);                                        // in parts
  float* queries = reinterpret_cast<float*>(solve_shared + 3 * Shape::KEY_APART * sizeof(bf16));
  float *kk = reinterpret_cast<float*>(solve_shared), *qk = kk + CHUNK * SQUARE_PITCH, *matrix = qk + CHUNK * SQUARE_PITCH;
  __shared__ double rq[CHUNK];
  __shared__ float rk[CHUNK], decay[2][CHUNK], beta[2][CHUNK], upto[2][CHUNK];
  if (!p.beside) pdl_wait();
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, p.first_chunk + blockIdx.x);
  const bool waits = p.beside && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0;
  if (seg < 0) {
    if (waits) pdl_wait();
    return;
  }
  const int kv = blockIdx.y, first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;

  {      // rows of keys (parts to shared memory and to the chain) and queries with one over their norms; D / 4 lanes have a row
    constexpr int PIECES = CHUNK * ROW_LANES / 256;
    bf16* parts = p.key_parts + ((size_t)blockIdx.x * p.kv_heads + kv) * 3 * Shape::KEY_APART;
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      float4 piece[PIECES];
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        const int idx = t + i * 256, row = idx / ROW_LANES, d = idx % ROW_LANES * 4;
        const float* from = (which ? p.q + (size_t)(first + row) * p.q_stride : p.k + (size_t)(first + row) * p.k_stride) + (size_t)kv * D + d;
        piece[i] = row < count ? __ldcg(reinterpret_cast<const float4*>(from)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        const int idx = t + i * 256, row = idx / ROW_LANES, d = idx % ROW_LANES * 4;
        const float4 x = piece[i];
        double sum = fmaf(x.x, x.x, x.y * x.y) + fmaf(x.z, x.z, x.w * x.w);
#pragma unroll
        for (int offset = ROW_LANES / 2; offset > 0; offset >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, offset);
        const double inverse = row < count ? rsqrt(sum + p.unit_eps) : 0.;      // rows behind the segment are nothing, whatever unit_eps
        if (d == 0) {
          if (which) rq[row] = p.q_scale * inverse; else rk[row] = (float)inverse;
        }
        if (which) {
          *reinterpret_cast<float4*>(queries + row * Shape::QUERY_PITCH + d) = x;
        } else {
          float4 rest = x;
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const uint32_t low = take_part(rest.x, rest.y), high = take_part(rest.z, rest.w);
            const int to = q * Shape::KEY_APART + row * Shape::KEY_PITCH + d;
            *reinterpret_cast<uint2*>(keys + to) = make_uint2(low, high);
            *reinterpret_cast<uint2*>(parts + to) = make_uint2(low, high);
          }
        }
      }
    }
  }
  __syncthreads();
  {      // warps 0 .. 3 keys with keys, 4 .. 7 queries with keys, 16 rows each, columns up to the diagonal (one to four pairs of tiles)
    const bool of_queries = warp >= 4;
    const int tile = of_queries ? 7 - warp : warp, r = lane >> 2, c2 = (lane & 3) * 2;
    float total[8][4], lead[8][4], low[8][4];
    clear(total);
    clear(lead);
    clear(low);
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      uint32_t x[3][4];
      if (of_queries) {
        float v[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float* from = queries + (tile * 16 + r) * Shape::QUERY_PITCH + ks * 16 + j * 8 + c2;
          const float2 top = *reinterpret_cast<const float2*>(from), bottom = *reinterpret_cast<const float2*>(from + 8 * Shape::QUERY_PITCH);
          v[j][0] = top.x; v[j][1] = top.y; v[j][2] = bottom.x; v[j][3] = bottom.y;
        }
        split_operand(x, v[0], v[1]);
      } else {
#pragma unroll
        for (int q = 0; q < 3; ++q)
          ldmatrix_x4(x[q], keys + q * Shape::KEY_APART + (tile * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * Shape::KEY_PITCH + ks * 16 + (lane >> 4) * 8);
      }
      add_products<false, 4>(lead, low, x, keys + ((lane & 7) + ((lane >> 4) << 3)) * Shape::KEY_PITCH + ks * 16 + ((lane >> 3) & 1) * 8,
                             16 * Shape::KEY_PITCH, Shape::KEY_APART, 0, tile + 1);
      if (ks % 4 == 3) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            total[j][e] += lead[j][e];
            low[j][e] = with_dropped(lead[j][e], low[j][e], 1.f);
          }
        clear(lead);
      }
    }
    __syncthreads();      // keys and queries have been read
    float* out = (of_queries ? qk : kk) + (tile * 16 + r) * SQUARE_PITCH + c2;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      *reinterpret_cast<float2*>(out + j * 8) = make_float2(total[j][0] + low[j][0], total[j][1] + low[j][1]);
      *reinterpret_cast<float2*>(out + 8 * SQUARE_PITCH + j * 8) = make_float2(total[j][2] + low[j][2], total[j][3] + low[j][3]);
    }
  }
  const int per = p.heads / p.kv_heads, half = (t >> 6) & 1, s = t & 63, row_half = t >> 7;
  for (int h0 = 0; h0 < per; h0 += 2) {
    const bool mine = h0 + half < per;
    const int head = kv * per + (mine ? h0 + half : h0);
    const size_t at = (size_t)blockIdx.x * p.heads + head;
    float g = 1.f, step = 0.f;
    if (s < count) {
      const float z = __ldcg(p.a + (size_t)(first + s) * p.a_stride + head) + p.dt_bias[head];
      g = expf(-expf(p.A_log[head]) * (z > 20.f ? z : log1pf(expf(z))));
      step = 1.f / (1.f + expf(-__ldcg(p.b + (size_t)(first + s) * p.b_stride + head)));
    }
    if (row_half == 0) {
      decay[half][s] = g;
      beta[half][s] = step;
    }
    __syncthreads();      // also: kk and qk are there, the heads before are done
    float* A = matrix + half * CHUNK * SQUARE_PITCH;
    const float own = rk[s];
    double since = 1.;      // D(row, s)
    float* P = p.P + at * DC_SQUARE;
    {      // two threads per column, one for the earlier rows and one for the later
      const int row0 = row_half * HALF;
      if (row_half == 1) {      // four chains of products instead of one: 2,048 rows of 32 heads 218 -> 212 us
        double chain[4] = {1., 1., 1., 1.};
#pragma unroll
        for (int row = 0; row < HALF; ++row)
          if (row > s) chain[row & 3] *= decay[half][row];
        since = (chain[0] * chain[1]) * (chain[2] * chain[3]);
      }
#pragma unroll 8
      for (int row = row0; row < row0 + HALF; ++row) {
        if (row > s) since *= decay[half][row];
        const double weight = since * own;
        if (mine) P[row * CHUNK + s] = row >= s ? (float)(weight * rq[row] * qk[row * SQUARE_PITCH + s]) : 0.f;
        A[row * SQUARE_PITCH + s] = row > s ? (float)weight * rk[row] * beta[half][row] * kk[row * SQUARE_PITCH + s] : 0.f;
        if (s == 0) upto[half][row] = (float)(decay[half][0] * since);
      }
    }
    __syncthreads();
    if (mine && row_half == 1) {      // since is D(last, s) here
      float* factors = p.factors + at * DC_FACTORS;
      factors[s] = step * upto[half][s] * own;
      factors[CHUNK + s] = step;
      factors[2 * CHUNK + s] = (float)(since * own);
      factors[3 * CHUNK + s] = (float)(upto[half][s] * rq[s]);
      if (s == 0) p.decays[at] = upto[half][CHUNK - 1];
    }
    float x[HALF];      // column s of its triangle's inverse
    if (row_half == 0) {
      const float* triangle = A + (s / HALF) * HALF * (SQUARE_PITCH + 1);
      const int column = s & (HALF - 1);
#pragma unroll
      for (int b = 0; b < HALF; b += 16) {
        float sum[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i] = b + i == column ? 1.f : 0.f;
#pragma unroll
        for (int k = 0; k < b; k += 4)
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float4 r = *reinterpret_cast<const float4*>(triangle + (b + i) * SQUARE_PITCH + k);
            sum[i] = fmaf(-r.w, x[k + 3], fmaf(-r.z, x[k + 2], fmaf(-r.y, x[k + 1], fmaf(-r.x, x[k], sum[i]))));
          }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          x[b + i] = sum[i];
#pragma unroll
          for (int j = i + 1; j < 16; ++j) sum[j] = fmaf(-triangle[(b + j) * SQUARE_PITCH + b + i], x[b + i], sum[j]);
        }
      }
    }
    __syncthreads();
    if (row_half == 0) {
#pragma unroll
      for (int i = 0; i < HALF; ++i) A[(s / HALF * HALF + i) * SQUARE_PITCH + s] = x[i];
    }
    __syncthreads();
    // A_21 T_11, then -T_22 times that, both where A_21 was: 128 threads per head, two rows x four columns each
    {
      const int i = row_half * 64 + s, row = HALF + (i >> 3) * 2, col = (i & 7) * 4;
#pragma unroll
      for (int turn = 0; turn < 2; ++turn) {
        const float *left = A + row * SQUARE_PITCH + turn * HALF, *right = A + turn * HALF * SQUARE_PITCH + col;
        float sum[2][4] = {};
#pragma unroll
        for (int k = 0; k < HALF; k += 4) {
          const float4 u0 = *reinterpret_cast<const float4*>(left + k), u1 = *reinterpret_cast<const float4*>(left + SQUARE_PITCH + k);
          const float l0[4] = {u0.x, u0.y, u0.z, u0.w}, l1[4] = {u1.x, u1.y, u1.z, u1.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // T_22 ends at its diagonal: what lies behind must not even be multiplied by its zeros
            const int behind = turn == 0 ? -1 : k + e - (row - HALF);
            if (behind > 1) break;
            const float4 w = *reinterpret_cast<const float4*>(right + (k + e) * SQUARE_PITCH);
            if (behind < 1) {
              sum[0][0] = fmaf(l0[e], w.x, sum[0][0]); sum[0][1] = fmaf(l0[e], w.y, sum[0][1]);
              sum[0][2] = fmaf(l0[e], w.z, sum[0][2]); sum[0][3] = fmaf(l0[e], w.w, sum[0][3]);
            }
            sum[1][0] = fmaf(l1[e], w.x, sum[1][0]); sum[1][1] = fmaf(l1[e], w.y, sum[1][1]);
            sum[1][2] = fmaf(l1[e], w.z, sum[1][2]); sum[1][3] = fmaf(l1[e], w.w, sum[1][3]);
          }
        }
        __syncthreads();
        const float sign = turn == 0 ? 1.f : -1.f;
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<float4*>(A + (row + e) * SQUARE_PITCH + col) = make_float4(sign * sum[e][0], sign * sum[e][1], sign * sum[e][2], sign * sum[e][3]);
        __syncthreads();
      }
      bf16* T = p.T + at * 3 * CHUNK * DC_PITCH;
      if (mine) {
#pragma unroll
        for (int n = 0; n < DC_SQUARE / 4 / 128; ++n) {
          const int idx = i + n * 128, r = idx / (CHUNK / 4), c = idx % (CHUNK / 4) * 4;
          store_parts(T + r * DC_PITCH + c, CHUNK * DC_PITCH, *reinterpret_cast<const float4*>(A + r * SQUARE_PITCH + c));
        }
      }
    }
    __syncthreads();      // A, decays and factors are rewritten by the next heads
  }
  if (waits) pdl_wait();
}

// ---------------------------------------------------------------- the chain
template <int D>
struct ChainShape {
  static constexpr int KEY_PITCH = D + 8, KEY_APART = CHUNK * KEY_PITCH, T_APART = CHUNK * DC_PITCH, LEFT_APART = DC_COLS * DC_PITCH;
  static constexpr size_t KEYS = 3 * KEY_APART * sizeof(bf16), SQUARE = 3 * T_APART * sizeof(bf16);
  static constexpr size_t VALUES = DC_COLS * DC_PITCH * sizeof(float), ROW = CHUNK * sizeof(float);
  static constexpr size_t BUFFER = KEYS + SQUARE + VALUES + 3 * ROW;
  static constexpr size_t LEFT = 3 * LEFT_APART * sizeof(bf16);
  static constexpr size_t SHARED = 2 * BUFFER + 4 * VALUES + 2 * LEFT + 4 * DC_COLS * sizeof(int);      // the four warps' sums, R and u in parts
  static_assert(KEYS % 16 == 0 && SQUARE % 16 == 0 && BUFFER % 16 == 0, "bulk copies");
};

// A left operand of 16 rows x 16 k whose parts lie in shared memory, DC_PITCH entries per row.
__device__ __forceinline__ void load_operand(uint32_t (&x)[3][4], const bf16* tile, int k, int lane) {
#pragma unroll
  for (int q = 0; q < 3; ++q)
    ldmatrix_x4(x[q], tile + q * DC_COLS * DC_PITCH + ((lane & 7) + ((lane >> 3) & 1) * 8) * DC_PITCH + k + (lane >> 4) * 8);
}
// .. and its way there, from two neighbouring accumulators
__device__ __forceinline__ void store_operand(bf16* tile, int k, const float (&left)[4], const float (&right)[4], int r, int c2) {
  uint32_t x[3][4];
  split_operand(x, left, right);
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<uint32_t*>(tile + q * DC_COLS * DC_PITCH + (r + 8 * (i & 1)) * DC_PITCH + k + (i >> 1) * 8 + c2) = x[q][i];
}

// grid: (long segments, heads, vdim / 16)
template <int D>
__global__ void __launch_bounds__(256, 1)
delta_chain_kernel(DeltaChunkArgs p) {
  using Shape = ChainShape<D>;
  constexpr int SLICE = D / 4, STEPS = SLICE / 16, TILES = SLICE / 8;      // a warp's share of dim
  extern __shared__ __align__(128) uint8_t chain_shared[];
  float* sums = reinterpret_cast<float*>(chain_shared + 2 * Shape::BUFFER);                          // [4][16][DC_PITCH]
  bf16* right_side = reinterpret_cast<bf16*>(sums + 4 * DC_COLS * DC_PITCH);                          // R in parts
  bf16* u_parts = right_side + 3 * Shape::LEFT_APART;                                                 // u times its factors
  int* broken_of = reinterpret_cast<int*>(u_parts + 3 * Shape::LEFT_APART);                           // [4][16]
  __shared__ uint64_t there[2];                                                                       // keys and T of a buffer
  if (threadIdx.x == 0) {
    mbar_init(&there[0], 1);
    mbar_init(&there[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();
  const ChunkAt segment = chunk_at<false>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.x);
  if (segment.seg < 0) return;
  const int seg = segment.seg, length = segment.length, start = segment.start, slot = segment.slot;
  const int head = blockIdx.y, kv = head / (p.heads / p.kv_heads), col0 = blockIdx.z * DC_COLS, V = p.vdim;
  // of the segment's chunks those of this round; `place` of the first chunk is where its numbers would lie in scratch
  const int place = chunks_before(p.seg_q_len, seg, p.least) - p.first_chunk;
  const int begin = max(0, -place), end = min((length + CHUNK - 1) / CHUNK, p.chunks - place);
  if (begin >= end) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane >> 2, c2 = (lane & 3) * 2;      // of an accumulator: rows r and r + 8, columns c2 and c2 + 1

  auto keys_of = [&](int which) { return reinterpret_cast<bf16*>(chain_shared + which * Shape::BUFFER); };
  auto square_of = [&](int which) { return reinterpret_cast<bf16*>(chain_shared + which * Shape::BUFFER + Shape::KEYS); };
  auto values_of = [&](int which) { return reinterpret_cast<float*>(chain_shared + which * Shape::BUFFER + Shape::KEYS + Shape::SQUARE); };

  // The last four warps fetch: parts of keys and T by a bulk copy each, values and factors through registers, asked for a chunk before.
  constexpr int V_PIECES = CHUNK * DC_COLS / 4 / 128;
  float4 v_piece[V_PIECES];
  float factor, beta;
  const int i0 = threadIdx.x - 128;
  auto copy = [&](int chunk, int which) {
    const size_t at = (size_t)(place + chunk);
    mbar_expect_tx(&there[which], (uint32_t)(Shape::KEYS + Shape::SQUARE));
    auto bulk = [&](bf16* dst, const bf16* src, size_t bytes) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(shared_address(dst)), "l"(src), "r"((uint32_t)bytes), "r"(smem_u32(&there[which])) : "memory");
    };
    bulk(keys_of(which), p.key_parts + (at * p.kv_heads + kv) * 3 * Shape::KEY_APART, Shape::KEYS);
    bulk(square_of(which), p.T + (at * p.heads + head) * 3 * Shape::T_APART, Shape::SQUARE);
  };
  auto ask = [&](int chunk) {
    const int row0 = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK);
    const float* factors = p.factors + ((size_t)(place + chunk) * p.heads + head) * DC_FACTORS;
#pragma unroll
    for (int n = 0; n < V_PIECES; ++n) {
      const int idx = i0 + n * 128, row = idx / (DC_COLS / 4), c = idx % (DC_COLS / 4) * 4;
      v_piece[n] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < count) v_piece[n] = __ldcg(reinterpret_cast<const float4*>(p.v + (size_t)(row0 + row) * p.v_stride + (size_t)head * V + col0 + c));
    }
    factor = __ldcg(factors + (i0 < CHUNK ? i0 : i0 + CHUNK));      // beta G rk | D(last, .) rk | beta
    beta = __ldcg(factors + CHUNK + i0 % CHUNK);
  };
  auto put = [&](int which) {
    float *values = values_of(which), *row_factor = values + DC_COLS * DC_PITCH;
#pragma unroll
    for (int n = 0; n < V_PIECES; ++n) {
      const int idx = i0 + n * 128, row = idx / (DC_COLS / 4), c = idx % (DC_COLS / 4) * 4;
      const float4 x = v_piece[n];
      values[c * DC_PITCH + row] = x.x;
      values[(c + 1) * DC_PITCH + row] = x.y;
      values[(c + 2) * DC_PITCH + row] = x.z;
      values[(c + 3) * DC_PITCH + row] = x.w;
    }
    row_factor[i0] = factor;
    if (i0 < CHUNK) row_factor[2 * CHUNK + i0] = beta;
  };
  // The fetching warps wait for the copies; the block's barrier behind it tells the others, who would pay for a look of their own.
  bool gave_up = false;
  auto arrived = [&](int chunk) {
    if (!gave_up) gave_up = !mbar_wait(&there[(chunk - begin) & 1], ((chunk - begin) >> 1) & 1, p.error_word, 51);
  };
  float* state = p.states + ((size_t)slot * p.heads + head) * V * D + (size_t)col0 * D;
  float S[TILES][4];
  __syncthreads();      // the barriers are set up
  if (warp >= 4) {
    if (i0 == 0) copy(begin, 0);
    ask(begin);
    put(0);
    if (begin + 1 < end) ask(begin + 1);
    arrived(begin);
  } else {
#pragma unroll
    for (int j = 0; j < TILES; ++j) {
      const float2 top = __ldcg(reinterpret_cast<const float2*>(state + r * D + warp * SLICE + j * 8 + c2));
      const float2 bottom = __ldcg(reinterpret_cast<const float2*>(state + (r + 8) * D + warp * SLICE + j * 8 + c2));
      S[j][0] = top.x; S[j][1] = top.y; S[j][2] = bottom.x; S[j][3] = bottom.y;
    }
  }
  __syncthreads();

  for (int chunk = begin; chunk < end; ++chunk) {
    const int which = (chunk - begin) & 1;
    if (warp >= 4) {
      if (chunk + 1 < end) {
        if (i0 == 0) copy(chunk + 1, which ^ 1);
        put(which ^ 1);
      }
      if (chunk + 2 < end) ask(chunk + 2);
      if (chunk + 1 < end) arrived(chunk + 1);
    } else {

      const bf16 *keys = keys_of(which), *square = square_of(which);
      const float *values = values_of(which), *row_factor = values + DC_COLS * DC_PITCH;
      const size_t at = (size_t)(place + chunk) * p.heads + head;
      const float last = __ldcg(p.decays + at);
      {      // this warp's share of S^T k_t
        float lead[8][4], low[8][4];
        clear(lead);
        clear(low);
#pragma unroll
        for (int ks = 0; ks < STEPS; ++ks) {
          uint32_t x[3][4];
          split_operand(x, S[2 * ks], S[2 * ks + 1]);
          add_products<false, 4>(lead, low, x, keys + ((lane & 7) + ((lane >> 4) << 3)) * Shape::KEY_PITCH + warp * SLICE + ks * 16 + ((lane >> 3) & 1) * 8,
                                 16 * Shape::KEY_PITCH, Shape::KEY_APART);
        }
        float* mine = sums + warp * DC_COLS * DC_PITCH;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float z[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) z[e] = lead[j][e] + with_dropped(lead[j][e], low[j][e], 0.75f);
          *reinterpret_cast<float2*>(mine + r * DC_PITCH + j * 8 + c2) = make_float2(z[0], z[1]);
          *reinterpret_cast<float2*>(mine + (r + 8) * DC_PITCH + j * 8 + c2) = make_float2(z[2], z[3]);
        }
      }
      // the state before the chunk, for the outputs
      float* before = p.before + (at * V + col0) * D + warp * SLICE;
#pragma unroll
      for (int j = 0; j < TILES; ++j) {
        *reinterpret_cast<float2*>(before + r * D + j * 8 + c2) = make_float2(S[j][0], S[j][1]);
        *reinterpret_cast<float2*>(before + (r + 8) * D + j * 8 + c2) = make_float2(S[j][2], S[j][3]);
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      {      // R of this warp's 16 tokens
        float R[2][4];
        int broken[2] = {CHUNK, CHUNK};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int t = warp * 16 + j * 8 + c2;
          const float2 f = *reinterpret_cast<const float2*>(row_factor + t), beta = *reinterpret_cast<const float2*>(row_factor + 2 * CHUNK + t);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int cell = (r + 8 * i) * DC_PITCH + t;
            float2 z = *reinterpret_cast<const float2*>(sums + cell);
#pragma unroll
            for (int w = 1; w < 4; ++w) {
              const float2 add = *reinterpret_cast<const float2*>(sums + w * DC_COLS * DC_PITCH + cell);
              z.x += add.x;
              z.y += add.y;
            }
            const float2 v = *reinterpret_cast<const float2*>(values + cell);
            R[j][2 * i] = fmaf(beta.x, v.x, -f.x * z.x);
            R[j][2 * i + 1] = fmaf(beta.y, v.y, -f.y * z.y);
          }
        }
        if (take_out(R, warp * 16 + c2, broken)) earliest_of_row(broken);
        broken_of[warp * DC_COLS + r] = broken[0];
        broken_of[warp * DC_COLS + r + 8] = broken[1];
        store_operand(right_side, warp * 16, R[0], R[1], r, c2);
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      {      // u of this warp's 16 tokens: T R, where T ends at the diagonal
        float part[6][2][4];
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) part[q][j][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          if (ks > warp) break;
          uint32_t x[3][4];
          load_operand(x, right_side, ks * 16, lane);
          const bf16* from = square + (warp * 16 + (lane & 7) + ((lane >> 4) << 3)) * DC_PITCH + ks * 16 + ((lane >> 3) & 1) * 8;
          int number = 0;
#pragma unroll
          for (int q = 2; q >= 0; --q) {      // as add_products, every product in a sum of its own: two accumulators would be a chain
            uint32_t w[4];
            ldmatrix_x4(w, from + q * Shape::T_APART);
#pragma unroll
            for (int i = 2 - q; i >= 0; --i, ++number) {
              mma_bf16(part[number][0], x[i], w[0], w[1]);
              mma_bf16(part[number][1], x[i], w[2], w[3]);
            }
          }
        }
        int broken[2] = {CHUNK, CHUNK};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          broken[0] = min(broken[0], broken_of[w * DC_COLS + r]);
          broken[1] = min(broken[1], broken_of[w * DC_COLS + r + 8]);
        }
        float* u = p.u + (at * V + col0) * CHUNK;
        float scaled[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int t = warp * 16 + j * 8 + c2;
          const float2 f = *reinterpret_cast<const float2*>(row_factor + CHUNK + t);
          float total[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float low = part[0][j][e], lead = part[5][j][e];
#pragma unroll
            for (int q = 1; q < 5; ++q) low += part[q][j][e];
            low = with_dropped(lead, low, 0.75f);
            if (t + (e & 1) >= broken[e >> 1]) lead = NAN;
            const float factor = e & 1 ? f.y : f.x;
            total[e] = lead + low;
            scaled[j][e] = fmaf(lead, factor, low * factor);
          }
          *reinterpret_cast<float2*>(u + r * CHUNK + t) = make_float2(total[0], total[1]);
          *reinterpret_cast<float2*>(u + (r + 8) * CHUNK + t) = make_float2(total[2], total[3]);
        }
        store_operand(u_parts, warp * 16, scaled[0], scaled[1], r, c2);
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      {      // this warp's share of the state
        float lead[TILES][4], low[TILES][4];
        clear(lead);
        clear(low);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t x[3][4];
          load_operand(x, u_parts, ks * 16, lane);
          add_products<true, TILES / 2>(lead, low, x, keys + (ks * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * Shape::KEY_PITCH + warp * SLICE + (lane >> 4) * 8,
                                        16, Shape::KEY_APART);
        }
#pragma unroll
        for (int j = 0; j < TILES; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[j][e] = fmaf(last, S[j][e], lead[j][e] + with_dropped(lead[j][e], low[j][e], 0.75f));
      }
    }
    __syncthreads();      // the next chunk's tiles are there, this one's are read
  }
  if (warp < 4) {
#pragma unroll
    for (int j = 0; j < TILES; ++j) {
      *reinterpret_cast<float2*>(state + r * D + warp * SLICE + j * 8 + c2) = make_float2(S[j][0], S[j][1]);
      *reinterpret_cast<float2*>(state + (r + 8) * D + warp * SLICE + j * 8 + c2) = make_float2(S[j][2], S[j][3]);
    }
  }
}

// ---------------------------------------------------------------- the outputs
template <int D>
struct ReadShape {
  static constexpr int Q_PITCH = D + 8, Q_APART = CHUNK * Q_PITCH, P_APART = CHUNK * DC_PITCH;
  static constexpr size_t SHARED = 3 * (Q_APART + P_APART) * sizeof(bf16);
};

// A CTA per chunk, head and 64 value channels, a warp per 16 of them.  grid: (heads, chunks, vdim / 64 rounded up)
template <int D>
__global__ void __launch_bounds__(128, 2)
delta_read_kernel(DeltaChunkArgs p) {
  using Shape = ReadShape<D>;
  extern __shared__ __align__(128) uint8_t read_shared[];
  bf16 *queries = reinterpret_cast<bf16*>(read_shared), *pairs = queries + 3 * Shape::Q_APART;
  pdl_trigger();
  pdl_wait();
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, p.first_chunk + blockIdx.y);
  if (seg < 0) return;
  const int head = blockIdx.x, kv = head / (p.heads / p.kv_heads), V = p.vdim;
  const int first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c2 = (lane & 3) * 2;
  const size_t at = (size_t)blockIdx.y * p.heads + head;
  const int col0 = blockIdx.z * 64 + warp * 16;
  constexpr int BATCH = 8;
#pragma unroll
  for (int n0 = 0; n0 < CHUNK * D / 4 / 128; n0 += BATCH) {
    float4 piece[BATCH];
#pragma unroll
    for (int n = 0; n < BATCH; ++n) {
      const int idx = threadIdx.x + (n0 + n) * 128, row = idx / (D / 4), d = idx % (D / 4) * 4;
      piece[n] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < count) piece[n] = __ldcg(reinterpret_cast<const float4*>(p.q + (size_t)(first + row) * p.q_stride + (size_t)kv * D + d));
    }
#pragma unroll
    for (int n = 0; n < BATCH; ++n) {
      const int idx = threadIdx.x + (n0 + n) * 128, row = idx / (D / 4), d = idx % (D / 4) * 4;
      store_parts(queries + row * Shape::Q_PITCH + d, Shape::Q_APART, piece[n]);
    }
  }
  {
    float4 piece[DC_SQUARE / 4 / 128];
#pragma unroll
    for (int n = 0; n < DC_SQUARE / 4 / 128; ++n) piece[n] = __ldcg(reinterpret_cast<const float4*>(p.P + at * DC_SQUARE) + threadIdx.x + n * 128);
#pragma unroll
    for (int n = 0; n < DC_SQUARE / 4 / 128; ++n) {
      const int idx = threadIdx.x + n * 128;
      store_parts(pairs + idx / 16 * DC_PITCH + idx % 16 * 4, Shape::P_APART, piece[n]);
    }
  }
  __syncthreads();
  if (col0 >= V) return;
  float total[8][4], lead[8][4], low[8][4];
  auto flush = [&]() {
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        total[j][e] += lead[j][e];
        low[j][e] = with_dropped(lead[j][e], low[j][e], 1.f);
      }
    clear(lead);
  };
  clear(total);
  clear(lead);
  clear(low);
  int broken[2] = {CHUNK, CHUNK};
  // left operands: 16 channels x 16 k, first of S, then of u
  constexpr int STEPS = D / 16, ALL = STEPS + CHUNK / 16, AHEAD = 3;
  const float *before = p.before + (at * V + col0) * D, *u = p.u + (at * V + col0) * CHUNK;
  float asked[AHEAD][2][4];
  auto ask = [&](int step, float (&v)[2][4]) {
    const float* from = step < STEPS ? before + (size_t)r * D + step * 16 : u + (size_t)r * CHUNK + (step - STEPS) * 16;
    const int down = 8 * (step < STEPS ? D : CHUNK);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 top = __ldcg(reinterpret_cast<const float2*>(from + j * 8 + c2)), bottom = __ldcg(reinterpret_cast<const float2*>(from + down + j * 8 + c2));
      v[j][0] = top.x; v[j][1] = top.y; v[j][2] = bottom.x; v[j][3] = bottom.y;
    }
  };
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) ask(i, asked[i]);
#pragma unroll
  for (int step = 0; step < STEPS; ++step) {
    uint32_t x[3][4];
    split_operand(x, asked[step % AHEAD][0], asked[step % AHEAD][1]);
    ask(step + AHEAD, asked[step % AHEAD]);
    add_products<false, 4>(lead, low, x, queries + ((lane & 7) + ((lane >> 4) << 3)) * Shape::Q_PITCH + step * 16 + ((lane >> 3) & 1) * 8,
                           16 * Shape::Q_PITCH, Shape::Q_APART);
    if (step % 4 == 3) flush();
  }
  const float* factors = p.factors + at * DC_FACTORS + 3 * CHUNK;      // G rq
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 f = __ldcg(reinterpret_cast<const float2*>(factors + j * 8 + c2));
#pragma unroll
    for (int e = 0; e < 4; ++e) total[j][e] = (total[j][e] + low[j][e]) * (e & 1 ? f.y : f.x);
  }
  clear(low);
#pragma unroll
  for (int step = STEPS; step < ALL; ++step) {
    const int ks = step - STEPS;
    uint32_t x[3][4];
    take_out(asked[step % AHEAD], ks * 16 + c2, broken);
    split_operand(x, asked[step % AHEAD][0], asked[step % AHEAD][1]);
    if (step + AHEAD < ALL) ask(step + AHEAD, asked[step % AHEAD]);
    // tokens before these 16 see none of them
    add_products<false, 4>(lead, low, x, pairs + ((lane & 7) + ((lane >> 4) << 3)) * DC_PITCH + ks * 16 + ((lane >> 3) & 1) * 8, 16 * DC_PITCH,
                           Shape::P_APART, ks);
  }
  earliest_of_row(broken);
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int t = j * 8 + c2 + (e & 1);
      if (t < count)
        p.y[((size_t)(first + t) * p.heads + head) * V + col0 + r + (e >> 1) * 8] = t < broken[e >> 1] ? total[j][e] + (lead[j][e] + with_dropped(lead[j][e], low[j][e], 1.f)) : NAN;
    }
}

// Scratch of a chunk, in float32 numbers (two bfloat16 numbers count for one).
inline long long scratch_of_chunk(int heads, int kv_heads, int dim, int vdim) {
  return (long long)heads * (DC_SQUARE + 3ll * CHUNK * DC_PITCH / 2 + DC_FACTORS + 4 + (long long)vdim * (CHUNK + dim)) + (long long)kv_heads * (3ll * CHUNK * (dim + 8) / 2);
}

// Chunks that a round of launches takes: as many as have their scratch in DC_SCRATCH_BYTES, the rounds as even as can be.  The state goes from one
// to the next where it lies.  8,192 rows of 32 heads of 128 x 64 in rounds of 64, 160 MB and without a bound (470 MB): 826, 811, 732 us, 4,096 rows
// 417, 416, 388; this bound takes 4,400 of these rows at a time, 13,300 of 14 heads of 64 x 64.
constexpr long long DC_SCRATCH_BYTES = 256ll << 20;
inline int chunks_of_round(int chunks, int heads, int kv_heads, int dim, int vdim) {
  const long long most = DC_SCRATCH_BYTES / 4 / scratch_of_chunk(heads, kv_heads, dim, vdim), room = most < 1 ? 1 : most;
  const long long rounds = (chunks + room - 1) / room;
  return (int)((chunks + rounds - 1) / rounds);
}

template <int D>
int launch_delta_chunks(DeltaChunkArgs p, int rows, int chunks, cudaStream_t stream) {
  constexpr size_t solve_shared = SolveShape<D>::SHARED;
  static_assert(ChainShape<D>::SHARED <= 227 * 1024 && 2 * (ReadShape<D>::SHARED + 1024) <= 227 * 1024, "one and two CTAs per SM");
  cudaError_t err = cudaFuncSetAttribute(delta_solve_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)solve_shared);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(delta_chain_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ChainShape<D>::SHARED);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(delta_read_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ReadShape<D>::SHARED);
  if (err != cudaSuccess) return (int)err;
  const int round = p.chunks;
  for (p.first_chunk = 0; p.first_chunk < chunks; p.first_chunk += round) {
    p.chunks = chunks - p.first_chunk < round ? chunks - p.first_chunk : round;
    launch_kernel(delta_solve_kernel<D>, dim3(p.chunks, p.kv_heads), dim3(256), solve_shared, stream, p);
    int status = launch_status();
    if (status != MLR_OK) return status;
    launch_kernel(delta_chain_kernel<D>, dim3((unsigned)long_segments(rows, p.segments, p.least), p.heads, p.vdim / DC_COLS), dim3(256),
                  ChainShape<D>::SHARED, stream, p);
    if ((status = launch_status()) != MLR_OK) return status;
    launch_kernel(delta_read_kernel<D>, dim3(p.heads, p.chunks, (p.vdim + 63) / 64), dim3(128), ReadShape<D>::SHARED, stream, p);
    if ((status = launch_status()) != MLR_OK) return status;
    p.beside = 0;
  }
  return MLR_OK;
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// float32 scratch of a step whose long segments have `chunks` chunks, in numbers.
MLR_EXPORT long long mlr_delta_chunk_scratch(int chunks, int heads, int kv_heads, int dim, int vdim) {
  if (chunks <= 0 || heads <= 0 || kv_heads <= 0 || dim <= 0 || vdim <= 0) return 0;
  return chunks_of_round(chunks, heads, kv_heads, dim, vdim) * scratch_of_chunk(heads, kv_heads, dim, vdim);
}

// As mlr_delta_rule_scan, for the segments of least_rows rows and more, which have `chunks` chunks of 64 rows or fewer in all: dim 64 or 128,
// vdim a multiple of 16, every row of q, k and v, states and scratch on 16-byte boundaries.  rows: the step's rows.  beside: the stream's last
// launch was mlr_delta_rule_scan for the segments below least_rows, and scratch is older than it.  error_word: host-visible int that
// receives a code if a wait runs out.
MLR_EXPORT int mlr_delta_rule_chunks(const float* q, long long q_stride, const float* k, long long k_stride, const float* v,
                                     long long v_stride, const float* a, long long a_stride, const float* b, long long b_stride,
                                     const float* dt_bias, const float* A_log, float* scratch, float* states, float* y,
                                     const int* seg_q_start, const int* seg_q_len, const int* seg_slot, int segments, int rows,
                                     int least_rows, int chunks, int beside, int heads, int kv_heads, int dim, int vdim, float unit_eps, float q_scale,
                                     int* error_word, cudaStream_t stream) {
  if (segments == 0 || chunks == 0) return MLR_OK;
  if (segments < 0 || rows <= 0 || chunks < 0 || least_rows <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0 || scratch == nullptr)
    return MLR_BAD_SIZE;
  if ((dim != 64 && dim != 128) || vdim <= 0 || vdim % DC_COLS != 0) return MLR_BAD_SIZE;
  if (heads > 65535 || vdim > 65535) return MLR_TOO_LARGE;
  const uintptr_t pointers = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)states | (uintptr_t)scratch;
  if (pointers % 16 != 0 || (q_stride | k_stride | v_stride) % 4 != 0) return MLR_BAD_ALIGNMENT;
  const int round = chunks_of_round(chunks, heads, kv_heads, dim, vdim);      // a few thousand at most: a grid's y
  DeltaChunkArgs p{q, k, v, a, b, q_stride, k_stride, v_stride, a_stride, b_stride, dt_bias, A_log, states, y, nullptr, nullptr, scratch, nullptr,
                   nullptr, nullptr, nullptr, seg_q_start, seg_q_len, seg_slot, segments, least_rows, heads, kv_heads, vdim, 0, round, beside, unit_eps,
                   q_scale, error_word};
  const long long places = (long long)round * heads;
  p.factors = p.P + places * DC_SQUARE;
  p.u = p.factors + places * DC_FACTORS;
  p.before = p.u + places * vdim * CHUNK;
  p.T = reinterpret_cast<bf16*>(p.before + places * vdim * dim);
  p.key_parts = p.T + places * 3 * CHUNK * DC_PITCH;
  p.decays = reinterpret_cast<float*>(p.key_parts + (long long)round * kv_heads * 3 * CHUNK * (dim + 8));
  return dim == 64 ? launch_delta_chunks<64>(p, rows, chunks, stream) : launch_delta_chunks<128>(p, rows, chunks, stream);
}
