// The state-space recurrence (see state_space.cu) of steps with long segments, in chunks of 64 tokens side by side.
//
// With one decay g per head and token, a chunk's outputs are a masked product of its tokens plus a read of the state before it,
//   y_t = sum_{s <= t} (prod_{s < u <= t} g_u) (C_t . B_s) dt_s x_s + (prod_{u <= t} g_u) S^T C_t + D x_t,
// and its end state is the decays' product times S plus sum_s (prod_{u > s} g_u) B_s (dt_s x_s)^T.  Four kernels:
//   pairs    C_t . B_s of a chunk, once for all heads of a group, and both in bfloat16 parts
//   ends     per head and chunk: what the chunk's own tokens leave behind; blocks of its own take the step's shorter segments token by
//            token (portions of 1,531, 77, 1 and 439 rows, 32 heads, by multiply-adds: 139 us with all in chunks, 153 with a launch for the
//            shorter ones, 127 so)
//   carry    per state entry, the chunks of a segment in order: the state before each
//   outputs  per head and chunk: the masked product and the read of the state
// Decay products are products of numbers up to one, formed step by step in 64 bits and rounded once (which more than gives back what the
// tensor cores' sums drop), never differences of
// logarithms (whose sums grow large while the differences stay small) nor quotients, so decays may be zero.
//
// The products per (head, chunk) run on the tensor cores, mma.sync with operands in three bfloat16 parts (part_products.cuh), sums of at most 64 k
// at a time.  A weight of zero times an infinity would reach tokens that do not see it: from the first row with a number whose parts are not
// finite on, a chunk goes by multiply-adds (ends_plain, outputs_plain), where such weights are left out; the rows before keep their bits.
//
// Bound by latency and instructions, three or four CTAs of four warps per SM (1.5 and 1.1 of 4 instructions per cycle in ends and outputs, tensor pipes 31 and
// 30 %): splitting of states and inputs, decays, copies.  Measured (B200, repeated calls), token by token / by multiply-adds / so: 2,048 rows of 32 heads with states
// of 128 639 / 120 / 100 us, of 14 heads with states of 64 424 / 56 / 45; 512 rows 161 / 56 / 35 and 108 / 40 / 24; 4,000 rows 218 / 180 (32 heads); portions of 1,531, 77, 1
// and 439 rows 124 / 107 and 60 / 47.  Errors against 64 bits (means of seven lengths, outputs / states) 7.8e-8 / 7.9e-8 by multiply-adds, 7.4e-8 / 7.8e-8 so.
//
#include "chunk_places.cuh"
#include "copy_async.cuh"
#include "part_products.cuh"
#include "state_space_scan.cuh"

namespace mlr {

constexpr int VD = 64;              // value channels of a head
constexpr int W_PITCH = CHUNK + 8;  // rows of the chunk's token-by-token weights: float pairs without bank conflicts
constexpr int TILE_PITCH = 64 + 8, TILE_APART = CHUNK * TILE_PITCH;      // a part of 64 rows of 64 numbers: ldmatrix without bank conflicts
constexpr size_t TILE_BYTES = 3 * TILE_APART * sizeof(bf16);
constexpr int SPACE_THREADS = 128;
constexpr int HALF_N = 64;          // state entries taken at a time
constexpr float DROPPED = 0.75f, ENDS_DROPPED = 0.4f;    // see with_dropped
constexpr float PART_LIMIT = 3.39617752923046e38f;              // half a last place above the largest bfloat16 number: what is not below has no finite parts

struct SpaceArgs {
  const float *x, *B, *C, *dt_raw;
  long long x_stride, b_stride, c_stride, dt_stride;
  const float *dt_bias, *A_log, *D;
  float* states;                     // [slots, heads, VD, n]
  float* y;                          // [rows, heads * VD]
  float* pairs;                      // [rows, groups, CHUNK]: C of the row against B of its chunk's tokens
  float* ends;                       // [chunk places, heads, VD, n]: end states, then the states before
  float* decays;                     // [chunk places, heads]: products over the chunk
  int* broken;                       // [chunks, groups, 2]: the first of a chunk's rows of B and C with a number that has no finite parts, or CHUNK
  bf16* parts;                       // [chunks, groups, B and C, n / 64, 3, CHUNK, TILE_PITCH]
  const int *seg_q_start, *seg_q_len, *seg_slot;
  int heads, groups;
  int segments, least;               // segments of `least` rows and more go in chunks
  int scans;                         // blocks per head that take the others token by token
  bool halves;                       // .. their first rows beside the ends, the others beside the outputs
};

__device__ __forceinline__ bool partless(const float4& v) {
  return !(fabsf(v.x) < PART_LIMIT && fabsf(v.y) < PART_LIMIT && fabsf(v.z) < PART_LIMIT && fabsf(v.w) < PART_LIMIT);
}

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

constexpr int PAIRS_THREADS = 256, PAIRS_ROWS = 32;

// A CTA takes 32 of a chunk's rows against its tokens up to them, a warp 16 rows and 16 tokens.  (By multiply-adds: 6.4 us beside 69 of the two
// products per head, 36 chunks of states of 128; errors of the sums 1.7 times as large.)  grid: (chunks, groups * 2)
template <int N>
__global__ void __launch_bounds__(PAIRS_THREADS)
space_pairs_kernel(SpaceArgs p) {
  constexpr int TILES = N / HALF_N, C_APART = PAIRS_ROWS * TILE_PITCH, PIECES = CHUNK * N / 4 / PAIRS_THREADS;
  extern __shared__ __align__(16) float shared[];
  bf16 *s_b = reinterpret_cast<bf16*>(shared), *s_c = s_b + TILES * 3 * TILE_APART;      // [TILES][3][rows][TILE_PITCH]
  pdl_wait();
  const int group = blockIdx.y >> 1, side = blockIdx.y & 1, t0 = side * PAIRS_ROWS;
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.x);
  if (seg < 0) return;
  const int first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK), tid = threadIdx.x;
  const float *B = p.B + (size_t)first * p.b_stride + (size_t)group * N, *C = p.C + (size_t)first * p.c_stride + (size_t)group * N;
  __shared__ int s_broken;
  if (tid == 0) s_broken = CHUNK;
  float4 v[PIECES + PIECES / 2];      // rows of B, then this CTA's of C; rows past the segment's end are zeros
#pragma unroll
  for (int k = 0; k < PIECES + PIECES / 2; ++k) {
    const bool of_c = k >= PIECES;
    const int idx = tid + (of_c ? k - PIECES : k) * PAIRS_THREADS, t = idx / (N / 4) + (of_c ? t0 : 0), i = idx % (N / 4) * 4;
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < count) v[k] = __ldcg(reinterpret_cast<const float4*>(of_c ? C + t * p.c_stride + i : B + t * p.b_stride + i));
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < PIECES + PIECES / 2; ++k)
    if (partless(v[k])) atomicMin(&s_broken, (tid + (k >= PIECES ? k - PIECES : k) * PAIRS_THREADS) / (N / 4) + (k >= PIECES ? t0 : 0));
  __syncthreads();
  const int broken = s_broken;
  {      // in parts here and (this CTA's half of both) for the kernels behind, zeros from a broken row on: its own rows go by multiply-adds
    bf16* to = p.parts + ((size_t)blockIdx.x * p.groups + group) * 2 * TILES * 3 * TILE_APART;
#pragma unroll
    for (int k = 0; k < PIECES + PIECES / 2; ++k) {
      const bool of_c = k >= PIECES;
      const int idx = tid + (of_c ? k - PIECES : k) * PAIRS_THREADS, row = idx / (N / 4), i = idx % (N / 4) * 4, tile = i / HALF_N;
      const int t = row + (of_c ? t0 : 0);
      if (t >= broken) v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const uint32_t low = take_part(v[k].x, v[k].y), high = take_part(v[k].z, v[k].w);
        bf16* here = of_c ? s_c + (tile * 3 + q) * C_APART : s_b + (tile * 3 + q) * TILE_APART;
        *reinterpret_cast<uint2*>(here + row * TILE_PITCH + i % HALF_N) = make_uint2(low, high);
        if (t / PAIRS_ROWS == side)
          *reinterpret_cast<uint2*>(to + (((of_c ? TILES : 0) + tile) * 3 + q) * TILE_APART + t * TILE_PITCH + i % HALF_N) = make_uint2(low, high);
      }
    }
  }
  if (tid == 0) p.broken[((size_t)blockIdx.x * p.groups + group) * 2 + side] = broken;
  if (t0 >= count) return;
  __syncthreads();
  float* pairs = p.pairs + ((size_t)first * p.groups + group) * CHUNK;
  const size_t pair_stride = (size_t)p.groups * CHUNK;
  if (broken < CHUNK) {
    for (int idx = tid; idx < PAIRS_ROWS * CHUNK; idx += PAIRS_THREADS) {
      const int t = t0 + idx / CHUNK, token = idx % CHUNK;
      if (t >= count || t < broken) continue;
      float sum = 0.f;
      if (token < count)
        for (int i = 0; i < N; ++i) sum = fmaf(C[t * p.c_stride + i], B[token * p.b_stride + i], sum);
      pairs[t * pair_stride + token] = sum;
    }
  }
  const int lane = tid & 31, warp = tid >> 5, tile = warp & 1, token0 = (warp >> 1) * 16, r = lane >> 2, c2 = (lane & 3) * 2;
  if (token0 > t0 + tile * 16) return;      // later than these rows
  float total[2][4], lead[2][4], low[2][4];
  clear(total);
  clear(lead);
  clear(low);
#pragma unroll
  for (int ks = 0; ks < N / 16; ++ks) {
    uint32_t a[3][4];
#pragma unroll
    for (int q = 0; q < 3; ++q)
      ldmatrix_x4(a[q], s_c + (ks / 4 * 3 + q) * C_APART + (tile * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * TILE_PITCH + ks % 4 * 16 + (lane >> 4) * 8);
    add_products<false, 1>(lead, low, a, s_b + ks / 4 * 3 * TILE_APART + (token0 + (lane & 7) + ((lane >> 4) << 3)) * TILE_PITCH + ks % 4 * 16 + ((lane >> 3) & 1) * 8,
                           0, TILE_APART);
    if (ks % 4 == 3) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          total[j][e] += lead[j][e];
          low[j][e] = with_dropped(lead[j][e], low[j][e], DROPPED);
        }
      clear(lead);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = t0 + tile * 16 + r + 8 * i;
    if (t >= min(count, broken)) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      *reinterpret_cast<float2*>(pairs + t * pair_stride + token0 + j * 8 + c2) =
          make_float2(total[j][2 * i] + low[j][2 * i], total[j][2 * i + 1] + low[j][2 * i + 1]);
  }
  pdl_trigger();
}

// Parts of 64 entries of a chunk's rows of B (which 0) or C (1) into shared memory, as they are.
template <int N>
__device__ __forceinline__ void fetch_parts(bf16* dst, const SpaceArgs& p, int chunk_index, int group, int which, int part) {
  const bf16* from = p.parts + ((((size_t)chunk_index * p.groups + group) * 2 + which) * (N / HALF_N) + part) * 3 * TILE_APART;
#pragma unroll 4
  for (int idx = threadIdx.x; idx < 3 * TILE_APART / 8; idx += SPACE_THREADS)
    copy_async_16(reinterpret_cast<float*>(dst + idx * 8), reinterpret_cast<const float*>(from + idx * 8));
}
__device__ __forceinline__ int parts_broken(const SpaceArgs& p, int chunk_index, int group) {
  const int2 first = *reinterpret_cast<const int2*>(p.broken + ((size_t)chunk_index * p.groups + group) * 2);
  return min(first.x, first.y);
}
// Four neighbouring numbers of a row of 64 in parts.
__device__ __forceinline__ void store_tile(bf16* tile, int row, int i, float4 v) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const uint32_t low = take_part(v.x, v.y), high = take_part(v.z, v.w);
    *reinterpret_cast<uint2*>(tile + q * TILE_APART + row * TILE_PITCH + i) = make_uint2(low, high);
  }
}
// Step sizes and decays of a chunk's tokens, one thread each; tokens behind the segment's end change nothing.
__device__ __forceinline__ void token_steps(const SpaceArgs& p, float* s_dt, float* s_g, int first, int count, int head, float rate, float bias) {
  const int t = threadIdx.x;
  if (t >= CHUNK) return;
  float dt = 0.f;
  if (t < count) {
    const float z = p.dt_raw[(size_t)(first + t) * p.dt_stride + head] + bias;
    dt = z > 20.f ? z : log1pf(expf(z));
  }
  s_dt[t] = dt;
  s_g[t] = t < count ? expf(-rate * dt) : 1.f;
}
constexpr int X_PIECES = CHUNK * VD / 4 / SPACE_THREADS;
// A chunk's inputs of a head, four numbers of a row per piece; rows behind the segment's end are zeros.
__device__ __forceinline__ void ask_inputs(float4 (&x)[X_PIECES], const SpaceArgs& p, int first, int count, int head) {
#pragma unroll
  for (int k = 0; k < X_PIECES; ++k) {
    const int idx = threadIdx.x + k * SPACE_THREADS, t = idx / (VD / 4), i = idx % (VD / 4) * 4;
    x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < count) x[k] = __ldcg(reinterpret_cast<const float4*>(p.x + (size_t)(first + t) * p.x_stride + (size_t)head * VD + i));
  }
}

// ---------------------------------------------------------------- what a chunk's tokens leave behind
// The kernels' arguments are grid constants: the functions that are not inlined take them by address, and a copy on the stack of every thread (192 bytes) cost
// 2,048 rows of 32 heads 118 instead of 112 us, one request of 512 rows 48 and 46.
// By multiply-adds: step sizes times inputs [CHUNK][VD], then 64 entries of the rows of B.
template <int N>
__device__ __noinline__ void ends_plain(const SpaceArgs& p, float* shared, const float* s_factor, float* to, int first, int count,
                                        int head, int group, int part) {
  float *s_x = shared, *s_b = shared + CHUNK * VD;
  float4 x[X_PIECES];
  ask_inputs(x, p, first, count, head);
#pragma unroll
  for (int k = 0; k < X_PIECES; ++k) {
    const int idx = threadIdx.x + k * SPACE_THREADS;
    const float f = s_factor[idx / (VD / 4)];
    *reinterpret_cast<float4*>(s_x + idx * 4) = make_float4(x[k].x * f, x[k].y * f, x[k].z * f, x[k].w * f);
  }
  fetch_rows<HALF_N, SPACE_THREADS>(s_b, HALF_N, p.B + (size_t)first * p.b_stride + (size_t)group * N + part * HALF_N, p.b_stride, count);
  copy_async_commit();
  copy_async_wait<0>();
  __syncthreads();
  // value channels j .. j + 7, state entries i .. i + 3
  const int i = (threadIdx.x & 15) * 4, j = (threadIdx.x >> 4) * 8;
  float end[8][4] = {};
#pragma unroll 4
  for (int s = 0; s < CHUNK; ++s) {
    float b[4], v[8];
    load_columns<4>(reinterpret_cast<float (&)[4]>(v[0]), s_x + s * VD + j);
    load_columns<4>(reinterpret_cast<float (&)[4]>(v[4]), s_x + s * VD + j + 4);
    load_columns<4>(b, s_b + s * HALF_N + i);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
#pragma unroll
      for (int c = 0; c < 4; ++c) end[r][c] = fmaf(v[r], b[c], end[r][c]);
    }
  }
#pragma unroll
  for (int r = 0; r < 8; ++r) store_columns<4>(to + (size_t)(j + r) * N + i, end[r]);
}

// Segments that go token by token have blocks beside the ends.  What follows waits for them, so where the chunks are a round of the outputs' blocks or less and a
// segment is longer than those take, half of its rows go beside the outputs.  In us, all beside the ends / halves: 300, 100 and 70 rows 44 / 38 (14 heads) and
// 60 / 56 (32 heads), 1,000 and three of 100 rows 52 / 47 (224 blocks); but 99 / 101 (512 blocks) and, of 1,531, 77, 1 and 439 rows of 32 heads, 116 / 120.
// Staged 16 tokens at a time, their shared memory leaves the ends their four blocks per SM: 400 rows beside 64 decoded ones, 32 heads, 93 us with 32 tokens, 83 so.
constexpr int SCAN_STAGED = 16;
template <int N>
struct ScanShape {
  static constexpr int SL = N / SCAN_NPT, PARTS = VD * SL / SCAN_THREADS;      // blocks of a head
};
template <int N>
__device__ __forceinline__ ScanArgs scan_args(const SpaceArgs& p) {
  return {p.x, p.B, p.C, p.dt_raw, p.x_stride, p.b_stride, p.c_stride, p.dt_stride, p.dt_bias, p.A_log, p.D, p.states, p.y,
          p.seg_q_start, p.seg_q_len, p.seg_slot, p.heads, VD, N, p.groups, p.least - 1};
}

constexpr size_t ENDS_SHARED = 2 * TILE_BYTES;      // inputs and B in parts
static_assert(ENDS_SHARED >= sizeof(float) * CHUNK * (VD + HALF_N), "by multiply-adds");

// A CTA takes 64 entries of the state, a warp 16 value channels of them.  grid: (heads * n / 64, scans + chunks)
template <int N, bool SCANS>
__global__ void __launch_bounds__(SPACE_THREADS, 4)
space_ends_kernel(const __grid_constant__ SpaceArgs p) {
  extern __shared__ __align__(16) float shared[];
  __shared__ float s_g[CHUNK], s_dt[CHUNK], s_factor[CHUNK];      // decays, step sizes, the latter times the decays' product behind a token
  const int head = blockIdx.x / (N / HALF_N), part = blockIdx.x % (N / HALF_N);
  if (SCANS && (int)blockIdx.y < p.scans / (N / HALF_N)) {
    constexpr int TAKEN = ScanShape<N>::PARTS / (N / HALF_N);
    scan_segment<ScanShape<N>::SL, true, SCAN_STAGED>(scan_args<N>(p), shared, blockIdx.y / TAKEN, head, blockIdx.y % TAKEN * (N / HALF_N) + part,
                                              p.halves ? FIRST_HALF : ALL_ROWS);
    return;
  }
  bf16 *s_x = reinterpret_cast<bf16*>(shared), *s_b = s_x + 3 * TILE_APART;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float rate = expf(p.A_log[head]), bias = p.dt_bias[head];
  pdl_wait();
  const int index = SCANS ? (int)blockIdx.y - p.scans / (N / HALF_N) : blockIdx.y;
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, index);
  if (seg < 0) return;
  const int first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK), group = head / (p.heads / p.groups);
  fetch_parts<N>(s_b, p, index, group, 0, part);
  copy_async_commit();
  float4 x[X_PIECES];
  ask_inputs(x, p, first, count, head);
  bool bad = parts_broken(p, index, group) < CHUNK;
  token_steps(p, s_dt, s_g, first, count, head, rate, bias);
  __syncthreads();
  const size_t place = chunk_place(first, chunk == 0) * p.heads + head;
  if (tid < CHUNK) {
    double product = 1.;
    for (int t = tid + 1; t < CHUNK; ++t) product *= s_g[t];
    s_factor[tid] = (float)(s_dt[tid] * product);
    if (tid == 0 && part == 0) p.decays[place] = (float)(product * s_g[0]);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < X_PIECES; ++k) {
    const int idx = tid + k * SPACE_THREADS, t = idx / (VD / 4);
    const float f = s_factor[t];
    const float4 v = make_float4(x[k].x * f, x[k].y * f, x[k].z * f, x[k].w * f);
    bad |= partless(v);
    store_tile(s_x, t, idx % (VD / 4) * 4, v);
  }
  copy_async_wait<0>();
  bad = __syncthreads_or(bad);
  float* to = p.ends + place * VD * N + part * HALF_N;
  if (bad) {
    ends_plain<N>(p, shared, s_factor, to, first, count, head, group, part);
    return;
  }
  const int r = lane >> 2, c2 = (lane & 3) * 2;
  float lead[8][4], low[8][4];
  clear(lead);
  clear(low);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    uint32_t a[3][4];
#pragma unroll
    for (int q = 0; q < 3; ++q)
      ldmatrix_x4_trans(a[q], s_x + q * TILE_APART + (ks * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * TILE_PITCH + warp * 16 + ((lane >> 3) & 1) * 8);
    add_products<true, 4>(lead, low, a, s_b + (ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * TILE_PITCH + (lane >> 4) * 8, 16, TILE_APART);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float2 e;
      e.x = lead[j][2 * i] + with_dropped(lead[j][2 * i], low[j][2 * i], ENDS_DROPPED);
      e.y = lead[j][2 * i + 1] + with_dropped(lead[j][2 * i + 1], low[j][2 * i + 1], ENDS_DROPPED);
      *reinterpret_cast<float2*>(to + (size_t)(warp * 16 + r + 8 * i) * N + j * 8 + c2) = e;
    }
  // At the end, in all of these kernels: blocks of the next that come in while these still fill some SMs land several to an SM beside empty ones.
  // Trigger in front / at the end (with arguments copied to the stack still): 14 heads of 64, 512 rows 30.5 / 23.9 us, 2,048 rows 51 / 46, 3 times 300 rows 34 / 29; 32 heads of 128, 2,048 rows 106 / 104.
  pdl_trigger();
}

// ---------------------------------------------------------------- the chunks of a segment in order
// A thread owns four neighbouring entries and takes the chunks of its segment in order; BATCH chunks are asked for together.  Leaves the state before
// every chunk where what its tokens left behind was.
// All launches from a flushed L2 (products by multiply-adds), batches of 8 / 16: 32 heads 132.4 / 128.0 us at 2,048 rows, 235 / 223 at 4,000, 128.4 / 126.7 for
// 1,531 + 77 + 1 + 439; 14 heads 59.8 / 58.3 and 97.8 / 89.5; segments of few chunks pay for the registers, 512 rows of 14 heads 37.3 / 38.8.
__global__ void __launch_bounds__(256)
space_carry_kernel(SpaceArgs p, int cells) {
  constexpr int BATCH = 16;
  pdl_wait();
  const auto [seg, which, length, start, slot] = chunk_at<false>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, blockIdx.y);
  if (seg < 0) return;
  const int first = start, chunks = (length + CHUNK - 1) / CHUNK;
  const int at = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (at >= p.heads * cells) return;
  const int head = at / cells, cell = at - head * cells;
  auto place_of = [&](int chunk) { return chunk_place(first + chunk * CHUNK, chunk == 0) * p.heads + head; };
  float4* state = reinterpret_cast<float4*>(p.states + ((size_t)slot * p.heads + head) * cells + cell);
  float4 S = *state;
  for (int c0 = 0; c0 < chunks; c0 += BATCH) {
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
  *state = S;
  pdl_trigger();
}

// ---------------------------------------------------------------- outputs
// Rows from `from` on by multiply-adds: weights in s_w; inputs, then the state before and the rows of C, behind and over them.
template <int N>
__device__ __noinline__ void outputs_plain(const SpaceArgs& p, float* s_w, const float* s_dt, const float* s_since, const float* before, int from, int first,
                                           int count, int head, int group, float skip) {
  constexpr int PITCH = N + 4;
  float* s_x = s_w + CHUNK * W_PITCH;
  const int tid = threadIdx.x;
  float4 piece[X_PIECES];
  ask_inputs(piece, p, first, count, head);
#pragma unroll
  for (int k = 0; k < X_PIECES; ++k) {
    const int idx = tid + k * SPACE_THREADS;
    const float dt = s_dt[idx / (VD / 4)];
    *reinterpret_cast<float4*>(s_x + idx * 4) = make_float4(piece[k].x * dt, piece[k].y * dt, piece[k].z * dt, piece[k].w * dt);
  }
  __syncthreads();
  // the chunk's own tokens: rows t, t + 8, .., value channels j .. j + 3; rows before a token have no part in it (where a step of k mixes
  // both, the later tokens are left out rather than weighed with zero: an infinity is theirs alone)
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
  // the state's rows and those of C take the place of what is done with
  __syncthreads();
  float *s_s = s_w, *s_c = s_w + VD * PITCH;
  for (int idx = tid; idx < VD * (N / 4); idx += SPACE_THREADS) copy_async_16(s_s + idx / (N / 4) * PITCH + idx % (N / 4) * 4, before + idx * 4);
  fetch_rows<N, SPACE_THREADS>(s_c, PITCH, p.C + (size_t)first * p.c_stride + (size_t)group * N, p.c_stride, count);
  copy_async_commit();
  copy_async_wait<0>();
  __syncthreads();
  float read[8][4] = {};
  for (int i0 = 0; i0 < N; i0 += 16) {      // sums of 16 entries each, then of those
    float sum[8][4] = {};
#pragma unroll 2
    for (int i = i0; i < i0 + 16; i += 4) {
      float s[4][4];
#pragma unroll
      for (int c = 0; c < 4; ++c) load_columns<4>(s[c], s_s + (j + c) * PITCH + i);
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
      for (int c = 0; c < 4; ++c) read[k][c] += sum[k][c];
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int row = t + 8 * k;
    if (row >= count || row < from) continue;
    float y[4];
    load_columns<4>(y, p.x + (size_t)(first + row) * p.x_stride + (size_t)head * VD + j);
#pragma unroll
    for (int c = 0; c < 4; ++c) y[c] = fmaf(s_since[row], read[k][c], fmaf(skip, y[c], acc[k][c]));
    store_columns<4>(p.y + ((size_t)(first + row) * p.heads + head) * VD + j, y);
  }
}

constexpr size_t WEIGHT_BYTES = CHUNK * W_PITCH * sizeof(float);
constexpr size_t OUTPUTS_SHARED = WEIGHT_BYTES + 2 * TILE_BYTES;      // weights, inputs (then a part of the state), a part of C
static_assert(OUTPUTS_SHARED >= sizeof(float) * (VD + CHUNK) * (128 + 4), "by multiply-adds");

// A warp takes 16 rows.  grid: (heads, scans + chunks)
template <int N, bool SCANS>
__global__ void __launch_bounds__(SPACE_THREADS, 3)
space_outputs_kernel(const __grid_constant__ SpaceArgs p) {
  extern __shared__ __align__(16) float shared[];
  __shared__ float s_g[CHUNK], s_dt[CHUNK], s_since[CHUNK];      // decays, step sizes, decays' product from the chunk's start on
  __shared__ int s_broken;                                       // the first row that goes by multiply-adds
  float* s_w = shared;                                                                                 // [CHUNK][W_PITCH]: weight of token s in row t
  bf16 *s_x = reinterpret_cast<bf16*>(s_w + CHUNK * W_PITCH), *s_c = s_x + 3 * TILE_APART;
  if (SCANS && (int)blockIdx.y < (p.halves ? p.scans : 0)) {
    constexpr int PARTS = ScanShape<N>::PARTS;
    scan_segment<ScanShape<N>::SL, true, SCAN_STAGED>(scan_args<N>(p), shared, blockIdx.y / PARTS, blockIdx.x, blockIdx.y % PARTS, SECOND_HALF);
    return;
  }
  const int head = blockIdx.x, index = SCANS && p.halves ? (int)blockIdx.y - p.scans : blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float rate = expf(p.A_log[head]), bias = p.dt_bias[head], skip = p.D[head];
  pdl_wait();
  const auto [seg, chunk, length, start, slot] = chunk_at<true>(p.seg_q_start, p.seg_q_len, p.seg_slot, p.segments, p.least, index);
  if (seg < 0) return;
  const int first = start + chunk * CHUNK, count = min(CHUNK, length - chunk * CHUNK), group = head / (p.heads / p.groups);
  fetch_rows<CHUNK, SPACE_THREADS>(s_w, W_PITCH, p.pairs + ((size_t)first * p.groups + group) * CHUNK, (long long)p.groups * CHUNK, count);
  copy_async_commit();
  fetch_parts<N>(s_c, p, index, group, 1, 0);
  copy_async_commit();
  float4 x[X_PIECES];
  ask_inputs(x, p, first, count, head);
  if (tid == 0) s_broken = parts_broken(p, index, group);
  token_steps(p, s_dt, s_g, first, count, head, rate, bias);
  copy_async_wait<1>();
  __syncthreads();
  int broken = CHUNK;      // as this thread sees it
  {
    // thread (s, half): the weights of token s in the rows of one half, the product of the decays growing along the rows
    const int s = tid & (CHUNK - 1), half = tid / CHUNK;
    double product = 1.;
    if (half == 1)
      for (int t = s + 1; t < CHUNK / 2; ++t) product *= s_g[t];
#pragma unroll 8
    for (int t = half * (CHUNK / 2); t < (half + 1) * (CHUNK / 2); ++t) {
      if (t > s) product *= s_g[t];
      float& w = s_w[t * W_PITCH + s];
      const float weight = t >= s ? (float)(w * product) : 0.f;
      if (!(fabsf(weight) < PART_LIMIT)) broken = min(broken, t);
      w = weight;
      if (s == 0) s_since[t] = (float)(product * s_g[0]);
    }
  }
#pragma unroll
  for (int k = 0; k < X_PIECES; ++k) {
    const int idx = tid + k * SPACE_THREADS, t = idx / (VD / 4);
    const float dt = s_dt[t];
    x[k] = make_float4(x[k].x * dt, x[k].y * dt, x[k].z * dt, x[k].w * dt);
    if (partless(x[k])) broken = min(broken, t);
  }
  if (broken < CHUNK) atomicMin(&s_broken, broken);
  __syncthreads();
  broken = s_broken;
#pragma unroll
  for (int k = 0; k < X_PIECES; ++k) {      // rows before a broken one give it a weight of zero, which must not meet an infinity
    const int idx = tid + k * SPACE_THREADS, t = idx / (VD / 4);
    store_tile(s_x, t, idx % (VD / 4) * 4, t < broken ? x[k] : make_float4(0.f, 0.f, 0.f, 0.f));
  }
  const float* before = p.ends + (chunk_place(first, chunk == 0) * p.heads + head) * VD * N;
  // 64 entries of the state before the chunk, a row's 16 pieces side by side
  float4 piece[X_PIECES];
  auto ask_state = [&](int part) {
#pragma unroll
    for (int k = 0; k < X_PIECES; ++k) {
      const int idx = tid + k * SPACE_THREADS;
      piece[k] = __ldcg(reinterpret_cast<const float4*>(before + (size_t)(idx / (HALF_N / 4)) * N + part * HALF_N + idx % (HALF_N / 4) * 4));
    }
  };
  ask_state(0);
  __syncthreads();
  const int r = lane >> 2, c2 = (lane & 3) * 2;
  float lead[8][4], low[8][4], total[8][4];
  clear(lead);
  clear(low);
  if (broken > 0) {
    bool bad = false;      // a number of the state without parts: every row sees it
    for (int ks = 0; ks <= warp; ++ks) {      // the chunk's own tokens; later ones are not seen
      float w[2][4];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float* from = s_w + (warp * 16 + r) * W_PITCH + ks * 16 + j * 8 + c2;
        const float2 top = *reinterpret_cast<const float2*>(from), bottom = *reinterpret_cast<const float2*>(from + 8 * W_PITCH);
        w[j][0] = top.x; w[j][1] = top.y; w[j][2] = bottom.x; w[j][3] = bottom.y;
      }
      uint32_t a[3][4];
      split_operand(a, w[0], w[1]);
      add_products<true, 4>(lead, low, a, s_x + (ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * TILE_PITCH + (lane >> 4) * 8, 16, TILE_APART);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        total[j][e] = lead[j][e] + with_dropped(lead[j][e], low[j][e], DROPPED);
        lead[j][e] = low[j][e] = 0.f;
      }
    const float since[2] = {s_since[warp * 16 + r], s_since[warp * 16 + r + 8]};
    float read[N > HALF_N ? 8 : 1][4];      // of the entries before
#pragma unroll
    for (int part = 0; part < N / HALF_N; ++part) {
      __syncthreads();      // what lies there has been read
      if (part > 0) {
        fetch_parts<N>(s_c, p, index, group, 1, part);
        copy_async_commit();
      }
#pragma unroll
      for (int k = 0; k < X_PIECES; ++k) {
        const int idx = tid + k * SPACE_THREADS;
        bad |= partless(piece[k]);
        store_tile(s_x, idx / (HALF_N / 4), idx % (HALF_N / 4) * 4, piece[k]);
      }
      if (part + 1 < N / HALF_N) ask_state(part + 1);
      copy_async_wait<0>();
      bad = __syncthreads_or(bad);
      if (bad) break;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint32_t a[3][4];
#pragma unroll
        for (int q = 0; q < 3; ++q)
          ldmatrix_x4(a[q], s_c + q * TILE_APART + (warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * TILE_PITCH + ks * 16 + (lane >> 4) * 8);
        add_products<false, 4>(lead, low, a, s_x + ((lane & 7) + ((lane >> 4) << 3)) * TILE_PITCH + ks * 16 + ((lane >> 3) & 1) * 8, 16 * TILE_PITCH, TILE_APART);
      }
      if (part + 1 < N / HALF_N) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            read[N > HALF_N ? j : 0][e] = lead[j][e];
            low[j][e] = with_dropped(lead[j][e], low[j][e], DROPPED);
            lead[j][e] = 0.f;
          }
      }
    }
    if (!bad) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = warp * 16 + r + 8 * i;
        if (t >= min(count, broken)) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 own = *reinterpret_cast<const float2*>(p.x + (size_t)(first + t) * p.x_stride + (size_t)head * VD + j * 8 + c2);
          float y[2] = {own.x, own.y};
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float sum = lead[j][2 * i + e];
            const float rest = with_dropped(sum, low[j][2 * i + e], DROPPED);
            if (N > HALF_N) sum += read[N > HALF_N ? j : 0][2 * i + e];
            y[e] = fmaf(since[i], sum + rest, fmaf(skip, y[e], total[j][2 * i + e]));
          }
          *reinterpret_cast<float2*>(p.y + ((size_t)(first + t) * p.heads + head) * VD + j * 8 + c2) = make_float2(y[0], y[1]);
        }
      }
      if (broken >= CHUNK) return;
    } else {
      broken = 0;
    }
  }
  // the weights are where they were; the inputs come again
  copy_async_wait<0>();
  __syncthreads();
  outputs_plain<N>(p, s_w, s_dt, s_since, before, broken, first, count, head, group, skip);
  pdl_trigger();
}

template <int N, bool SCANS>
int launch_space(const SpaceArgs& a, int rows, cudaStream_t stream) {
  constexpr size_t pairs_shared = (N / HALF_N) * 3 * TILE_PITCH * (CHUNK + PAIRS_ROWS) * sizeof(bf16);
  const size_t segment_shared = scan_shared(N, SCAN_THREADS / (N / SCAN_NPT), SCAN_STAGED);
  const size_t ends_shared = SCANS && segment_shared > ENDS_SHARED ? segment_shared : ENDS_SHARED;
  if (SCANS && segment_shared > OUTPUTS_SHARED) return MLR_TOO_LARGE;
  const unsigned chunks = (unsigned)long_chunks(rows, a.segments, a.least);
  static OncePerDevice once;
  const cudaError_t err = once([&] {
    cudaError_t err = cudaFuncSetAttribute(space_pairs_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pairs_shared);
    if (err == cudaSuccess) err = cudaFuncSetAttribute(space_ends_kernel<N, SCANS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ends_shared);
    if (err == cudaSuccess) err = cudaFuncSetAttribute(space_outputs_kernel<N, SCANS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OUTPUTS_SHARED);
    return err;
  });
  if (err != cudaSuccess) return (int)err;
  launch_kernel(space_pairs_kernel<N>, dim3(chunks, a.groups * 2), dim3(PAIRS_THREADS), pairs_shared, stream, a);
  int status = launch_status();
  if (status != MLR_OK) return status;
  launch_kernel(space_ends_kernel<N, SCANS>, dim3(a.heads * (N / HALF_N), a.scans / (N / HALF_N) + chunks), dim3(SPACE_THREADS), ends_shared, stream, a);
  if ((status = launch_status()) != MLR_OK) return status;
  launch_kernel(space_carry_kernel, dim3((a.heads * VD * N / 4 + 255) / 256, (unsigned)long_segments(rows, a.segments, a.least)), dim3(256), 0,
                stream, a, VD * N);
  if ((status = launch_status()) != MLR_OK) return status;
  launch_kernel(space_outputs_kernel<N, SCANS>, dim3(a.heads, (a.halves ? a.scans : 0) + chunks), dim3(SPACE_THREADS), OUTPUTS_SHARED, stream, a);
  return launch_status();
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// float32 scratch of a step, in numbers: end states first (16-byte aligned), the parts of B and C, then pairs, products over the chunks and the
// first broken rows.
MLR_EXPORT long long mlr_state_space_chunk_scratch(int rows, int segments, int least_rows, int heads, int n, int groups) {
  return chunk_places(rows) * heads * (VD * (long long)n + 1) + long_chunks(rows, segments, least_rows) * groups * (3ll * TILE_APART * (n / HALF_N) + 2) +
         (long long)rows * groups * CHUNK;
}

// As mlr_state_space_scan, for heads of 64 value channels with states of 64 or 128 entries and x, B, C, states, y and scratch whose
// rows begin on 16-byte boundaries.  rows: the step's rows.  Segments of fewer than least_rows rows
// go token by token as there; others: the longest of those, or what it may be (0: there are none).
MLR_EXPORT int mlr_state_space_chunks(const float* x, long long x_stride, const float* B, long long b_stride, const float* C,
                                      long long c_stride, const float* dt_raw, long long dt_stride, const float* dt_bias,
                                      const float* A_log, const float* D, float* states, float* y, float* scratch,
                                      const int* seg_q_start, const int* seg_q_len, const int* seg_slot, int segments, int rows,
                                      int max_q_len, int least_rows, int others, int heads, int vdim, int n, int groups, cudaStream_t stream) {
  if (segments == 0) return MLR_OK;
  if (segments < 0 || least_rows <= CHUNK || rows <= 0 || max_q_len < least_rows || heads <= 0 || groups <= 0 || heads % groups != 0 || scratch == nullptr)
    return MLR_BAD_SIZE;
  if (vdim != VD || (n != 64 && n != 128) || long_chunks(rows, segments, least_rows) + segments * 4ll > 65535 || groups > 65535 / 2) return MLR_TOO_LARGE;
  const uintptr_t pointers = (uintptr_t)x | (uintptr_t)B | (uintptr_t)C | (uintptr_t)states | (uintptr_t)y | (uintptr_t)scratch;
  if (pointers % 16 != 0 || (x_stride | b_stride | c_stride) % 4 != 0) return MLR_BAD_ALIGNMENT;
  const int parts = n / HALF_N, scans = others ? segments * (VD * (n / SCAN_NPT) / SCAN_THREADS) : 0;
  const size_t chunks = (size_t)long_chunks(rows, segments, least_rows);
  SpaceArgs a{x, B, C, dt_raw, x_stride, b_stride, c_stride, dt_stride, dt_bias, A_log, D, states, y,
              nullptr, scratch, nullptr, nullptr, nullptr, seg_q_start, seg_q_len, seg_slot, heads, groups, segments, least_rows, scans,
              others > CHUNK && chunks * heads <= 3 * (size_t)sm_count()};
  a.parts = reinterpret_cast<bf16*>(a.ends + (size_t)chunk_places(rows) * heads * VD * n);
  a.pairs = reinterpret_cast<float*>(a.parts + chunks * groups * parts * 6 * TILE_APART);
  a.decays = a.pairs + (size_t)rows * groups * CHUNK;
  a.broken = reinterpret_cast<int*>(a.decays + (size_t)chunk_places(rows) * heads);      // an even number of them: read in pairs
  if (others) return n == 64 ? launch_space<64, true>(a, rows, stream) : launch_space<128, true>(a, rows, stream);
  return n == 64 ? launch_space<64, false>(a, rows, stream) : launch_space<128, false>(a, rows, stream);
}
