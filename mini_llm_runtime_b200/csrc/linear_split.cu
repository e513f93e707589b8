// y[M,N] = x[M,K] * W[N,K]^T (+ bias[N]) of float32 operands on the 5th-generation tensor cores.
//
// A float32 number is the sum of three bfloat16 numbers (8 significand bits each, the remainder of each rounding being exact):
// x = x0 + x1 + x2.  Of the nine products of parts the six that reach 2^-24 of the whole are taken, smallest first:
// x2 w0, x0 w2, x1 w1, x1 w0, x0 w1, x0 w0; what is left out is below 2^-26.  Numbers below 2^-109 in magnitude lose bits of
// their last part, at most 2^-134 of them.  The tensor cores' sums drop bits at every step, always downwards, so they are
// kept short: the accumulator of each block of 64 k starts at zero and is added in float32, rounded to nearest, to sums in registers.
//
// One CTA computes 128 output columns (weight rows: the MMA's rows) x BN rows of x, walking k in blocks of 64:
//   warps 0, 18   copy into shared memory (TMA): W tiles (float32, two boxes of 32 k), and the tiles of x's three parts
//   warp 1        issues the 24 MMAs of a block: A = parts of W in tensor memory, B = parts of x in shared memory.  The tensor core holds few
//                 MMAs beyond the running one, about 250 cycles of work, and a look at a barrier costs 150 even when it has been passed;
//                 so one barrier per block tells all: x is there, W's parts are there, the accumulator is read
//   warps 2..9    split W, four warps the even blocks and four the odd ones: a thread takes one row, stores its parts to tensor memory
//   warps 10..17  add each block's accumulator to their sums; write the tile
// x is split once by a kernel of its own (every W tile uses it), W inside (it is read from memory once, in float32).  Up to 32 rows
// warps 10..17 split x themselves, two blocks ahead of the accumulators they read, in every CTA: a launch less, and the tiles of W are asked for
// as soon as the kernel before is complete (1 row, cold weights, us per product of a chain: [896, 896] 7.9 with the launch, 6.2 without, 6.5 on
// the CUDA cores; [9728, 896] 14.3, 12.6, 14.2).  One more warp for all of x would have been the bound: [16384, 2048] 31 us at 1 row, 48 at 16;
// 27 and 28 so.
//
// Long sums of narrow outputs are cut into 2 to 8 parts along k, one CTA each, that form a cluster and exchange their
// sums through shared memory.  How k is cut depends on N and K alone and an element's additions on nothing else, so results do not
// depend on how rows are batched.
//
// An output that is not finite is computed again as one chain of fmaf over k: a part of an infinity times a part that is zero
// would have made NaN of it, and sums may pass the largest float on the way.  All warps of the CTA do so at its end, on the CUDA cores:
// 600 rows of NaN, [9728, 896], 0.85 ms.  (A chain per thread in the epilogue took 50 ms, while the MMA warp's bounded waits ran on, and its call
// cost the epilogue registers: 600 rows of a feed-forward, all finite, 141 us with it, 128 without.)
// Every wait is bounded; one that runs out stores a code into the error word and the CTA stops issuing work and returns.
//
// For many rows bound by the MMAs, six per product: 1,500 rows [16384, 2048] 2,461 us on the CUDA cores (41 TFLOP/s), 505 us here, 1.2
// PFLOP/s of bfloat16 multiply-adds, near what the power limit sustains.  For few by the stream of W: 8 rows [16384, 2048] 51 / 28 us,
// 4.8 TB/s; 600 rows [9728, 896] with its gate 318 / 83, [896, 4864] 173 / 70.  Errors against 64 bits (2-norm) at 896, 4,864 and
// 8,192 k: 1.1e-7, 1.1e-7, 1.2e-7, on the CUDA cores 5.4e-7, 6.2e-7, 8.1e-7.  One MMA of 128 x 128 x 16 takes 64 cycles
// either way, but of 128 x 16 x 16 takes 12 with its rows in tensor memory and 39 with them in shared memory.
#include "copy_async.cuh"
#include "float_parts.cuh"
#include "tcgen05.cuh"

namespace mlr {

constexpr int LS_ROWS = 128;                    // weight rows of a tile
constexpr int LS_K = 64;                        // k of a block
constexpr int LS_THREADS = 19 * 32;
constexpr uint32_t LS_RAW_BYTES = LS_ROWS * LS_K * 4;        // W tile, float32
constexpr int LS_MOST_PARTS = 8;                // CTAs that may share the sums over k
constexpr int LS_EXCHANGE = 16;                 // columns of x rows exchanged at a time by the gated epilogue

struct LinearSplitArgs {
  int M, N, K;
  int n_tiles, m_tiles, parts;      // parts: CTAs that share the sums over k
  const float *x, *w, *bias;
  float* out;                       // [M, N], gated: [M, N / 2]
  int* error_word;
};

template <int BN>
struct LinearSplitShape {
  static constexpr bool OWN_X = BN <= 32;                      // x is split here
  static constexpr int OWN_X_STAGES = BN == 16 ? 8 : BN == 32 ? 4 : 0;      // its tiles under way, in float32
  static constexpr uint32_t X_BYTES = 3u * BN * LS_K * 2;      // the three parts of a tile of x
  // even, so that a stage of the ring of W tiles is always converted by the same warps: a barrier's parity only tells phases apart to
  // those who wait for every one of them
  static constexpr int RAW_STAGES = BN >= 128 ? 2 : 4;
  static constexpr int X_STAGES = OWN_X ? 4 : 3;
  static_assert(RAW_STAGES % 2 == 0 && X_STAGES >= 3, "see above; arrivals for a block's stage come up to two blocks ahead of its MMAs");
  static constexpr uint32_t TMEM_COLS = 2 * BN + 192 <= 256 ? 256 : 512;      // two accumulators, two slots of three W parts of 32 columns
  static constexpr size_t EXCHANGE_BYTES = 2ull * LS_EXCHANGE * LS_ROWS * 4;
  static constexpr size_t SHARED = 1024 + RAW_STAGES * (size_t)LS_RAW_BYTES + X_STAGES * (size_t)X_BYTES + EXCHANGE_BYTES +
                                    OWN_X_STAGES * (size_t)BN * LS_K * 4;
  static_assert(SHARED <= 226 * 1024, "tiles fit the shared memory");
  static_assert((size_t)BN * LS_ROWS * 4 <= RAW_STAGES * (size_t)LS_RAW_BYTES, "a tile's sums fit where W's tiles were");
};

// parts [3][M][pitch], pitch = K rounded up to 8; what lies behind K becomes zero.  K % 4 == 0.
// It brings in the product only behind its own wait: so all that came before is complete when the product's first copies read W, which may
// have been written by the kernel just before.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* x, uint2* parts, int M, int K, int pitch) {
  pdl_wait();
  pdl_trigger();
  const int per_row = pitch / 4;
  const bool wide = ((uintptr_t)x & 15) == 0;
  const long long count = (long long)M * per_row;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < count; i += (long long)gridDim.x * 256) {
    const int row = (int)(i / per_row), k = (int)(i - (long long)row * per_row) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < K) {
      const float* src = x + (size_t)row * K + k;
      if (wide) v = __ldcg(reinterpret_cast<const float4*>(src));
      else v = make_float4(__ldcg(src), __ldcg(src + 1), __ldcg(src + 2), __ldcg(src + 3));
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint32_t low = take_part(v.x, v.y), high = take_part(v.z, v.w);
      parts[p * count + i] = make_uint2(low, high);
    }
  }
}

__device__ __forceinline__ uint32_t ls_address_in_cta(uint32_t local, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}
__device__ __forceinline__ float4 ls_load_remote(uint32_t address) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(address) : "memory");
  return v;
}
__device__ __forceinline__ void ls_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void ls_tmem_load8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}

__device__ __forceinline__ float ls_output(const LinearSplitArgs& p, float v, int n) { return p.bias != nullptr ? v + p.bias[n] : v; }
__device__ __forceinline__ float ls_gated(float gate, float up) { return (gate / (1.f + expf(-gate))) * up; }

// Of the tile of 128 weight rows from n0 on and the rows of x from `m_begin` to below `m_end`, the outputs in memory that are not finite, again: sums as
// chains over k.  A thread of the first 512 takes weight rows 2 a, 2 a + 1 and the two 64 rows on (of a gated tile the ups of the same
// outputs) and X rows of x.  The whole CTA comes here; `tiles`: shared memory, 64 (132 + 16 X) numbers.
template <bool GATED, int X>
__device__ __noinline__ void ls_chains(const LinearSplitArgs& p, int n0, int m_begin, int m_end, float* tiles) {
  constexpr int STEP = 64, W_PITCH = 132, X_ROWS = 16 * X;
  float *w_tile = tiles, *x_tile = tiles + STEP * W_PITCH;      // [k][row]
  const int t = threadIdx.x, a = t & 31, group = t >> 5, width = GATED ? p.N >> 1 : p.N;
  const bool wide = ((uintptr_t)p.x & 15) == 0;
  for (int m0 = m_begin; m0 < m_end; m0 += X_ROWS) {
    // outputs: of row m0 + group * X + i columns column(0) .. column(3), gated columns column(0) and column(1)
    auto column = [&](int j) { return GATED ? (n0 >> 1) + 2 * a + j : n0 + 2 * a + (j & 1) + (j >> 1) * 64; };
    auto broken = [&](int i, int j) {
      const int m = m0 + group * X + i;
      return t < 512 && m < m_end && column(j) < width && !(fabsf(__ldcg(p.out + (size_t)m * width + column(j))) <= 3.402823466e38f);
    };
    bool any = false;
#pragma unroll
    for (int i = 0; i < X; ++i)
#pragma unroll
      for (int j = 0; j < (GATED ? 2 : 4); ++j) any |= broken(i, j);
    if (!__syncthreads_or(any)) continue;
    float sum[X][4];
#pragma unroll
    for (int i = 0; i < X; ++i) sum[i][0] = sum[i][1] = sum[i][2] = sum[i][3] = 0.f;
    for (int k0 = 0; k0 < p.K; k0 += STEP) {
#pragma unroll
      for (int at = t; at < (LS_ROWS + X_ROWS) * (STEP / 4); at += LS_THREADS) {
        const int row = at / (STEP / 4), k = at % (STEP / 4) * 4;
        const bool of_w = row < LS_ROWS;
        const int from = of_w ? n0 + row : m0 + row - LS_ROWS;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (from < (of_w ? p.N : m_end) && k0 + k < p.K) {
          const float* src = (of_w ? p.w : p.x) + (size_t)from * p.K + k0 + k;
          if (of_w || wide) v = __ldcg(reinterpret_cast<const float4*>(src));
          else v = make_float4(__ldcg(src), __ldcg(src + 1), __ldcg(src + 2), __ldcg(src + 3));
        }
        const int pitch = of_w ? W_PITCH : X_ROWS;
        float* dst = (of_w ? w_tile + row : x_tile + row - LS_ROWS) + k * pitch;
        dst[0] = v.x; dst[pitch] = v.y; dst[2 * pitch] = v.z; dst[3 * pitch] = v.w;
      }
      __syncthreads();
      const int steps = min(STEP, p.K - k0);
      if (t < 512) {
        for (int k = 0; k < steps; ++k) {
          const float2 low = *reinterpret_cast<const float2*>(w_tile + k * W_PITCH + 2 * a), high = *reinterpret_cast<const float2*>(w_tile + k * W_PITCH + 64 + 2 * a);
#pragma unroll
          for (int i = 0; i < X; ++i) {
            const float x = x_tile[k * X_ROWS + group * X + i];
            sum[i][0] = fmaf(x, low.x, sum[i][0]); sum[i][1] = fmaf(x, low.y, sum[i][1]);
            sum[i][2] = fmaf(x, high.x, sum[i][2]); sum[i][3] = fmaf(x, high.y, sum[i][3]);
          }
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < X; ++i)
#pragma unroll
      for (int j = 0; j < (GATED ? 2 : 4); ++j)
        if (broken(i, j)) {
          const int n = n0 + 2 * a + (j & 1) + (j >> 1) * 64;
          p.out[(size_t)(m0 + group * X + i) * width + column(j)] =
              GATED ? ls_gated(ls_output(p, sum[i][j], n), ls_output(p, sum[i][2 + (j & 1)], n + 64)) : ls_output(p, sum[i][j], n);
        }
  }
}

// grid: parts == 1: as many CTAs as fill the device (or tiles, if those are fewer), each taking every gridDim.x-th tile; else one
// cluster of `parts` CTAs per tile.  GATED: weight rows come in blocks of 64 gate rows and the 64 up rows of the same
// outputs; the tile's results are silu(gate) * up.
template <int BN, bool GATED>
__global__ void __launch_bounds__(LS_THREADS, 1)
linear_split_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ LinearSplitArgs p) {
  using Shape = LinearSplitShape<BN>;
  constexpr int RAW_STAGES = Shape::RAW_STAGES, X_STAGES = Shape::X_STAGES;
  constexpr uint32_t W_COLUMNS = 2 * BN;      // tensor memory: accumulators at 0 and BN, then W's parts
  extern __shared__ uint8_t ls_shared[];
  uint8_t* raw_tiles = (uint8_t*)(((uintptr_t)ls_shared + 1023) & ~(uintptr_t)1023);
  uint8_t* x_tiles = raw_tiles + RAW_STAGES * LS_RAW_BYTES;
  float* exchange = reinterpret_cast<float*>(x_tiles + X_STAGES * Shape::X_BYTES);
  // of every block: its x (1 arrival with the copies' bytes), its parts of W (4 warps) and the accumulator two blocks before (8 warps; where
  // they split x as well, these arrivals stand for it too)
  __shared__ uint64_t ready[X_STAGES];
  __shared__ uint64_t raw_full[RAW_STAGES], raw_empty[RAW_STAGES], x_empty[X_STAGES], done[2];      // done: a block's MMAs, by its parity
  __shared__ uint32_t tmem_holder;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < RAW_STAGES; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 4); }
    for (int s = 0; s < X_STAGES; ++s) { mbar_init(&ready[s], Shape::OWN_X ? 12 : 13); mbar_init(&x_empty[s], 1); }
    mbar_init(&done[0], 1);
    mbar_init(&done[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&w_map) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&x_map) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)), "r"(Shape::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fa_fence_before();
  __syncthreads();
  fa_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_holder, 0);
  pdl_trigger();

  const int part = blockIdx.x % p.parts;
  const int items = p.n_tiles * p.m_tiles, first_item = blockIdx.x / p.parts, item_step = gridDim.x / p.parts;
  const int all_blocks = (p.K + LS_K - 1) / LS_K;
  const int first_block = (int)((long long)all_blocks * part / p.parts), end_block = (int)((long long)all_blocks * (part + 1) / p.parts);
  bool gave_up = false;
  float probe = 0.f;      // not zero: this thread has written an output that is not finite

  if (warp == 0) {
    if (lane == 0) {
      if (Shape::OWN_X) pdl_wait();      // else W does not depend on the kernel before this one, split_rows_kernel
      int raw = 0;
      uint32_t turn = 0;
      for (int item = first_item; item < items; item += item_step) {
        const int n0 = (item % p.n_tiles) * LS_ROWS;
        for (int block = first_block; block < end_block; ++block) {
          if (turn > 0) fa_wait(&raw_empty[raw], (turn - 1) & 1, p.error_word, 41, gave_up);
          if (gave_up) break;
          mbar_expect_tx(&raw_full[raw], LS_RAW_BYTES);
          uint8_t* dst = raw_tiles + raw * LS_RAW_BYTES;
          tma_load_2d(&w_map, &raw_full[raw], dst, block * LS_K, n0);
          tma_load_2d(&w_map, &raw_full[raw], dst + LS_RAW_BYTES / 2, block * LS_K + 32, n0);
          if (++raw == RAW_STAGES) { raw = 0; ++turn; }
        }
        if (gave_up) break;
      }
    }
  } else if (warp == 18) {
    if (!Shape::OWN_X && lane == 0) {
      pdl_wait();
      int xs = 0;
      uint32_t turn = 0;
      for (int item = first_item; item < items; item += item_step) {
        const int m0 = item / p.n_tiles * BN;
        for (int block = first_block; block < end_block; ++block) {
          if (turn > 0) fa_wait(&x_empty[xs], (turn - 1) & 1, p.error_word, 42, gave_up);
          if (gave_up) break;
          mbar_expect_tx(&ready[xs], Shape::X_BYTES);
#pragma unroll
          for (int q = 0; q < 3; ++q)
            tma_load_2d(&x_map, &ready[xs], x_tiles + xs * Shape::X_BYTES + q * (BN * LS_K * 2), block * LS_K, q * p.M + m0);
          if (++xs == X_STAGES) { xs = 0; ++turn; }
        }
        if (gave_up) break;
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = fa_idesc(LS_ROWS, BN, false);
    const uint32_t x_address = __shfl_sync(0xffffffffu, smem_u32(x_tiles), 0);
    const uint32_t blocks = first_item < items ? (uint32_t)((items - first_item - 1) / item_step + 1) * (end_block - first_block) : 0;
    uint32_t xs = 0, turn = 0, slot = 0;
    bool good = true;
    for (uint32_t n = 0; n < blocks; ++n) {
      fa_wait(&ready[xs], turn & 1, p.error_word, 43, gave_up);
      good = __all_sync(0xffffffffu, !gave_up);      // the same in the whole warp: its control flow stays uniform
      if (!good) break;
      fa_fence_after();
      if (elect_one()) {
        // (part of W, part of x), the smallest products first
        constexpr int W_PART[6] = {0, 2, 1, 0, 1, 0}, X_PART[6] = {2, 0, 1, 1, 0, 0};
        const uint32_t d = tmem + slot * BN, a = tmem + W_COLUMNS + slot * 96;
        const uint64_t b = fa_desc_k_major(x_address + xs * Shape::X_BYTES);
#pragma unroll
        for (int q = 0; q < 6; ++q) {
#pragma unroll
          for (int k = 0; k < LS_K / 16; ++k)
            fa_mma_tmem(d, a + W_PART[q] * 32 + k * 8, b + (uint64_t)((X_PART[q] * (BN * LS_K * 2) + k * 32) >> 4), idesc,
                        q > 0 || k > 0 ? 1u : 0u);
        }
        fa_commit(&x_empty[xs]);
        fa_commit(&done[slot]);
      }
      __syncwarp();
      slot ^= 1;
      if (++xs == X_STAGES) { xs = 0; ++turn; }
    }
    // nobody else looks at the last blocks' x_empty: their arrivals must have come before the CTA ends
    if (good && blocks > 0) fa_wait(&x_empty[(blocks - 1) % X_STAGES], ((blocks - 1) / X_STAGES) & 1, p.error_word, 44, gave_up);
    __syncwarp();
  } else if (warp < 10) {
    const int quarter = warp & 3, group = (warp - 2) >> 2, row = quarter * 32 + lane;
    uint32_t n = 0;      // blocks so far
    for (int item = first_item; item < items; item += item_step) {
      for (int block = first_block; block < end_block; ++block, ++n) {
        if ((int)(n & 1) != group) continue;
        const uint32_t raw = n % RAW_STAGES, turn = n >> 1;
        fa_wait(&raw_full[raw], (n / RAW_STAGES) & 1, p.error_word, 46, gave_up);
        const uint32_t to = tmem + ((uint32_t)(quarter * 32) << 16) + W_COLUMNS + group * 96;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          const uint8_t* line = raw_tiles + raw * LS_RAW_BYTES + half * (LS_RAW_BYTES / 2) + row * 128;
          float v[32];
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float4 piece = *reinterpret_cast<const float4*>(line + ((c ^ (row & 7)) << 4));
            v[4 * c] = piece.x; v[4 * c + 1] = piece.y; v[4 * c + 2] = piece.z; v[4 * c + 3] = piece.w;
          }
          if (half == 1) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[raw]);
          }
          uint32_t parts[3][16];
#pragma unroll
          for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int i = 0; i < 16; ++i) parts[q][i] = take_part(v[2 * i], v[2 * i + 1]);
          if (half == 0) {
            if (turn > 0) fa_wait(&done[group], (turn - 1) & 1, p.error_word, 47, gave_up);      // the block before with these parts
            __syncwarp();
            fa_fence_after();
          }
#pragma unroll
          for (int q = 0; q < 3; ++q) fa_tmem_store16(to + q * 32 + half * 16, parts[q]);
        }
        fa_tmem_wait_st();
        fa_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ready[n % X_STAGES]);
      }
    }
  } else if (warp < 18) {
    constexpr int COLS = BN / 2;      // columns (rows of x) of this warp
    const int quarter = warp & 3, side = (warp - 10) >> 2, row = quarter * 32 + lane;
    uint32_t n = 0;      // blocks so far
    // Own x: half a warp per row, 2 (w + 8 i) and the next for piece i of the w-th warp; a lane reads only what it has copied itself.  A stage
    // is free: block n + 2 takes that of block n - 2, whose accumulator has been read.  Rows and columns behind the last are zeros.
    constexpr int PIECES = BN / 16, AHEAD = Shape::OWN_X ? Shape::OWN_X_STAGES - 1 : 0;
    const int c = lane & 15, pair = 2 * (warp - 10), turns = end_block - first_block;
    const int count = first_item < items ? ((items - first_item - 1) / item_step + 1) * turns : 0;
    const bool wide = ((uintptr_t)p.x & 15) == 0;
    uint8_t* raw_x = reinterpret_cast<uint8_t*>(exchange) + Shape::EXCHANGE_BYTES + (warp - 10) * (Shape::OWN_X_STAGES * PIECES * 512) + lane * 16;
    auto x_slot = [&](int stage, int i) {
      const int x_row = pair + 16 * i + (lane >> 4);
      return x_tiles + stage * Shape::X_BYTES + x_row * 128 + (((c >> 1) ^ (x_row & 7)) << 4) + (c & 1) * 8;
    };
    auto ask = [&](int block) {
      if (block < count) {
        const int k = (first_block + block % turns) * LS_K + c * 4;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
          const int x_row = pair + 16 * i + (lane >> 4);
          float* dst = reinterpret_cast<float*>(raw_x + ((block % (AHEAD + 1)) * PIECES + i) * 512);
          const float* src = p.x + (size_t)x_row * p.K + k;
          if (x_row >= p.M || k >= p.K) {
            *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
          } else if (wide) {
            copy_async_16(dst, src);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) copy_async_4(dst + e, src + e);
          }
        }
      }
      copy_async_commit();
    };
    auto split_x = [&](int block) {
      ask(block + AHEAD);
      copy_async_wait<AHEAD>();
      if (block >= count) return;
#pragma unroll
      for (int i = 0; i < PIECES; ++i)
        if (pair + 16 * i < p.M) {
          float4 v = *reinterpret_cast<const float4*>(raw_x + ((block % (AHEAD + 1)) * PIECES + i) * 512);
          uint8_t* dst = x_slot(block % X_STAGES, i);
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const uint32_t low = take_part(v.x, v.y), high = take_part(v.z, v.w);
            *reinterpret_cast<uint2*>(dst + q * (BN * LS_K * 2)) = make_uint2(low, high);
          }
        }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    };
    if constexpr (Shape::OWN_X) {
#pragma unroll
      for (int i = 0; i < PIECES; ++i)
        if (pair + 16 * i >= p.M) {
          for (int stage = 0; stage < X_STAGES; ++stage)
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(x_slot(stage, i) + q * (BN * LS_K * 2)) = make_uint2(0u, 0u);
        }
      pdl_wait();
      for (int block = 0; block < AHEAD; ++block) ask(block);
      split_x(0);
      split_x(1);
      __syncwarp();
    }
    if (lane == 0) {     // both accumulators are free
      mbar_arrive(&ready[0]);
      mbar_arrive(&ready[1]);
    }
    for (int item = first_item; item < items; item += item_step) {
      const int n0 = (item % p.n_tiles) * LS_ROWS, m0 = item / p.n_tiles * BN;
      float sum[COLS];
#pragma unroll
      for (int c = 0; c < COLS; ++c) sum[c] = 0.f;
      for (int block = first_block; block < end_block; ++block, ++n) {
        const uint32_t slot = n & 1;
        if constexpr (Shape::OWN_X) split_x((int)n + 2);
        fa_wait(&done[slot], (n >> 1) & 1, p.error_word, 48, gave_up);
        __syncwarp();
        fa_fence_after();
        const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + slot * BN + side * COLS;
        if constexpr (COLS >= 16) {
          constexpr int ROUND = COLS >= 32 ? 32 : 16;
#pragma unroll
          for (int c0 = 0; c0 < COLS; c0 += ROUND) {
            uint32_t r[ROUND];
#pragma unroll
            for (int c = 0; c < ROUND; c += 16) fa_tmem_load16(from + c0 + c, r + c);
            fa_tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < ROUND; ++c) sum[c0 + c] += __uint_as_float(r[c]);
          }
        } else {
          uint32_t r[8];
          ls_tmem_load8(from, r);
          fa_tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 8; ++c) sum[c] += __uint_as_float(r[c]);
        }
        fa_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ready[(n + 2) % X_STAGES]);
      }
      if (item == first_item) pdl_wait();      // before the first write
      if (p.parts > 1) {                       // the ring of W tiles has no more use: the sums go there, [column][row]
        float* mine = reinterpret_cast<float*>(raw_tiles);
#pragma unroll
        for (int c = 0; c < COLS; ++c) mine[(side * COLS + c) * LS_ROWS + row] = sum[c];
      } else if constexpr (!GATED) {
        if (n0 + row < p.N) {
#pragma unroll
          for (int c = 0; c < COLS; ++c) {
            const int m = m0 + side * COLS + c;
            if (m < p.M) {
              const float v = ls_output(p, sum[c], n0 + row);
              p.out[(size_t)m * p.N + n0 + row] = v;
              probe = fmaf(v, 0.f, probe);
            }
          }
        }
      } else {
        constexpr int STEP = COLS < LS_EXCHANGE ? COLS : LS_EXCHANGE;
        float* mine = exchange + side * LS_EXCHANGE * LS_ROWS;
        const int t = quarter * 32 + lane, inner = p.N >> 1;
        const int j = t & 63, out_col = (n0 >> 1) + j;
#pragma unroll
        for (int c0 = 0; c0 < COLS; c0 += STEP) {
          asm volatile("bar.sync %0, 128;" ::"r"(1 + side) : "memory");
#pragma unroll
          for (int c = 0; c < STEP; ++c) mine[c * LS_ROWS + row] = sum[c0 + c];
          asm volatile("bar.sync %0, 128;" ::"r"(1 + side) : "memory");
#pragma unroll
          for (int c = t >> 6; c < STEP; c += 2) {
            const int m = m0 + side * COLS + c0 + c;
            if (m < p.M) {
              const float v = ls_gated(ls_output(p, mine[c * LS_ROWS + j], n0 + j), ls_output(p, mine[c * LS_ROWS + 64 + j], n0 + 64 + j));
              p.out[(size_t)m * inner + out_col] = v;
              probe = fmaf(v, 0.f, probe);
            }
          }
        }
      }
    }
  }
  if (p.parts > 1) {
    __syncwarp();
    ls_cluster_sync();
    if (warp >= 10 && warp < 18) {
      // a warp takes a column (a row of x) of this CTA's share, a lane four of its 128 outputs
      const int mine = BN / p.parts, n0 = (first_item % p.n_tiles) * LS_ROWS, m0 = first_item / p.n_tiles * BN, n = n0 + 4 * lane;
      const uint32_t base = smem_u32(raw_tiles);
      for (int c = part * mine + warp - 10; c < (part + 1) * mine; c += 8) {
        const int m = m0 + c;
        if (m >= p.M) break;
        float4 piece[LS_MOST_PARTS];
#pragma unroll
        for (int q = 0; q < LS_MOST_PARTS; ++q)
          if (q < p.parts) piece[q] = ls_load_remote(ls_address_in_cta(base, q) + (uint32_t)(c * LS_ROWS + 4 * lane) * 4);
        float v[4] = {piece[0].x, piece[0].y, piece[0].z, piece[0].w};
#pragma unroll
        for (int q = 1; q < LS_MOST_PARTS; ++q)      // the parts in the order of k
          if (q < p.parts) { v[0] += piece[q].x; v[1] += piece[q].y; v[2] += piece[q].z; v[3] += piece[q].w; }
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < p.N) {
            v[e] = ls_output(p, v[e], n + e);
            if (!GATED) probe = fmaf(v[e], 0.f, probe);
          }
        if constexpr (!GATED) {
          float* dst = p.out + (size_t)m * p.N + n;
          if ((p.N & 3) == 0) {
            if (n < p.N) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (n + e < p.N) dst[e] = v[e];
          }
        } else {      // lanes 0 .. 15 hold gates, lanes 16 .. 31 the ups of the same outputs
          float r[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) r[e] = ls_gated(v[e], __shfl_down_sync(0xffffffffu, v[e], 16));
          if (lane < 16) {
            *reinterpret_cast<float4*>(p.out + (size_t)m * (p.N >> 1) + (n0 >> 1) + 4 * lane) = make_float4(r[0], r[1], r[2], r[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) probe = fmaf(r[e], 0.f, probe);
          }
        }
      }
    }
    __syncwarp();
    ls_cluster_sync();      // the others have read this CTA's sums
  }
  fa_fence_before();
  const bool chains = __syncthreads_or(probe != 0.f);
  if (warp == 1) {
    fa_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Shape::TMEM_COLS) : "memory");
  }
  if (chains && !__syncthreads_or(gave_up)) {      // every copy has arrived and been read: the tiles' memory is free
    float* tiles = reinterpret_cast<float*>(raw_tiles);
    constexpr int X = BN < 64 ? 1 : 4;
    static_assert(64 * (132 + 16 * X) * 4 <= RAW_STAGES * (size_t)LS_RAW_BYTES, "tiles of the chains");
    const int mine = BN / p.parts;      // rows of x of this CTA's share
    for (int item = first_item; item < items; item += item_step) {
      const int m_begin = item / p.n_tiles * BN + part * mine;
      ls_chains<GATED, X>(p, (item % p.n_tiles) * LS_ROWS, m_begin, min(p.M, m_begin + mine), tiles);
    }
  }
}

// ---------------------------------------------------------------- host side
// rows x K float32, row-major; box = [128 x 32], 128-byte swizzle, out-of-range reads give zero.
static bool float_tile_map(CUtensorMap* map, const void* base, long long rows, long long K) {
  auto encode = encode_tiled();
  if (encode == nullptr) return false;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K * 4};
  cuuint32_t box[2] = {32u, (cuuint32_t)LS_ROWS};
  cuuint32_t element_strides[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, element_strides,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// CTAs that share the sums over k of one output tile, each at least 192 k: as many as fill half of the device, beyond that clusters wait for
// room beside one another (us with 2, 4, 8 of them: [896, 4864] 1 row - 24 17, 600 rows - 79 71; [2048, 2048] 8 rows - 17 21, 600 - 70 91).
inline int split_parts(int N, int K) {
  const int tiles = (N + LS_ROWS - 1) / LS_ROWS, blocks = (K + LS_K - 1) / LS_K;
  int parts = LS_MOST_PARTS;
  while (parts > 1 && (parts * tiles > 74 || blocks < 3 * parts)) parts /= 2;
  return parts;
}

// Rows whose parts are in scratch at a time: at most 128 MB of them.
inline int split_block_rows(int M, int K) {
  const long long most = ((128ll << 20) / (6ll * ((K + 7) / 8 * 8))) / 128 * 128;
  return most < 128 ? 128 : most < M ? (int)most : M;
}

template <int BN, bool GATED>
static int launch_split(const LinearSplitArgs& p, const void* parts, int pitch, cudaStream_t stream) {
  using Shape = LinearSplitShape<BN>;
  auto kernel = linear_split_kernel<BN, GATED>;
  static bool configured = false;
  if (!configured) {
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape::SHARED);
    if (err != cudaSuccess) return (int)err;
    configured = true;
  }
  CUtensorMap w_map, x_map;
  if (!float_tile_map(&w_map, p.w, p.N, p.K)) return MLR_BAD_ALIGNMENT;
  if (Shape::OWN_X) x_map = w_map;      // not read
  else if (!make_tile_map(&x_map, parts, 3ll * p.M, pitch, BN)) return MLR_BAD_ALIGNMENT;
  const int items = p.n_tiles * p.m_tiles;
  if (p.parts > 1) {
    launch_kernel_clustered(kernel, dim3(items * p.parts), dim3(LS_THREADS), Shape::SHARED, stream, p.parts, w_map, x_map, p);
  } else {
    launch_kernel(kernel, dim3(items < sm_count() ? items : sm_count()), dim3(LS_THREADS), Shape::SHARED, stream, w_map, x_map, p);
  }
  return launch_status();
}

template <bool GATED>
static int launch_split_width(LinearSplitArgs p, const void* parts, int pitch, cudaStream_t stream) {
  const int bn = p.M <= 16 ? 16 : p.M <= 32 ? 32 : p.M <= 64 ? 64 : 128;
  p.m_tiles = (p.M + bn - 1) / bn;
  if (bn == 16) return launch_split<16, GATED>(p, parts, pitch, stream);
  if (bn == 32) return launch_split<32, GATED>(p, parts, pitch, stream);
  if (bn == 64) return launch_split<64, GATED>(p, parts, pitch, stream);
  return launch_split<128, GATED>(p, parts, pitch, stream);
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// Rows whose parts the scratch of mlr_linear_split holds: 3 x rows x (K rounded up to 8) bfloat16.  0: it needs none.
MLR_EXPORT int mlr_linear_split_rows(int M, int K) { return M <= 32 || K <= 0 ? 0 : mlr::split_block_rows(M, K); }

// x [M,K], w [N,K], bias [N] or null, out [M,N] (gated: [M, N/2], w in blocks of 64 gate rows and their 64 up rows,
// silu(gate) * up), all float32.  K % 4 == 0, w and scratch on 16-byte boundaries.  error_word: host-visible int that receives a
// code if a wait inside the kernel runs out.
MLR_EXPORT int mlr_linear_split(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int gated,
                                void* scratch, int* error_word, cudaStream_t stream) {
  if (M == 0) return MLR_OK;
  if (M < 0 || N <= 0 || K <= 0 || (scratch == nullptr && M > 32)) return MLR_BAD_SIZE;
  if (K % 4 != 0 || ((uintptr_t)w & 15) || ((uintptr_t)scratch & 15)) return MLR_BAD_ALIGNMENT;
  if (gated && N % LS_ROWS != 0) return MLR_BAD_SIZE;
  const int pitch = (K + 7) / 8 * 8, block = split_block_rows(M, K), width = gated ? N / 2 : N;
  for (int row = 0; row < M; row += block) {
    LinearSplitArgs p{};
    p.M = M - row < block ? M - row : block;
    p.N = N;
    p.K = K;
    p.n_tiles = (N + LS_ROWS - 1) / LS_ROWS;
    p.parts = split_parts(N, K);
    p.x = x + (size_t)row * K;
    p.w = w;
    p.bias = bias;
    p.out = out + (size_t)row * width;
    p.error_word = error_word;
    int status = MLR_OK;
    if (p.M > 32) {
      const long long pieces = (long long)p.M * (pitch / 4), blocks = (pieces + 255) / 256;
      launch_kernel(split_rows_kernel, dim3((unsigned)(blocks < 8 * sm_count() ? blocks : 8 * sm_count())), dim3(256), 0, stream,
                    p.x, (uint2*)scratch, p.M, K, pitch);
      if ((status = launch_status()) != MLR_OK) return status;
    }
    status = gated ? launch_split_width<true>(p, scratch, pitch, stream) : launch_split_width<false>(p, scratch, pitch, stream);
    if (status != MLR_OK) return status;
  }
  return MLR_OK;
}
