// The products of routed experts on the 5th-generation tensor cores: rows that are sorted by expert, each expert's with its own matrix.
//
// An expert of a step has as many rows as chose it, rarely a multiple of 128.  So its weights are the MMA's 128 rows and its tokens the
// columns, of which an MMA takes any multiple of 16: no work for padding (tiles of 128 tokens x 256 weight rows were three quarters full
// with 192 rows per expert).  A tile is 256 weight rows, as two accumulators of 128 rows, and up to 128 tokens; a gated product's two
// accumulators are the gate rows and the up rows of the same 128 outputs, so that both lie in one thread.  One CTA per SM walks the
// tiles, with two pairs of accumulators: one tile is written out under the next one's MMAs, and loads never stop.
//
// Bound by the memory's rate for weights with few tokens per expert (a step of 40 rows reads 1.07 GB in 178 us, sorting, gathering and summing
// included), by the round trips of four stages beside MMAs with many.  Measured (B200), whole feed-forward, tokens as the MMA's rows / so: 64 experts of
// 2,048 -> 1,408, six per row, 2,048 rows 424 / 368 us (371 / 319 in a captured sequence, as the following), 1,000 rows 250 / 234, 300 rows 211 / 196, 40 rows 199 / 178; 16 experts of 896 -> 2,432, two per
// row, 700 rows 69 / 66, 100 rows 63 / 55.  From a flushed L2, 16 experts, 2,000 rows 111 / 94, 2,048 rows, whose down product has 160 tiles, 111 / 115 and, with tiles half
// as high, 109; 300 rows of three experts 51 / 49 / 45.  Tiles of 256 tokens with one accumulator pair and three stages: 382 us at 2,048 rows (a
// stage's round trip and its MMAs one behind the other); four warps that write instead of eight: 323, and 122 us for the 16 experts.
//
// Warp 0 loads (weights in boxes of 64 rows, tokens in boxes of 32, four stages of 48 KB), warp 1 issues MMAs, warps 2 to 9 write out.
#include "tcgen05.cuh"

namespace mlr {

constexpr int EP_TOKENS = 128;       // of a tile at most
constexpr int EP_WEIGHTS = 256;      // rows of a tile
constexpr int EP_K = 64;
constexpr int EP_STAGES = 4;
constexpr int EP_THREADS = 320;
constexpr int EP_W_BOX = 64, EP_X_BOX = 32;
constexpr int EP_W_BYTES = EP_WEIGHTS * EP_K * 2, EP_STAGE_BYTES = EP_W_BYTES + EP_TOKENS * EP_K * 2;
constexpr int EP_PITCH = 128 + 8, EP_STAGED = 32;      // outputs of a gated tile are staged 32 tokens at a time, twice
constexpr int EP_SHARED = 1024 + EP_STAGES * EP_STAGE_BYTES + 2 * EP_STAGED * EP_PITCH * 2;
constexpr uint32_t EP_TMEM_COLS = 512;

struct ExpertArgs {
  void* out;
  const int* tiles;            // [max_tiles][3]: expert (negative: unused), first row, end row; then how many are used
  const float* row_scale;      // factor of every row's product, before the gate, or null
  int N, K;                    // rows of an expert's matrix, columns
  int entries;                 // of the list
  int act;
  int* error_word;
};

// Tiles are numbered weights first; CTA b takes tiles b, b + grid, ..
template <bool GATED>
__global__ void __launch_bounds__(EP_THREADS, 1)
expert_product_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, const ExpertArgs p) {
  extern __shared__ uint8_t ep_shared_raw[];
  uint8_t* ring = (uint8_t*)(((uintptr_t)ep_shared_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full_bar[EP_STAGES], empty_bar[EP_STAGES], done_bar[2], read_bar[2];      // the latter per accumulator
  __shared__ uint32_t tmem_holder;
  __shared__ __align__(16) float scales[2][EP_TOKENS];      // factors of a tile's tokens, once per group of warps that write
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < EP_STAGES; ++s) mbar_init(&full_bar[s], 1), mbar_init(&empty_bar[s], 1);
    for (int b = 0; b < 2; ++b) mbar_init(&done_bar[b], 1), mbar_init(&read_bar[b], 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&w_map) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&x_map) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)), "r"(EP_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fa_fence_before();
  pdl_trigger();
  __syncthreads();
  fa_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_holder, 0);
  pdl_wait();                                // the list comes from an earlier kernel
  const int k_blocks = (p.K + EP_K - 1) / EP_K;
  int high = EP_WEIGHTS;      // weight rows of a tile
  if (!GATED) {
    // Half as high, with one accumulator, where that saves so many rounds of CTAs that it pays for the smaller tiles, which take some 0.7 of the time.
    const int used = __ldcg(p.tiles + 3 * p.entries), grid = (int)gridDim.x;
    auto rounds = [&](int rows) { return ((p.N + rows - 1) / rows * used + grid - 1) / grid; };
    if (rounds(EP_WEIGHTS / 2) * 7 < rounds(EP_WEIGHTS) * 10) high = EP_WEIGHTS / 2;
  }
  const int across = (p.N + high - 1) / high;
  const int tiles = across * p.entries;
  bool gave_up = false;
  struct Tile { int expert, row0, tokens, column; };
  auto tile_at = [&](int tile) {      // tokens: 0 for an unused entry
    const int entry = tile / across;
    Tile t;
    t.column = tile - entry * across;
    t.expert = __ldcg(p.tiles + 3 * entry);
    t.row0 = __ldcg(p.tiles + 3 * entry + 1);
    t.tokens = t.expert < 0 ? 0 : min(__ldcg(p.tiles + 3 * entry + 2) - t.row0, EP_TOKENS);
    return t;
  };

  if (warp == 0) {
    // lanes 0 .. 3: 64 weight rows each (of a gated product: gate, gate, up, up), from lane 4 on 32 tokens each
    const int block = lane & 3;
    uint8_t* own = ring + (lane < 4 ? block * EP_W_BOX * 128 : EP_W_BYTES + (lane - 4) * EP_X_BOX * 128);
    int s = 0;
    uint32_t phase = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const Tile t = tile_at(tile);
      if (t.tokens <= 0) continue;
      const int x_boxes = (t.tokens + EP_X_BOX - 1) / EP_X_BOX;
      const int w_row = t.expert * p.N + t.column * high + (GATED ? (block & 1) * 128 + (block >> 1) * 64 : block * 64);
      const int x_row = t.row0 + (lane - 4) * EP_X_BOX;
      const uint32_t bytes = (uint32_t)(high * EP_K * 2 + x_boxes * EP_X_BOX * 128);
      for (int i = 0; i < k_blocks; ++i) {
        fa_wait(&empty_bar[s], phase ^ 1u, p.error_word, 0xb1, gave_up);
        gave_up = __any_sync(0xffffffffu, gave_up);
        if (!gave_up) {
          if (lane == 0) mbar_expect_tx(&full_bar[s], bytes);
          __syncwarp();
          if (lane < high / EP_W_BOX) tma_load_2d(&w_map, &full_bar[s], own + s * EP_STAGE_BYTES, i * EP_K, w_row);
          else if (lane >= 4 && lane - 4 < x_boxes) tma_load_2d(&x_map, &full_bar[s], own + s * EP_STAGE_BYTES, i * EP_K, x_row);
        }
        if (++s == EP_STAGES) s = 0, phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    const uint64_t w_desc = fa_desc_k_major(smem_u32(ring)), x_desc = fa_desc_k_major(smem_u32(ring) + EP_W_BYTES);
    int s = 0;
    uint32_t phase = 0, turn = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const Tile t = tile_at(tile);
      if (t.tokens <= 0) continue;
      const uint32_t idesc = fa_idesc(128, (t.tokens + 15) & ~15, false);
      if (turn > 1) fa_wait(&read_bar[turn & 1u], ((turn >> 1) - 1) & 1u, p.error_word, 0xb4, gave_up);      // the sums of the tile two before are in registers
      for (int i = 0; i < k_blocks; ++i) {
        fa_wait(&full_bar[s], phase, p.error_word, 0xb2, gave_up);
        gave_up = __any_sync(0xffffffffu, gave_up);
        fa_fence_after();
        if (elect_one() && !gave_up) {
          const uint64_t w = w_desc + (uint64_t)(s * (EP_STAGE_BYTES >> 4)), x = x_desc + (uint64_t)(s * (EP_STAGE_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < EP_K / 16; ++k)
#pragma unroll
            for (int half = 0; half < 2; ++half)
              if (half * 128 < high) fa_mma(tmem_base + (turn & 1u) * 2 * EP_TOKENS + half * EP_TOKENS, w + half * (128 * 128 >> 4) + 2 * k, x + 2 * k, idesc, i > 0 || k > 0 ? 1u : 0u);
          fa_commit(&empty_bar[s]);
          if (i == k_blocks - 1) fa_commit(&done_bar[turn & 1u]);
        }
        __syncwarp();
        if (++s == EP_STAGES) s = 0, phase ^= 1u;
      }
      ++turn;
    }
  } else {
    // two groups of four warps: of a gated tile the first and the last 64 tokens, else an accumulator each
    const int quarter = warp & 3, own = quarter * 32 + lane, side = (warp - 2) >> 2;      // own: the accumulators' row
    bf16* staged = reinterpret_cast<bf16*>(ring + EP_STAGES * EP_STAGE_BYTES) + side * EP_STAGED * EP_PITCH;
    uint32_t turn = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const Tile t = tile_at(tile);
      if (t.tokens <= 0) continue;
      if (p.row_scale != nullptr) {      // under the products; read one by one behind them they cost 55 of 156 us (2,048 rows, 16 experts of 896 -> 2,432)
        const float scale = own < t.tokens ? __ldcg(p.row_scale + t.row0 + own) : 0.f;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + side) : "memory");      // those of the tile before have been read
        scales[side][own] = scale;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + side) : "memory");
      }
      fa_wait(&done_bar[turn & 1u], (turn >> 1) & 1u, p.error_word, 0xb3, gave_up);
      const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + (turn & 1u) * 2 * EP_TOKENS;
      uint64_t* read = &read_bar[turn & 1u];
      ++turn;
      fa_fence_after();
      if (GATED) {
        // outputs in bfloat16, through shared memory, written in rows of 256 bytes
        const int inner = p.N / 2, n0 = t.column * 128 + (own & 15) * 8, end = min(t.tokens, (side + 1) * EP_TOKENS / 2);
        bf16* out = reinterpret_cast<bf16*>(p.out) + (size_t)t.row0 * inner + n0;
        for (int c0 = side * EP_TOKENS / 2; c0 < end; c0 += EP_STAGED) {
#pragma unroll
          for (int c = c0; c < c0 + EP_STAGED; c += 16) {
            if (c >= end) break;
            uint32_t g[16], u[16];
            fa_tmem_load16(lane_base + c, g);
            fa_tmem_load16(lane_base + EP_TOKENS + c, u);
            fa_tmem_wait_ld();
            if (p.row_scale != nullptr) {
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                g[e] = __float_as_uint(__uint_as_float(g[e]) * scales[side][c + e]);
                u[e] = __float_as_uint(__uint_as_float(u[e]) * scales[side][c + e]);
              }
            }
#pragma unroll
            for (int e = 0; e < 16; ++e)
              staged[(c - c0 + e) * EP_PITCH + own] = __float2bfloat16_rn(gate_times(p.act, __uint_as_float(g[e]), __uint_as_float(u[e])));
          }
          asm volatile("bar.sync %0, 128;" ::"r"(1 + side) : "memory");
          if (!gave_up && n0 + 8 <= inner)      // inner is a multiple of 64
            for (int r = own >> 4; r < EP_STAGED && c0 + r < end; r += 8)
              *reinterpret_cast<uint4*>(out + (size_t)(c0 + r) * inner) = *reinterpret_cast<const uint4*>(staged + r * EP_PITCH + (own & 15) * 8);
          asm volatile("bar.sync %0, 128;" ::"r"(1 + side) : "memory");      // staged again
        }
      } else {
        const bool both = high == EP_WEIGHTS;      // accumulators; else a group of warps takes the first or the last 64 tokens of the one
        const int n = t.column * high + (both ? side * 128 : 0) + own, from = both ? 0 : side * (EP_TOKENS / 2);
        const int end = both ? t.tokens : min(t.tokens, from + EP_TOKENS / 2);
        const uint32_t sums = lane_base + (both ? side * EP_TOKENS : 0);
        float* column = reinterpret_cast<float*>(p.out) + (size_t)t.row0 * p.N + n;
        for (int c = from; c < end; c += 32) {
          uint32_t v[32];
          fa_tmem_load16(sums + c, v);
          fa_tmem_load16(sums + c + 16, v + 16);
          fa_tmem_wait_ld();
          if (gave_up || n >= p.N) continue;
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (c + e < t.tokens) {
              float value = __uint_as_float(v[e]);
              if (p.row_scale != nullptr) value *= scales[side][c + e];
              column[(size_t)(c + e) * p.N] = value;
            }
        }
      }
      fa_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(read);
    }
  }
  fa_fence_before();
  __syncthreads();
  if (warp == 1) {
    fa_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(EP_TMEM_COLS) : "memory");
  }
}

template <bool GATED>
static int launch_experts(const void* x, const void* w, const ExpertArgs& a, int rows, int groups, cudaStream_t stream) {
  CUtensorMap w_map, x_map;
  if (!cached_tile_map(&w_map, w, (long long)groups * a.N, a.K, EP_W_BOX) || !cached_tile_map(&x_map, x, rows, a.K, EP_X_BOX)) return MLR_BAD_ALIGNMENT;
  static OncePerDevice once;
  const cudaError_t err = once([] { return cudaFuncSetAttribute(expert_product_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, EP_SHARED); });
  if (err != cudaSuccess) return (int)err;
  const int least = GATED ? EP_WEIGHTS : EP_WEIGHTS / 2;      // rows of a tile
  const long long tiles = (long long)((a.N + least - 1) / least) * a.entries;
  if (tiles > 0x3fffffff) return MLR_TOO_LARGE;
  launch_kernel(expert_product_kernel<GATED>, dim3((unsigned)(tiles < sm_count() ? tiles : sm_count())), dim3(EP_THREADS), (size_t)EP_SHARED, stream, w_map, x_map, a);
  return launch_status();
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// x: bfloat16 [rows, K], sorted by expert; w: bfloat16 [groups, N, K]; tiles: device memory, int32 [max_tiles][3] = (expert, first row, end row)
// per tile of up to 128 rows of one expert, expert < 0 for unused entries, and their number behind them; it may be written by the kernel just before this one.
// gated: w holds blocks of 64 gate rows followed by the 64 up rows of the same outputs, out is act(gate) * up, bfloat16 [rows, N / 2] (act 0:
// silu, 1: the tanh form of gelu); else out is float32 [rows, N].  row_scale: float32 [rows] or null, multiplies each row's product, before the gate.
MLR_EXPORT int mlr_expert_product(const void* x, const void* w, void* out, const int* tiles, int max_tiles, int rows, int groups, int N, int K,
                                  int gated, int act, const float* row_scale, int* error_word, cudaStream_t stream) {
  if (rows == 0 || max_tiles == 0) return MLR_OK;
  if (rows < 0 || max_tiles < 0 || groups <= 0 || N <= 0 || K <= 0 || tiles == nullptr || error_word == nullptr || (gated && N % 128 != 0)) return MLR_BAD_SIZE;
  if (K % 8 != 0 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)out & 15)) return MLR_BAD_ALIGNMENT;
  if ((long long)groups * N > 0x7fffffffll) return MLR_TOO_LARGE;
  const ExpertArgs a{out, tiles, row_scale, N, K, max_tiles, act, error_word};
  return gated ? launch_experts<true>(x, w, a, rows, groups, stream) : launch_experts<false>(x, w, a, rows, groups, stream);
}
