// Attention over latents (see attention_latent.cu: absorbed queries, one cached row [latent | turned key part] per token for all heads,
// the latents are the values) for prompt portions, on the 5th-generation tensor cores.
//
// All heads read the same keys, so the rows of the products are (token, head) pairs: 128 / heads tokens with all their heads make
// the 128 rows of an item, 128 neighbouring rows of q seen as [rows * heads, width].  One key tile in shared memory serves
// both products: S = Q K^T over the whole width, O += P V over its first columns.  Six warps as in attention_tcgen05.cu: four of
// softmax (a thread per row), one that issues MMAs, one that loads.
//
// What bounds the layout is room.  A row's output of 512 columns of 32 bits is all of an SM's tensor memory, so latents of more
// than 256 numbers are cut in two halves of value columns, units of their own that both form the scores (1.5 times the work of one
// pass).  Queries of 128 x 576 and one tile of 64 keys would fill the shared memory; with the first 384 columns of the queries in
// tensor memory (A operands may lie there), beside the output's 256 and two buffers of scores, whose places the probabilities
// (also an A operand) take over, four stages of 32 keys fit.  Latents of up to 256 numbers (up to 320 with the turned part): queries
// in shared memory, three stages of 64 keys.
//
// Measured (B200; mma.sync kernel before, this one with MMAs issued behind a test of the lane, by an elected lane): 1,024 rows behind
// 1,024 cached ones, 16 heads of 512 + 64: 509, 188, 112 us; 14 heads of 256 + 32: 350, 52, 47 us; 2,048 rows: 581, 250, 160 and 400, 56,
// 51 us.  A tile of 32 keys then takes 1,600 cycles: 1,100 for the issue of its 36 score MMAs, one per 31 cycles, which is also what
// reading 128 rows of A takes; the softmax of a tile 900.
#include "tcgen05.cuh"

namespace mlr {

constexpr int LA_ROWS = 128;
constexpr int LA_THREADS = 192;
constexpr int LA_VALUES = 256;       // value columns of a unit at most
constexpr uint32_t LA_TMEM_COLS = 512;

// KEYS per tile, STAGES of tiles, Q_TMEM: query columns in tensor memory.
template <int KEYS_, int STAGES_, int Q_TMEM_, int BLOCKS_>
struct LaShape {
  static constexpr int KEYS = KEYS_, STAGES = STAGES_, Q_TMEM = Q_TMEM_;
  static constexpr int BLOCKS = BLOCKS_;                                  // 64-wide column blocks of a key row at most
  static constexpr int Q_BLOCKS = BLOCKS - Q_TMEM / 64;                   // of them of the queries in shared memory
  static constexpr int Q_BLOCK_BYTES = LA_ROWS * 128, K_BLOCK_BYTES = KEYS * 128;
  static constexpr int STAGE_BYTES = BLOCKS * K_BLOCK_BYTES;
  static constexpr int DATA_BYTES = Q_BLOCKS * Q_BLOCK_BYTES + STAGES * STAGE_BYTES;
  // tensor memory: output | scores x 2 | queries.  A row's probabilities take the place of its scores once those are in registers.
  static constexpr uint32_t S_AT = LA_VALUES, Q_AT = S_AT + 2 * KEYS;
  static_assert(Q_AT + Q_TMEM / 2 <= LA_TMEM_COLS, "tensor memory");
};
typedef LaShape<64, 3, 0, 5> LaNarrow;      // rank <= 256, width <= 320
typedef LaShape<32, 4, 384, 9> LaWide;      // rank <= 512, width <= 576

struct LaControl {
  uint64_t q_full, q_stored, k_full[4], s_done[4], pv_done[4], p_ready;
  uint32_t tmem_holder;
  int unit;
};
constexpr int LA_CONTROL_BYTES = 256;
static_assert(sizeof(LaControl) <= LA_CONTROL_BYTES, "control block");

struct LaArgs {
  const bf16* q;
  float* out;
  const int *tile_seg, *tile_row0, *seg_q_start, *seg_q_len, *seg_pos0, *block_table, *seg_slot;
  int table_width, tiles, heads, rank, width, page_size, page_shift, window;
  int tokens;            // of an item
  int values, splits;    // value columns of a unit, units of an item
  float scale_log2;
  const float* sink;
  int *queue, *error_word;
  int shared_bytes;
};

template <typename Shape>
__global__ void __launch_bounds__(LA_THREADS, 1)
latent_prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, const LaArgs a) {
  constexpr int KEYS = Shape::KEYS, STAGES = Shape::STAGES;
  extern __shared__ uint8_t la_shared_raw[];
  uint8_t* q_tile = (uint8_t*)(((uintptr_t)la_shared_raw + 1023) & ~(uintptr_t)1023);      // [blocks][128][64]
  if (q_tile + Shape::DATA_BYTES + LA_CONTROL_BYTES > la_shared_raw + a.shared_bytes) {
    if (threadIdx.x == 0) atomicCAS(a.error_word, 0, 0x7f);
    return;
  }
  uint8_t* ring = q_tile + Shape::Q_BLOCKS * Shape::Q_BLOCK_BYTES;                              // STAGES x [blocks][KEYS][64]
  LaControl& ctl = *reinterpret_cast<LaControl*>(ring + STAGES * Shape::STAGE_BYTES);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&ctl.q_full, 1);
    mbar_init(&ctl.q_stored, 4);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&ctl.k_full[s], 1);
      mbar_init(&ctl.s_done[s], 1);
      mbar_init(&ctl.pv_done[s], 1);
    }
    mbar_init(&ctl.p_ready, 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&q_map) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&k_map) : "memory");
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_holder)), "r"(LA_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fa_fence_before();
  pdl_trigger();
  __syncthreads();
  fa_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl.tmem_holder, 0);
  pdl_wait();

  const int heads = a.heads;
  const int subs = (LA_ROWS + a.tokens - 1) / a.tokens;      // items of a tile of 128 rows of the work list
  const int units = a.tiles * subs * a.splits;
  const int boxes = a.page_size >= KEYS ? 1 : KEYS >> a.page_shift;
  const int box_rows = a.page_size >= KEYS ? KEYS : a.page_size;
  const int k_blocks = (a.width + 63) / 64, k_steps = a.width / 16;
  const int q_blocks = max(0, k_blocks - Shape::Q_TMEM / 64);
  unsigned tiles_before = 0, units_before = 0;
  bool gave_up = false;

  for (;;) {
    if (threadIdx.x == 0) ctl.unit = atomicAdd(&a.queue[0], 1);
    __syncthreads();
    const int unit = ctl.unit;
    if (unit >= units) break;
    const int tile = unit / (subs * a.splits), within = unit - tile * subs * a.splits;
    const int sub = subs - 1 - within / a.splits, split = within % a.splits;      // later rows, which see more, first
    const int seg = a.tile_seg[tile], q_len = a.seg_q_len[seg];
    const int tile_row0 = a.tile_row0[tile], row0 = tile_row0 + sub * a.tokens;
    const int tokens = min(min(a.tokens, LA_ROWS - sub * a.tokens), q_len - row0);
    if (tokens <= 0) {
      __syncthreads();
      continue;
    }
    const int rows = tokens * heads, value0 = split * a.values;
    const int q_row = (a.seg_q_start[seg] + row0) * heads;
    const int first_pos = a.seg_pos0[seg] + row0, last_pos = first_pos + tokens - 1;
    const int* table = a.block_table + (size_t)a.seg_slot[seg] * a.table_width;
    const int lowest = a.window > 0 ? max(0, first_pos - a.window + 1) : 0;
    const int tile_begin = lowest / KEYS, tiles = last_pos / KEYS - tile_begin + 1;

    if (warp == 5) {
      // ------------------------------------------------------------ loads: the stage of tile j - STAGES is free once its P V is done
      if (lane == 0) {
        if (q_blocks > 0) mbar_expect_tx(&ctl.q_full, q_blocks * Shape::Q_BLOCK_BYTES);
        else mbar_arrive(&ctl.q_full);
        for (int b = 0; b < q_blocks; ++b)
          tma_load_2d(&q_map, &ctl.q_full, q_tile + b * Shape::Q_BLOCK_BYTES, Shape::Q_TMEM + b * 64, q_row);
      }
      auto lookup = [&](int j) -> int {                     // lane's page of tile j, or -1
        if (j >= tiles || lane >= boxes) return -1;
        const int logical = ((tile_begin + j) * KEYS + lane * box_rows) >> a.page_shift;
        return logical < a.table_width ? table[logical] : -1;
      };
      int page = lookup(0), next_page = lookup(1);
      for (int j = 0; j < tiles; ++j) {
        const int page_after = lookup(j + 2);               // in flight during this tile's copies
        const unsigned load = tiles_before + (unsigned)j;
        const int stage = load % STAGES;
        const unsigned use = load / STAGES;
        if (use > 0) fa_wait(&ctl.pv_done[stage], (use - 1) & 1u, a.error_word, 0x71, gave_up);
        gave_up = __any_sync(0xffffffffu, gave_up);
        if (!gave_up) {
          if (lane == 0) mbar_expect_tx(&ctl.k_full[stage], (uint32_t)(k_blocks * Shape::K_BLOCK_BYTES));
          __syncwarp();
          for (int base = 0; base < boxes * k_blocks; base += 32) {
            const int copy = base + lane, box = copy % boxes, block = copy / boxes;
            const int where = __shfl_sync(0xffffffffu, page, box);
            if (copy < boxes * k_blocks) {
              const int offset = where < 0 ? 0 : ((tile_begin + j) * KEYS + box * box_rows) & (a.page_size - 1);
              tma_load_2d(&k_map, &ctl.k_full[stage], ring + (size_t)stage * Shape::STAGE_BYTES + block * Shape::K_BLOCK_BYTES + box * box_rows * 128,
                          block * 64, (where < 0 ? 0 : where) * a.page_size + offset);
            }
          }
        }
        page = next_page;
        next_page = page_after;
      }
    } else if (warp == 4) {
      // ------------------------------------------------------------ MMAs
      const uint32_t idesc_s = fa_idesc(LA_ROWS, KEYS, false), idesc_pv = fa_idesc(LA_ROWS, a.values, true);
      const uint64_t q_desc = fa_desc_k_major(smem_u32(q_tile)), k_desc = fa_desc_k_major(smem_u32(ring));
      const uint64_t v_desc = fa_desc_mn_major(smem_u32(ring) + (value0 / 64) * Shape::K_BLOCK_BYTES, Shape::K_BLOCK_BYTES);
      auto issue_scores = [&](int j) {
        const unsigned t = __shfl_sync(0xffffffffu, tiles_before + (unsigned)j, 0);
        const int stage = t % STAGES;
        fa_wait(&ctl.k_full[stage], (t / STAGES) & 1u, a.error_word, 0x72, gave_up);
        gave_up = __any_sync(0xffffffffu, gave_up);
        fa_fence_after();
        if (!gave_up && elect_one()) {
          const uint64_t keys = k_desc + (uint64_t)((stage * Shape::STAGE_BYTES) >> 4);
          const uint32_t d = tmem_base + Shape::S_AT + (t & 1u) * KEYS;
          // unrolled over the most column blocks there can be, so that a product costs its descriptors' additions and no more: one
          // thread that works out addresses takes longer per MMA than the MMA (see the measurements above)
#pragma unroll
          for (int block = 0; block < Shape::BLOCKS; ++block) {
            if (block * 4 >= k_steps) break;
#pragma unroll
            for (int k = 4 * block; k < 4 * block + 4; ++k) {
              if (k >= k_steps) break;
              const uint64_t b = keys + (uint64_t)((block * Shape::K_BLOCK_BYTES + (k & 3) * 32) >> 4);
              if (k < Shape::Q_TMEM / 16)
                fa_mma_tmem(d, tmem_base + Shape::Q_AT + k * 8, b, idesc_s, k > 0 ? 1u : 0u);
              else
                fa_mma(d, q_desc + (uint64_t)(((block - Shape::Q_TMEM / 64) * Shape::Q_BLOCK_BYTES + (k & 3) * 32) >> 4), b, idesc_s, k > 0 ? 1u : 0u);
            }
          }
          fa_commit(&ctl.s_done[stage]);
        }
        __syncwarp();
      };
      fa_wait(&ctl.q_full, units_before & 1u, a.error_word, 0x73, gave_up);
      if (Shape::Q_TMEM > 0) fa_wait(&ctl.q_stored, units_before & 1u, a.error_word, 0x74, gave_up);
      // scores two tiles ahead of the softmax, as in attention_tcgen05.cu
      issue_scores(0);
      if (tiles > 1) issue_scores(1);
      for (int j = 0; j < tiles; ++j) {
        const unsigned t = tiles_before + (unsigned)j;
        const int stage = t % STAGES;
        fa_wait(&ctl.p_ready, t & 1u, a.error_word, 0x75, gave_up);
        gave_up = __any_sync(0xffffffffu, gave_up);
        fa_fence_after();
        if (!gave_up && elect_one()) {
          const uint64_t values = v_desc + (uint64_t)((stage * Shape::STAGE_BYTES) >> 4);
          const uint32_t p = tmem_base + Shape::S_AT + (t & 1u) * KEYS;
#pragma unroll
          for (int k = 0; k < KEYS / 16; ++k)
            fa_mma_tmem(tmem_base, p + k * 8, values + (uint64_t)((k * 2048) >> 4), idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
          fa_commit(&ctl.pv_done[stage]);
        }
        __syncwarp();
        if (j + 2 < tiles) issue_scores(j + 2);
      }
    } else {
      // ------------------------------------------------------------ softmax, one thread per (token, head)
      const int r = threadIdx.x;
      const uint32_t lane_base = tmem_base + ((uint32_t)(warp * 32) << 16);
      if (Shape::Q_TMEM > 0) {
        const uint4* src = reinterpret_cast<const uint4*>(a.q + (size_t)(q_row + r) * a.width);
        for (int c = 0; c < Shape::Q_TMEM / 2; c += 16) {
          uint32_t v[16];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint4 piece = r < rows && 2 * c + 8 * e < a.width ? __ldcg(src + c / 4 + e) : make_uint4(0u, 0u, 0u, 0u);
            v[4 * e] = piece.x, v[4 * e + 1] = piece.y, v[4 * e + 2] = piece.z, v[4 * e + 3] = piece.w;
          }
          fa_tmem_store16(lane_base + Shape::Q_AT + c, v);
        }
        fa_tmem_wait_st();
        fa_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.q_stored);
      }
      const int position = first_pos + r / heads;
      const int limit_hi = r < rows ? position : -1;                // rows past the item see nothing
      const int limit_lo = a.window > 0 ? max(0, position - a.window + 1) : 0;
      // every row of this warp sees all of a tile between these keys
      const bool warp_full = warp * 32 + 31 < rows;
      const int warp_hi = first_pos + warp * 32 / heads;
      const int warp_lo = a.window > 0 ? max(0, first_pos + (warp * 32 + 31) / heads - a.window + 1) : 0;
      float m_run = -INFINITY, m_base = -INFINITY, l = 0.f;
      const float2 scale2 = make_float2(a.scale_log2, a.scale_log2);

      for (int j = 0; j < tiles; ++j) {
        const unsigned t = tiles_before + (unsigned)j;
        const int stage = t % STAGES, key0 = (tile_begin + j) * KEYS;
        fa_wait(&ctl.s_done[stage], (t / STAGES) & 1u, a.error_word, 0x76, gave_up);
        fa_fence_after();
        float s[KEYS];
#pragma unroll
        for (int c = 0; c < KEYS; c += 16) fa_tmem_load16(lane_base + Shape::S_AT + (t & 1u) * KEYS + c, reinterpret_cast<uint32_t*>(s) + c);
        fa_tmem_wait_ld();
        fa_fence_before();
        if (!(warp_full && key0 + KEYS - 1 <= warp_hi && key0 >= warp_lo)) {
#pragma unroll
          for (int c = 0; c < KEYS; ++c)
            if (!(key0 + c >= limit_lo && key0 + c <= limit_hi)) s[c] = -INFINITY;
        }
        float part_max[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
        for (int c = 4; c < KEYS - 4; c += 8) {
#pragma unroll
          for (int e = 0; e < 4; ++e) part_max[e] = fa_max3(part_max[e], s[c + 2 * e], s[c + 2 * e + 1]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) part_max[e] = fmaxf(part_max[e], s[KEYS - 4 + e]);
        const float tile_max = fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3]));
        m_run = fmaxf(m_run, tile_max * a.scale_log2);               // the scale is positive
        // Sums, probabilities and output are relative to the running max.  A base that followed it in steps of more than 2^8 would
        // spare most of the scaling below, but then the heavy weights lie anywhere in a binade, not in its upper part, where
        // bfloat16 rounds them relatively less: error against 64 bits, 240 rows of 16 heads of 512 + 64, 1.15e-3, now 1.06e-3 (mma.sync
        // 1.06e-3).  1,024 rows behind 1,024: 116 -> 121 us for it.
        const bool step = m_run > m_base;
        const float alpha = step ? fa_exp2(m_base - m_run) : 1.f;
        if (step) m_base = m_run;
        const float base = m_base == -INFINITY ? 0.f : m_base;
        const float2 minus_base = make_float2(-base, -base);
        float2 part_sum[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        uint32_t p[KEYS / 2];
#pragma unroll
        for (int c = 0; c < KEYS; c += 8) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 x = __ffma2_rn(make_float2(s[c + 2 * e], s[c + 2 * e + 1]), scale2, minus_base);
            const float2 w = make_float2(fa_exp2(x.x), fa_exp2(x.y));
            part_sum[e] = __fadd2_rn(part_sum[e], w);
            __nv_bfloat162 pair = __floats2bfloat162_rn(w.x, w.y);
            p[c / 2 + e] = *reinterpret_cast<uint32_t*>(&pair);
          }
        }
        const float2 sum2 = __fadd2_rn(__fadd2_rn(part_sum[0], part_sum[1]), __fadd2_rn(part_sum[2], part_sum[3]));
        l = fmaf(l, alpha, sum2.x + sum2.y);

        // the product before must be done: the output may have to be scaled, and no warp may arrive twice at p_ready
        if (j > 0) {
          fa_wait(&ctl.pv_done[(t - 1) % STAGES], ((t - 1) / STAGES) & 1u, a.error_word, 0x77, gave_up);
          fa_fence_after();
        }
        if (j > 0 && __any_sync(0xffffffffu, step)) {
          const float2 alpha2 = make_float2(alpha, alpha);
          for (int c = 0; c < a.values; c += 64) {      // four loads on their way at a time
            float o[64];
#pragma unroll
            for (int e = 0; e < 64; e += 16)
              if (c + e < a.values) fa_tmem_load16(lane_base + c + e, reinterpret_cast<uint32_t*>(o) + e);
            fa_tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 64; e += 16)
              if (c + e < a.values) {
#pragma unroll
                for (int d = e; d < e + 16; d += 2) {
                  const float2 scaled = __fmul2_rn(make_float2(o[d], o[d + 1]), alpha2);
                  o[d] = scaled.x;
                  o[d + 1] = scaled.y;
                }
                fa_tmem_store16(lane_base + c + e, reinterpret_cast<const uint32_t*>(o) + e);
              }
          }
        }
#pragma unroll
        for (int c = 0; c < KEYS / 2; c += 16) fa_tmem_store16(lane_base + Shape::S_AT + (t & 1u) * KEYS + c, p + c);
        fa_tmem_wait_st();
        if (key0 < lowest || key0 + KEYS - 1 > last_pos) {
          // ragged tile, its scores are formed: rows of keys outside the range become zeros for the second product
          uint8_t* rows_at = ring + (size_t)stage * Shape::STAGE_BYTES + (value0 / 64) * Shape::K_BLOCK_BYTES;
          const int blocks = (a.values + 63) / 64;
          for (int idx = threadIdx.x; idx < KEYS * 8 * blocks; idx += 128) {
            const int row = (idx >> 3) % KEYS;
            if (key0 + row < lowest || key0 + row > last_pos) *reinterpret_cast<uint4*>(rows_at + (size_t)idx * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        fa_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.p_ready);
      }
      // the finished rows, after the last tile's product
      const unsigned t = tiles_before + (unsigned)tiles - 1;
      fa_wait(&ctl.pv_done[t % STAGES], (t / STAGES) & 1u, a.error_word, 0x78, gave_up);
      fa_fence_after();
      float factor = 1.f / l;
      if (a.sink != nullptr) {
        const float sink = a.sink[r % heads] * 1.4426950408889634f, high = fmaxf(m_base, sink), share = fa_exp2(m_base - high);
        factor = share / fmaf(l, share, fa_exp2(sink - high));
      }
      float* dst = a.out + (size_t)(q_row + r) * a.rank + value0;
      for (int c = 0; c < a.values; c += 16) {
        float o[16];
        fa_tmem_load16(lane_base + c, reinterpret_cast<uint32_t*>(o));
        fa_tmem_wait_ld();
        if (r < rows) {
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            *reinterpret_cast<float4*>(dst + c + e) = make_float4(o[e] * factor, o[e + 1] * factor, o[e + 2] * factor, o[e + 3] * factor);
        }
      }
      fa_fence_before();
    }
    tiles_before += (unsigned)tiles;
    units_before += 1;
    __syncthreads();                // queries and ctl.unit are rewritten by the next unit
    fa_fence_after();
  }

  fa_fence_before();
  __syncthreads();
  if (warp == 4) {
    fa_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(LA_TMEM_COLS) : "memory");
  }
  // the CTA that leaves last puts the queue back for the next launch
  if (threadIdx.x == 0) {
    const int left = atomicAdd(&a.queue[1], 1);
    if (left == (int)gridDim.x - 1) { a.queue[0] = 0; a.queue[1] = 0; }
  }
}

template <typename Shape>
static int la_launch(LaArgs a, int q_rows, long long pool_rows, const void* pool, cudaStream_t stream) {
  CUtensorMap q_map, k_map;
  const int box_rows = a.page_size >= Shape::KEYS ? Shape::KEYS : a.page_size;
  if (!cached_tile_map(&q_map, a.q, (long long)q_rows * a.heads, a.width, LA_ROWS) ||
      !cached_tile_map(&k_map, pool, pool_rows, a.width, box_rows))
    return MLR_BAD_SIZE;
  a.shared_bytes = 1024 + Shape::DATA_BYTES + LA_CONTROL_BYTES;
  static bool configured = false;
  if (!configured) {
    cudaError_t err = cudaFuncSetAttribute(latent_prefill_tcgen05_kernel<Shape>, cudaFuncAttributeMaxDynamicSharedMemorySize, a.shared_bytes);
    if (err != cudaSuccess) return (int)err;
    configured = true;
  }
  const int subs = (LA_ROWS + a.tokens - 1) / a.tokens;
  const long long units = (long long)a.tiles * subs * a.splits;
  if (units >= (1ll << 30)) return MLR_TOO_LARGE;
  launch_kernel(latent_prefill_tcgen05_kernel<Shape>, dim3((unsigned)(units < sm_count() ? units : sm_count())), dim3(LA_THREADS),
                (size_t)a.shared_bytes, stream, q_map, k_map, a);
  return launch_status();
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// Whether the kernel takes these sizes: rows of whole 16-column steps; up to 256 numbers in the latent (320 with the turned part), or
// up to 512 (576) in two halves of whole 64-column blocks.
MLR_EXPORT int mlr_latent_attention_tcgen05_fits(int heads, int rank, int rot) {
  const int width = rank + rot;
  if (heads < 1 || heads > LA_ROWS || rank < 16 || rot < 0 || rank % 16 != 0 || width % 16 != 0 || width < 64) return 0;
  if (rank <= 256 && width <= 320) return 1;
  return rank > 256 && rank <= 512 && rank % 128 == 0 && width <= 576 ? 1 : 0;
}

// Prompt portions.  q: bfloat16 [q_rows, heads, rank + rot]; pool: bfloat16 [pool_pages, 1, page_size, rank + rot], page_size a power of
// two >= 8; out: float32 [q_rows, heads, rank]; tile_seg / tile_row0: tiles of up to 128 rows of one segment, best heaviest
// first; scale > 0; sink: float32 [heads] or null; queue: two zeroed ints in device memory (left zeroed); error_word: host-visible int.
MLR_EXPORT int mlr_latent_attention_prefill_tcgen05(
    const void* q, const void* pool, float* out, const int* tile_seg, const int* tile_row0, const int* seg_q_start, const int* seg_q_len,
    const int* seg_pos0, const int* block_table, const int* seg_slot, int table_width, int tiles, int q_rows, int heads, int rank, int rot,
    int page_size, int pool_pages, int window, float scale, const float* sink, int* queue, int* error_word, cudaStream_t stream) {
  if (tiles == 0) return MLR_OK;
  if (tiles < 0 || q_rows <= 0 || table_width <= 0 || pool_pages <= 0 || page_size < 8 || (page_size & (page_size - 1)) != 0 || window < 0 ||
      queue == nullptr || error_word == nullptr || !(scale > 0.f))
    return MLR_BAD_SIZE;
  if (!mlr_latent_attention_tcgen05_fits(heads, rank, rot)) return MLR_TOO_LARGE;
  const long long pool_rows = (long long)pool_pages * page_size;
  if (pool_rows >= (1ll << 31) || (long long)q_rows * heads >= (1ll << 31)) return MLR_TOO_LARGE;
  if (((uintptr_t)q & 15) || ((uintptr_t)pool & 15) || ((uintptr_t)out & 15)) return MLR_BAD_ALIGNMENT;
  LaArgs a;
  a.q = (const bf16*)q; a.out = out; a.tile_seg = tile_seg; a.tile_row0 = tile_row0; a.seg_q_start = seg_q_start;
  a.seg_q_len = seg_q_len; a.seg_pos0 = seg_pos0; a.block_table = block_table; a.seg_slot = seg_slot; a.table_width = table_width;
  a.tiles = tiles; a.heads = heads; a.rank = rank; a.width = rank + rot; a.page_size = page_size;
  a.page_shift = 0;
  while ((1 << a.page_shift) < page_size) ++a.page_shift;
  a.window = window; a.tokens = LA_ROWS / heads;
  a.splits = rank > 256 ? 2 : 1;
  a.values = rank / a.splits;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.sink = sink; a.queue = queue; a.error_word = error_word;
  return rank > 256 ? la_launch<LaWide>(a, q_rows, pool_rows, pool, stream) : la_launch<LaNarrow>(a, q_rows, pool_rows, pool, stream);
}
