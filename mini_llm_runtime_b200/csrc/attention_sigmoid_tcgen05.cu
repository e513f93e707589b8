// The sigmoid attention of attention_sigmoid_mma.cu (same formula, same roundings: weights and their mixing across heads in float32, mixed
// weights bfloat16) on the 5th-generation tensor cores.
//
// All heads' weights of a (row, key) pair are mixed, so they should meet where they are formed.  Both large products are formed transposed:
//   S^T = K Q^T     per key head: 128 keys (lanes of tensor memory) x (query heads of the key head, 16 rows)
//   O^T = V^T W'^T  128 value columns (lanes) x (query heads, 16 rows), kept in tensor memory over all key tiles
// and the columns of S^T stand in an order (SG_SLOTS below) in which a tensor-memory load leaves in each thread of four the heads that mma.sync
// wants there as its second operand: W'^T = talk W^T is a third product (16 heads x 16 heads x 8 keys) without a weight leaving its
// thread.  Its operands are split exactly into three bfloat16 parts each, six of the nine products (the others are below 2^-26 of the
// magnitudes' sum; parts cut off instead of rounded would leave 2^-22 of one sign), float32 sums.  Equal heads whose factors cancel to 2^-17, errors by
// multiply-adds / with cut / with rounded parts: 3.3e-2 / 2.2e-2 / 0.5e-2 (16 heads of 128), 2.6e-2 / 2.1e-2 / 0.5e-2 (12 of 64).  By multiply-adds (a thread owning one key and eight rows with all heads) every factor of the mixing came from shared
// memory, four wavefronts per 16 bytes, whose bandwidth the MMAs' operands and the copies want.  A thread ends with eight rows of a
// (key, head), the 16 bytes that the second product reads together.  Value heads of 64 lie two to the 128 lanes; what a head's rows make of its
// neighbour's values is never read.
//
// Twelve warps: eight compute (two per scheduler, rows 0-7 and 8-15 of the same keys), two issue MMAs and two load, one each per product.
// Keys and values come in stages of 16 KB: 128 keys x 64 columns of one key head, or 64 keys x 128 value columns.  Scores and output
// fill the tensor memory (2 x 256 columns); the queries of 16 heads of 128, the mixed weights and five stages the shared memory, which
// sets 16 rows per CTA.
//
// The key tiles of all entries, one behind the other, are cut into as many equal runs as there are CTAs; an entry in several
// runs leaves its sums in float32, which a second kernel adds up in order.  (Whole entries would not balance: the last rows of a
// prompt see all of it.)
//
// A run's products with the values meet in one accumulator, which is cut at every 16 keys, where the kernel before added sums of up to 384 keys in float32.  Errors
// against 64 bits, that kernel / this one, 16 heads of 128: 2,048 rows 2.3552e-3 / 2.3556e-3, 4,000 rows 2.3645e-3 / 2.3645e-3, 4,000 rows behind 2,000
// 2.3483e-3 / 2.3483e-3, 2,048 rows behind 30,000 2.3059e-3 / 2.3061e-3; 14 of 64: 2.2882e-3 / 2.2881e-3, 2.2787e-3 / 2.2787e-3, 2.2724e-3 / 2.2721e-3, 2.4068e-3 /
// 2.4078e-3.  Only sums that cancel to 2^-9 and less tell them apart (by up to six times at 3,000 keys of a run).  Adding to float32 sums in device memory after every
// three tiles took 20 us each time (4,000 rows 249 -> 408 us), after every eight 249 -> 304.
//
// Bound by the computing warps: a tile of 128 keys takes 11,000 cycles, of which the special-function units (an exponential and a reciprocal
// per weight) need 4,100 and the mixing's products 2,000, two warps per scheduler hardly overlapping; then by what every piece costs whatever
// its keys (5,000 to 12,000 cycles until its first scores, of which 3 or 4 stages' copies at a time, 4,000 for its sums).  Measured (B200), mma.sync kernel / this one, with
// the adding: portions of 1,450, 401 and 197 rows, 16 heads of 128 166 / 68 us, 14 of 64 102 / 56; 2,048 rows 243 / 89 and 170 / 76; 4,000 rows
// 844 / 238 and 516 / 206; eight decoded rows at 2,000 keys 29 / 29 and 33 / 24, 32 at 3,000 140 / 62 and 81 / 45.
#include "part_products.cuh"
#include "tcgen05.cuh"

namespace mlr {

constexpr int SG_KEYS = 128;         // of a tile
constexpr int SG_KEY_BOX = 16;       // keys of a copy at most
constexpr int SG_ROWS = 16;          // of an entry
constexpr int SG_HEADS = 16;         // at most
constexpr int SG_COMPUTE = 256;      // computing threads
constexpr int SG_THREADS = SG_COMPUTE + 128;
// The launch's registers are shared out anew between the computing warps and the others.
constexpr int SG_LAUNCH_REGISTERS = 168, SG_COMPUTE_REGISTERS = 208, SG_OTHER_REGISTERS = 88;
static_assert(SG_COMPUTE * SG_COMPUTE_REGISTERS + 128 * SG_OTHER_REGISTERS <= SG_THREADS * SG_LAUNCH_REGISTERS, "registers");
constexpr int SG_STAGE = 16384;      // bytes
constexpr int SG_BIAS = 136;         // distances between eight rows and a tile's keys (135), per head: four heads' fall into different banks
constexpr int SG_P_STRIDE = SG_KEYS * 16 + 16;      // bytes of eight rows' mixed weights of a head; the odd 16 spread the stores over the banks
// A key head's query heads are filled up to whole fours; four (key head, 4 query heads) make the 16 slots.  Column of S^T (and row of the queries
// in shared memory) of slot 4 u + x and row q: 64 u + 8 (q / 2) + 2 x + q % 2.
constexpr int SG_SLOTS = 16;
constexpr uint32_t SG_TMEM_COLS = 512, SG_O_AT = 256;

template <int D>
struct SgShape {
  static constexpr int HALVES = D / 64;
  static constexpr int K_STAGES = 3, V_STAGES = D == 64 ? 4 : 2, STAGES = K_STAGES + V_STAGES;
};

// A place in a ring of N stages, and the parity of its turn.
template <int N>
struct SgStage {
  int stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++stage == N) stage = 0, phase ^= 1u;
  }
};

struct SgControl {
  uint64_t k_full[4], k_empty[4], v_full[4], v_empty[4], q_ready, s_full, s_free, p_ready[2], pv_done[2];
  uint32_t tmem_holder;
  int begin, end, entry, entry_at;      // the run's places; the entry that holds its first and the places before that entry
};
constexpr int SG_CONTROL_BYTES = 256;
static_assert(sizeof(SgControl) <= SG_CONTROL_BYTES, "control block");

struct SgArgs {
  const bf16* q;
  bf16* out;
  float* partial;       // [2 * CTAs][slot_rows][heads][V]: a run's first entry where it began before, its last where it goes on behind
  int* before;          // [tiles + 1]: places before an entry
  const int *tile_seg, *tile_row0, *seg_q_start, *seg_q_len, *seg_pos0, *block_table, *seg_slot;
  const float *r1, *r2, *pb, *talk;
  int table_width, tiles, heads, kv_heads, page_size, page_shift, pool_rows, slot_rows;
  bool whole;           // a CTA per entry
  float scale;
  int* error_word;
};

template <int D>
static size_t sg_shared(int heads) {
  return 1024 + SG_SLOTS * SG_ROWS * D * 2 + (size_t)SgShape<D>::STAGES * SG_STAGE + (size_t)heads * 2 * SG_P_STRIDE + 2 * SG_SLOTS * SG_BIAS * 4 +
         SG_CONTROL_BYTES;
}

// MN-major operand without swizzle: 8 MN-contiguous elements of one k are 16 bytes, 8 consecutive k follow one another (128 bytes), the
// next 8 k lie 128 bytes on, the next 8 elements along MN `mn_stride` bytes.
__device__ __forceinline__ uint64_t sg_desc_mn_plain(uint32_t address, uint32_t mn_stride) {
  uint64_t desc = 0;
  desc |= (uint64_t)((address & 0x3FFFFu) >> 4);
  desc |= (uint64_t)(128 >> 4) << 16;
  desc |= (uint64_t)(mn_stride >> 4) << 32;
  desc |= (uint64_t)1 << 46;
  return desc;
}
// Rows l / 4 and l / 4 + 8 of 16 lanes, columns 2 (l % 4) and the next, of four blocks of 8 columns: four numbers per block in that order.
__device__ __forceinline__ void sg_tmem_load_scores(uint32_t taddr, float* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
                 "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
               : "r"(taddr) : "memory");
}
// Two numbers as three parts each.
__device__ __forceinline__ void sg_parts(float2 x, uint32_t (&part)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) part[i] = take_part(x.x, x.y);
}
__device__ __forceinline__ void sg_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {      // may be moved among other products
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void sg_tmem_load8(uint32_t taddr, float* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ float sg_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sg_log2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// for the 128 computing threads of rows 0-7 or 8-15
__device__ __forceinline__ void sg_half_barrier(int half) { asm volatile("bar.sync %0, %1;" ::"r"(1 + half), "n"(SG_COMPUTE / 2) : "memory"); }

// Entries take a place per key tile and SG_ENTRY before them, for what a CTA spends on an entry whatever its keys (queries, sums out); the run of
// CTA b begins at place sg_run(b): equal shares, and as many runs as there are places where those are fewer than CTAs.
constexpr int SG_ENTRY = 1;
__device__ __forceinline__ int sg_run(int b, int total, int ctas) { return (int)((long long)b * total / ctas); }

// places of entry e
__device__ __forceinline__ int sg_places(const SgArgs& a, int e) {
  const int seg = a.tile_seg[e], row0 = a.tile_row0[e];
  return (a.seg_pos0[seg] + min(row0 + SG_ROWS, a.seg_q_len[seg]) - 1) / SG_KEYS + 1 + SG_ENTRY;
}

// An entry's part of a CTA's run.
struct SgPiece {
  int seg, row0, rows, first_pos, last_pos;
  int entry_tiles, tile_begin, tiles;      // key tiles of the entry; of them here
  size_t q_row;
};
// The pieces of a CTA's run in order.
struct SgWalk {
  int entry, at, begin, end;
  __device__ __forceinline__ SgWalk(const SgControl& ctl)
      : entry(ctl.entry), at(ctl.begin < ctl.end ? ctl.entry_at : ctl.end), begin(ctl.begin), end(ctl.end) {}
  __device__ __forceinline__ bool next(const SgArgs& a, SgPiece& p) {
    while (at < end) {
      p.seg = a.tile_seg[entry], p.row0 = a.tile_row0[entry];
      p.rows = min(SG_ROWS, a.seg_q_len[p.seg] - p.row0);
      p.first_pos = a.seg_pos0[p.seg] + p.row0, p.last_pos = p.first_pos + p.rows - 1;
      p.entry_tiles = p.last_pos / SG_KEYS + 1;
      p.q_row = (size_t)(a.seg_q_start[p.seg] + p.row0);
      const int first = at + SG_ENTRY;
      at = first + p.entry_tiles;
      entry += 1;
      p.tile_begin = max(begin - first, 0), p.tiles = min(end - first, p.entry_tiles) - p.tile_begin;
      if (end == 0x7fffffff) at = end;      // the run is this entry
      if (p.tiles > 0) return true;
    }
    return false;
  }
};

template <int D, int V>
__global__ void __launch_bounds__(SG_THREADS, 1)
attention_sigmoid_tcgen05_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, const SgArgs a) {
  constexpr int HALVES = SgShape<D>::HALVES, K_STAGES = SgShape<D>::K_STAGES, V_STAGES = SgShape<D>::V_STAGES;
  extern __shared__ uint8_t sg_shared_raw[];
  const int H = a.heads, G = a.kv_heads, per_kv = H / G, fours = (per_kv + 3) / 4;
  uint8_t* q_tile = (uint8_t*)(((uintptr_t)sg_shared_raw + 1023) & ~(uintptr_t)1023);      // [HALVES][256][64], swizzled by 128 bytes
  uint8_t* k_ring = q_tile + SG_SLOTS * SG_ROWS * D * 2;
  uint8_t* v_ring = k_ring + K_STAGES * SG_STAGE;
  float* bias = reinterpret_cast<float*>(v_ring + V_STAGES * SG_STAGE);                     // [2][SG_SLOTS][SG_BIAS]
  SgControl& ctl = *reinterpret_cast<SgControl*>(bias + 2 * SG_SLOTS * SG_BIAS);
  uint8_t* p_tile = reinterpret_cast<uint8_t*>(&ctl) + SG_CONTROL_BYTES;                    // per group of heads [2][heads][128 keys][8 rows]
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < K_STAGES; ++s) mbar_init(&ctl.k_full[s], 1), mbar_init(&ctl.k_empty[s], 1);
    for (int s = 0; s < V_STAGES; ++s) mbar_init(&ctl.v_full[s], 1), mbar_init(&ctl.v_empty[s], 1);
    mbar_init(&ctl.q_ready, 8);
    mbar_init(&ctl.s_full, 1);
    mbar_init(&ctl.s_free, 8);
    for (int b = 0; b < 2; ++b) mbar_init(&ctl.p_ready[b], 8), mbar_init(&ctl.pv_done[b], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&k_map) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&v_map) : "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_holder)), "r"(SG_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_trigger();
  const int half = (threadIdx.x >> 7) & 1, r0 = half * 8, x = lane & 3, quad = lane >> 2;      // of the computing threads
  auto head_of = [&](int slot) {      // -1: none
    const int c = (slot >> 2) / fours, within = slot - c * fours * 4;
    return c < G && within < per_kv ? c * per_kv + within : -1;
  };
  float* half_bias = bias + half * SG_SLOTS * SG_BIAS;
  pdl_wait();
  // the slot whose biases a thread fills in
  const int bias_slot = (threadIdx.x & 127) >> 3, bias_head = max(head_of(bias_slot), 0);
  const float decay = a.r1 != nullptr ? a.r1[bias_head] : 0.f, reach = a.r1 != nullptr ? a.r2[bias_head] : 0.f;
  const float shift = a.pb != nullptr ? a.pb[bias_head] * -1.4426950408889634f : 0.f;
  // the mixing's factors in parts, zeros outside the heads; without mixing the unit matrix, which leaves the rounded weights as they are
  uint32_t mix[3][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float t[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int h = quad + 8 * (e & 1), g = head_of(4 * ((e & 2) + i) + x);
      t[i] = h >= H || g < 0 ? 0.f : a.talk != nullptr ? a.talk[h * H + g] : h == g ? 1.f : 0.f;
    }
    uint32_t parts[3];
    sg_parts(make_float2(t[0], t[1]), parts);
#pragma unroll
    for (int part = 0; part < 3; ++part) mix[part][e] = parts[part];
  }
  // Where this CTA's run lies: every thread asks for an entry, so that they come together; their places lie where keys will
  int* places = reinterpret_cast<int*>(k_ring);
  if (a.whole) {
    if (threadIdx.x == 0) ctl.begin = 0, ctl.end = 0x7fffffff, ctl.entry = blockIdx.x, ctl.entry_at = 0;
  } else {
    for (int e = threadIdx.x; e < a.tiles; e += SG_THREADS) places[e] = sg_places(a, e);
    __syncthreads();
  }
  if (warp == 9 && !a.whole) {
    int total = 0;
    for (int base = 0; base < a.tiles; base += 32) {      // places become sums up to and with the entry's
      int upto = base + lane < a.tiles ? places[base + lane] : 0;
#pragma unroll
      for (int offset = 1; offset < 32; offset <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, upto, offset);
        if (lane >= offset) upto += other;
      }
      if (base + lane < a.tiles) {
        places[base + lane] = total + upto;
        if (blockIdx.x == 0) a.before[base + lane + 1] = total + upto;
      }
      total += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (blockIdx.x == 0 && lane == 0) a.before[0] = 0;
    __syncwarp();
    const int runs = min((int)gridDim.x, total), mine = blockIdx.x;      // a CTA without a run has an empty one at place 0
    const int first = mine < runs ? sg_run(mine, total, runs) : 0;
    int entry = 0;
    for (int base = 0; base < a.tiles; base += 32) entry += __popc(__ballot_sync(0xffffffffu, base + lane < a.tiles && places[base + lane] <= first));
    if (lane == 0) {
      ctl.begin = first;
      ctl.end = mine < runs ? sg_run(mine + 1, total, runs) : 0;
      ctl.entry = entry;
      ctl.entry_at = entry > 0 ? places[entry - 1] : 0;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // keys will be copied over them
  }
  fa_fence_before();
  __syncthreads();
  fa_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl.tmem_holder, 0);
  constexpr int V_PER_LANES = 128 / V;                        // value heads that share the 128 lanes
  const int v_groups = (G + V_PER_LANES - 1) / V_PER_LANES;
  bool gave_up = false;

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SG_OTHER_REGISTERS));
    if (warp == 9) {
      // ------------------------------------------------------------ keys: 128 of them x 64 columns of a key head per stage
      // Keys 64 b + 16 w + i become row 32 w + 16 b + i: every computing warp finishes some of the first 64 keys first, whose values are
      // a stage of their own.
      SgStage<K_STAGES> at;
      SgPiece p;
      for (SgWalk walk(ctl); walk.next(a, p);) {
        const int* table = a.block_table + (size_t)(a.seg_slot != nullptr ? a.seg_slot[p.seg] : p.seg) * a.table_width;
        const int box = min(a.page_size, SG_KEY_BOX), own = lane * box, place = (own >> 4 & 3) * 32 + (own >> 6) * 16 + (own & 15);
        auto lookup = [&](int j) -> int {      // pool row of the lane's keys of tile j in key head 0, -1 where there are none
          const int key = (p.tile_begin + j) * SG_KEYS + own;
          const int page = j < p.tiles && own < SG_KEYS && key <= p.last_pos ? table[key >> a.page_shift] : -1;
          return page < 0 ? -1 : page * G * a.page_size + (key & (a.page_size - 1));
        };
        int row = lookup(0);
        for (int j = 0; j < p.tiles; ++j) {
          const int next_row = lookup(j + 1);
          for (int c = 0; c < G; ++c)
            for (int half = 0; half < HALVES; ++half) {
              fa_wait(&ctl.k_empty[at.stage], at.phase ^ 1u, a.error_word, 0xa1, gave_up);
              if (elect_one() && !gave_up) mbar_expect_tx(&ctl.k_full[at.stage], SG_STAGE);
              __syncwarp();
              if (own < SG_KEYS && !gave_up)      // behind the pool: zeros
                tma_load_2d(&k_map, &ctl.k_full[at.stage], k_ring + at.stage * SG_STAGE + place * 128, half * 64, row < 0 ? a.pool_rows : row + c * a.page_size);
              at.next();
            }
          row = next_row;
        }
      }
    } else if (warp == 11) {
      // ------------------------------------------------------------ values: 64 keys x 128 columns, of one value head or of two
      SgStage<V_STAGES> at;
      SgPiece p;
      for (SgWalk walk(ctl); walk.next(a, p);) {
        const int* table = a.block_table + (size_t)(a.seg_slot != nullptr ? a.seg_slot[p.seg] : p.seg) * a.table_width;
        const int box = min(a.page_size, SG_KEYS / 2), boxes = SG_KEYS / 2 / box, block = lane / boxes, offset = lane % boxes * box;
        auto lookup = [&](int j, int half) -> int {
          const int key = (p.tile_begin + j) * SG_KEYS + half * (SG_KEYS / 2) + offset;
          const int page = j < p.tiles && block < 2 && key <= p.last_pos ? table[key >> a.page_shift] : -1;
          return page < 0 ? -1 : page * G * a.page_size + (key & (a.page_size - 1));
        };
        int row[2] = {lookup(0, 0), lookup(0, 1)};
        for (int j = 0; j < p.tiles; ++j) {
          const int next_row[2] = {lookup(j + 1, 0), lookup(j + 1, 1)};
#pragma unroll
          for (int half = 0; half < 2; ++half)
            for (int group = 0; group < v_groups; ++group) {
              const int kv = V == 128 ? group : min(2 * group + block, G - 1);
              fa_wait(&ctl.v_empty[at.stage], at.phase ^ 1u, a.error_word, 0xa2, gave_up);
              if (elect_one() && !gave_up) mbar_expect_tx(&ctl.v_full[at.stage], SG_STAGE);
              __syncwarp();
              if (block < 2 && !gave_up)
                tma_load_2d(&v_map, &ctl.v_full[at.stage], v_ring + at.stage * SG_STAGE + block * (SG_STAGE / 2) + offset * 128, V == 128 ? block * 64 : 0,
                            row[half] < 0 ? a.pool_rows : row[half] + kv * a.page_size);
              at.next();
            }
          row[0] = next_row[0], row[1] = next_row[1];
        }
      }
    } else if (warp == 8) {
      // ------------------------------------------------------------ scores
      SgStage<K_STAGES> at;
      const uint32_t idesc = fa_idesc(128, fours * 4 * SG_ROWS, false);
      const uint64_t k_desc = fa_desc_k_major(smem_u32(k_ring)), q_desc = fa_desc_k_major(smem_u32(q_tile));
      unsigned t = 0, pieces = 0;
      SgPiece p;
      for (SgWalk walk(ctl); walk.next(a, p); ++pieces) {
        fa_wait(&ctl.q_ready, pieces & 1u, a.error_word, 0xa3, gave_up);
        for (int j = 0; j < p.tiles; ++j, ++t) {
          if (t > 0) fa_wait(&ctl.s_free, (t - 1) & 1u, a.error_word, 0xa4, gave_up);
          uint32_t d = tmem_base;
          uint64_t queries = q_desc;
          for (int c = 0; c < G; ++c) {
#pragma unroll
            for (int half = 0; half < HALVES; ++half) {
              fa_wait(&ctl.k_full[at.stage], at.phase, a.error_word, 0xa5, gave_up);
              fa_fence_after();
              if (elect_one() && !gave_up) {
                const uint64_t keys = k_desc + (uint64_t)(at.stage * (SG_STAGE >> 4)), columns = queries + (uint64_t)(half * (SG_SLOTS * SG_ROWS * 128 >> 4));
#pragma unroll
                for (int k = 0; k < 4; ++k) fa_mma(d, keys + 2 * k, columns + 2 * k, idesc, half > 0 || k > 0 ? 1u : 0u);
                fa_commit(&ctl.k_empty[at.stage]);
              }
              at.next();
            }
            d += fours * 4 * SG_ROWS;
            queries += (uint64_t)(fours * (4 * SG_ROWS * 128 >> 4));
          }
          if (elect_one() && !gave_up) fa_commit(&ctl.s_full);
        }
      }
    } else {
      // ------------------------------------------------------------ products with the values
      SgStage<V_STAGES> at;
      const uint64_t v_desc = fa_desc_mn_major(smem_u32(v_ring), SG_STAGE / 2), p_desc = sg_desc_mn_plain(smem_u32(p_tile), SG_P_STRIDE);
      unsigned t = 0;
      SgPiece p;
      for (SgWalk walk(ctl); walk.next(a, p);) {
        for (int j = 0; j < p.tiles; ++j, ++t) {
          const int key0 = (p.tile_begin + j) * SG_KEYS;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            fa_wait(&ctl.p_ready[half], t & 1u, a.error_word, 0xa6, gave_up);
            const int seen = p.last_pos + 1 - key0 - half * (SG_KEYS / 2);      // keys of the half up to the last row's position
            for (int group = 0; group < v_groups; ++group) {
              const int head0 = group * V_PER_LANES * per_kv, heads = min(H - head0, V_PER_LANES * per_kv);
              const uint32_t idesc = fa_idesc(128, heads * SG_ROWS, true) | (1u << 15);      // both operands MN-major
              const uint32_t d = tmem_base + SG_O_AT + head0 * SG_ROWS;
              const uint64_t weights = p_desc + (uint64_t)(head0 * (2 * SG_P_STRIDE >> 4));
              fa_wait(&ctl.v_full[at.stage], at.phase, a.error_word, 0xa7, gave_up);
              // What the last page holds behind the last row's position is not the request's: its weights are zeros, but zero times infinity is
              // not.  (Pages behind it came as zeros.)
              if (seen > 0 && seen < SG_KEYS / 2) {
                uint8_t* tile = v_ring + at.stage * SG_STAGE;
                const int upto = min(SG_KEYS / 2, (seen + a.page_size - 1) & -a.page_size);
                for (int idx = seen * 8 + lane; idx < upto * 8; idx += 32) {
                  *reinterpret_cast<uint4*>(tile + idx * 16) = make_uint4(0u, 0u, 0u, 0u);
                  *reinterpret_cast<uint4*>(tile + SG_STAGE / 2 + idx * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
              }
              fa_fence_after();
              if (elect_one() && !gave_up) {
                const uint64_t values = v_desc + (uint64_t)(at.stage * (SG_STAGE >> 4));
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  fa_mma(d, values + (uint64_t)(k * (2048 >> 4)), weights + (uint64_t)((half * 4 + k) * (256 >> 4)), idesc, j > 0 || half > 0 || k > 0 ? 1u : 0u);
                fa_commit(&ctl.v_empty[at.stage]);
                if (group == v_groups - 1) fa_commit(&ctl.pv_done[half]);
              }
              at.next();
            }
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ weights
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SG_COMPUTE_REGISTERS));
    const float2 scale2 = make_float2(a.scale * -1.4426950408889634f, a.scale * -1.4426950408889634f);
    const int key = (warp & 3) * 16;                                                // of the warp's first, of each 64
    const float* own_bias = half_bias + x * SG_BIAS + SG_KEYS - 1 - key - quad;     // + 4 u SG_BIAS + row - 64 b - 8 i
    // of a head's rows within the mixed weights: its group of heads, this half of the rows
    auto p_row = [&](int h) {
      const int head0 = h / (V_PER_LANES * per_kv) * (V_PER_LANES * per_kv), heads = min(H - head0, V_PER_LANES * per_kv);
      return 2 * head0 + half * heads + h - head0;
    };
    uint8_t* own_p = p_tile + (key + 2 * x) * 16;
    const int p_at[2] = {p_row(min(quad, H - 1)) * SG_P_STRIDE, p_row(min(quad + 8, H - 1)) * SG_P_STRIDE};

    auto fetch_queries = [&](const SgPiece& p) {      // places of no head keep what they hold: nothing is made of it
      constexpr int CHUNKS = D / 8, STEP = SG_COMPUTE / (CHUNKS * SG_ROWS);
      const int chunk = threadIdx.x % CHUNKS, r = threadIdx.x / CHUNKS % SG_ROWS;
      const bf16* src = a.q + (p.q_row + (r < p.rows ? r : 0)) * H * D + chunk * 8;
      uint8_t* dst = q_tile + (size_t)(chunk / 8) * SG_SLOTS * SG_ROWS * 128;
      int c = 0, within = threadIdx.x / (CHUNKS * SG_ROWS);
      for (int h = within; h < H; h += STEP, within += STEP) {
        while (within >= per_kv) within -= per_kv, ++c;
        const int slot = c * fours * 4 + within, row = (slot >> 2) * 64 + (r >> 1) * 8 + (slot & 3) * 2 + (r & 1);
        cp_async_16(dst + row * 128 + (((chunk & 7) ^ (row & 7)) << 4), src + h * D, r < p.rows);
      }
      cp_async_commit();
    };
    auto queries_there = [&] {
      cp_async_wait<0>();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.q_ready);
    };
    unsigned t = 0;
    SgWalk walk(ctl);
    SgPiece p;
    bool more = walk.next(a, p);
    if (more) {
      fetch_queries(p);
      queries_there();
    }
    while (more) {
      SgPiece after;
      const int own_rows = p.rows - r0;
      more = false;
      for (int j = 0; j < p.tiles; ++j, ++t) {
        const int key0 = (p.tile_begin + j) * SG_KEYS;
        // Entry row - key + 127 of a slot: what is added to the scaled score, times -log2(e); distances below zero are not seen.
        // Logarithm, exponential and reciprocal are the hardware's approximate ones: errors of a few units in the last place of a float32, far
        // inside the bfloat16 rounding of the mixed weight.
        sg_half_barrier(half);      // those of the tile before are read
        for (int i = threadIdx.x & 7; i < SG_BIAS; i += 8) {
          const int distance = p.first_pos + r0 - key0 + i - (SG_KEYS - 1);
          half_bias[bias_slot * SG_BIAS + i] = distance > 0 ? fmaf(decay, sg_log2(fmaf(reach, (float)distance, 1.f)), shift) : shift;
        }
        sg_half_barrier(half);
        fa_wait(&ctl.s_full, t & 1u, a.error_word, 0xa8, gave_up);
        fa_fence_after();
        if (j == p.tiles - 1) {      // the queries are used: the next piece's scores are formed under what is left of this one
          more = walk.next(a, after);
          if (more) fetch_queries(after);
        }
        if (own_rows <= 0) {      // an entry of few rows: these eight are none of its own, and nothing is made of their weights
          if (lane == 0) mbar_arrive(&ctl.s_free);
#pragma unroll
          for (int b = 0; b < 2; ++b) {      // not twice before the other half's first
            if (t > 0) fa_wait(&ctl.pv_done[b], (t - 1) & 1u, a.error_word, 0xab, gave_up);
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl.p_ready[b]);
          }
          continue;
        }
#pragma unroll 1
        for (int b = 0; b < 2; ++b) {      // 16 of the warp's keys at a time (not unrolled: the instruction cache)
          float2 w[4][4][2];               // [four][pair of rows][key l / 4, l / 4 + 8]
#pragma unroll
          for (int u = 0; u < 4; ++u)
            sg_tmem_load_scores(tmem_base + ((uint32_t)(2 * key + 16 * b) << 16) + u * 64 + half * 32, reinterpret_cast<float*>(w[u]));
          fa_tmem_wait_ld();
          if (b == 1) {
            fa_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl.s_free);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const float* at = own_bias + 4 * u * SG_BIAS + 2 * r - 64 * b - 8 * i;
                float2 z = __ffma2_rn(w[u][r][i], scale2, make_float2(at[0], at[1]));
                z.x = fa_exp2(fminf(z.x, 115.4f));
                z.y = fa_exp2(fminf(z.y, 115.4f));
                z = __fadd2_rn(z, make_float2(1.f, 1.f));
                w[u][r][i] = make_float2(sg_rcp(z.x), sg_rcp(z.y));
              }
          if (key0 + 64 * b + 63 > p.first_pos) {      // some row does not see all of the keys
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int unseen = key0 + 64 * b + key + 8 * i + quad - p.first_pos - r0;      // rows r0 .. r0 + unseen - 1 lie before the key
#pragma unroll
              for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  w[u][r][i].x = 2 * r < unseen ? 0.f : w[u][r][i].x;
                  w[u][r][i].y = 2 * r + 1 < unseen ? 0.f : w[u][r][i].y;
                }
            }
          }
          if (t > 0) fa_wait(&ctl.pv_done[b], (t - 1) & 1u, a.error_word, 0xa9, gave_up);      // the mixed weights of the tile before are used
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float sum[8][4] = {};      // per row: heads l / 4 and l / 4 + 8 of keys 2 (l % 4) and the next
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              auto weight = [&](int u) { return q & 1 ? w[u][q >> 1][i].y : w[u][q >> 1][i].x; };
              uint32_t low[3], high[3];
              sg_parts(make_float2(weight(0), weight(1)), low);
              sg_parts(make_float2(weight(2), weight(3)), high);
#pragma unroll
              for (int order = 2; order >= 0; --order)      // the small products first
#pragma unroll
                for (int part = order; part >= 0; --part) sg_mma(sum[q], mix[order - part], low[part], high[part]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)      // head, key as in sum
              if (quad + 8 * (e >> 1) < H)
                *reinterpret_cast<uint4*>(own_p + p_at[e >> 1] + (64 * b + 8 * i + (e & 1)) * 16) =
                    make_uint4(pack_bf16(sum[0][e], sum[1][e]), pack_bf16(sum[2][e], sum[3][e]), pack_bf16(sum[4][e], sum[5][e]), pack_bf16(sum[6][e], sum[7][e]));
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl.p_ready[b]);
        }
      }
      if (more) queries_there();
      // the sums, after the last tile's product: a thread owns one value column and eight rows
      fa_wait(&ctl.pv_done[1], (t - 1) & 1u, a.error_word, 0xaa, gave_up);
      fa_fence_after();
      const int column = V == 128 ? 2 * key + lane : (2 * key + lane) & 63, row_step = H * V;
      const uint32_t sums_at = tmem_base + ((uint32_t)(2 * key) << 16) + SG_O_AT;
      auto leave = [&](auto* first, auto round) {      // eight rows of one head after the other, four heads asked for together
        decltype(first) rows[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) rows[i] = first + i * row_step + column;
        for (int group = 0; group < v_groups; ++group) {
          const int head0 = group * V_PER_LANES * per_kv, heads = min(H - head0, V_PER_LANES * per_kv);
          // of two value heads that share the lanes, this warp's
          const int from = V == 64 && key >= 32 ? per_kv : 0, to = V == 64 && key < 32 ? min(per_kv, heads) : heads;
          for (int h = from; h < to; h += 4) {
            float o[4][8];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (h + e < to) sg_tmem_load8(sums_at + head0 * SG_ROWS + (half * heads + h + e) * 8, o[e]);
            fa_tmem_wait_ld();
            const int offset = (head0 + h) * V;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (h + e < to) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  if (i < own_rows) rows[i][offset + e * V] = round(o[e][i]);
              }
          }
        }
      };
      if (p.tile_begin == 0 && p.tiles == p.entry_tiles)
        leave(a.out + (p.q_row + r0) * row_step, [](float v) { return __float2bfloat16_rn(v); });
      else
        leave(a.partial + ((size_t)(2 * blockIdx.x + (p.tile_begin == 0 ? 1 : 0)) * a.slot_rows + r0) * row_step, [](float v) { return v; });
      fa_fence_before();
      p = after;
    }
  }
  fa_fence_before();
  __syncthreads();
  if (warp == 8) {
    fa_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(SG_TMEM_COLS) : "memory");
  }
}

// Entries that lie in several runs: their sums added in the order of the keys.  grid: (entries, parts), four neighbouring numbers per thread.
__global__ void __launch_bounds__(256)
sigmoid_add_runs_kernel(const SgArgs a, int vdim, int most_runs) {
  constexpr int BATCH = 4;
  pdl_trigger();
  pdl_wait();
  const int total = __ldcg(a.before + a.tiles), begin = __ldcg(a.before + blockIdx.x) + SG_ENTRY, end = __ldcg(a.before + blockIdx.x + 1);
  // the run that holds place x is the last one to begin at x or before
  const int runs = min(most_runs, total);
  const int first = (int)(((long long)(begin + 1) * runs - 1) / total), last = (int)(((long long)end * runs - 1) / total);
  if (first == last) return;
  const int seg = a.tile_seg[blockIdx.x], row0 = a.tile_row0[blockIdx.x];
  const int width = a.heads * vdim, count = min(a.slot_rows, a.seg_q_len[seg] - row0) * width;
  bf16* out = a.out + (size_t)(a.seg_q_start[seg] + row0) * width;
  const size_t slot = (size_t)a.slot_rows * width;
  for (int index = (blockIdx.y * 256 + threadIdx.x) * 4; index < count; index += gridDim.y * 1024) {
    float4 sum = __ldcg(reinterpret_cast<const float4*>(a.partial + (2 * (size_t)first + 1) * slot + index));
    for (int b0 = first + 1; b0 <= last; b0 += BATCH) {
      float4 part[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH; ++i)
        if (b0 + i <= last) part[i] = __ldcg(reinterpret_cast<const float4*>(a.partial + 2 * (size_t)(b0 + i) * slot + index));
#pragma unroll
      for (int i = 0; i < BATCH; ++i)
        if (b0 + i <= last) { sum.x += part[i].x; sum.y += part[i].y; sum.z += part[i].z; sum.w += part[i].w; }
    }
    *reinterpret_cast<uint2*>(out + index) = make_uint2(pack_bf16(sum.x, sum.y), pack_bf16(sum.z, sum.w));
  }
}

// Whether the launch takes the registers that the warps share out anew.  (Another compiler may give the kernel others; a split above the launch's waits forever.)
template <int D, int V>
static bool sg_registers_fit() {
  static int registers = 0;
  cudaFuncAttributes attributes;
  if (registers == 0 && cudaFuncGetAttributes(&attributes, attention_sigmoid_tcgen05_kernel<D, V>) == cudaSuccess) registers = attributes.numRegs;
  return registers == SG_LAUNCH_REGISTERS;
}

template <int D, int V>
static int sg_launch(SgArgs a, const void* k_pool, const void* v_pool, int ctas, bool cut, cudaStream_t stream) {
  CUtensorMap k_map, v_map;
  if (!cached_tile_map(&k_map, k_pool, a.pool_rows, D, a.page_size < SG_KEY_BOX ? a.page_size : SG_KEY_BOX) ||
      !cached_tile_map(&v_map, v_pool, a.pool_rows, V, a.page_size < SG_KEYS / 2 ? a.page_size : SG_KEYS / 2))
    return MLR_BAD_SIZE;
  static OncePerDevice once;
  const cudaError_t err = once([] {
    return cudaFuncSetAttribute(attention_sigmoid_tcgen05_kernel<D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sg_shared<D>(SG_HEADS));
  });
  if (err != cudaSuccess) return (int)err;
  launch_kernel(attention_sigmoid_tcgen05_kernel<D, V>, dim3(ctas), dim3(SG_THREADS), sg_shared<D>(a.heads), stream, k_map, v_map, a);
  const int status = launch_status();
  if (status != MLR_OK || !cut) return status;
  // eight CTAs per entry of the largest size, more where that leaves the device empty
  const int most = (a.slot_rows * a.heads * V + 1023) / 1024, parts = a.tiles * most < 8 * sm_count() ? most : (most + 3) / 4;
  launch_kernel(sigmoid_add_runs_kernel, dim3(a.tiles, parts), dim3(256), 0, stream, a, V, ctas);
  return launch_status();
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// 1 if the kernel takes these sizes as it was compiled, else 0.
MLR_EXPORT int mlr_attention_sigmoid_tcgen05_fits(int heads, int kv_heads, int dim, int vdim, int page_size) {
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0 || heads > SG_HEADS) return 0;
  if ((dim != 64 && dim != 128) || (vdim != 64 && vdim != 128)) return 0;
  if (kv_heads * ((heads / kv_heads + 3) / 4) * 4 > SG_SLOTS) return 0;
  if (page_size < 8 || (page_size & (page_size - 1)) != 0) return 0;
  if (dim == 64) return vdim == 64 ? sg_registers_fit<64, 64>() : sg_registers_fit<64, 128>();
  return vdim == 64 ? sg_registers_fit<128, 64>() : sg_registers_fit<128, 128>();
}

// Entries of a call at most.
MLR_EXPORT int mlr_attention_sigmoid_tcgen05_most() { return SgShape<64>::K_STAGES * SG_STAGE / 4; }

// float32 scratch of a call on `ctas` CTAs, in numbers: the cut entries' sums, then the places before each entry.
MLR_EXPORT long long mlr_attention_sigmoid_tcgen05_scratch(int tiles, int ctas, int max_rows, int heads, int vdim) {
  return 2ll * ctas * (max_rows < SG_ROWS ? max_rows : SG_ROWS) * heads * vdim + tiles + 1;
}

// As mlr_attention_sigmoid_mma, pools of pool_pages pages of a power of two of 8 tokens and more.  Entries have at most max_tiles key
// tiles of 128 and max_rows rows; scratch: see above, on a 16-byte boundary; error_word: host-visible int.
MLR_EXPORT int mlr_attention_sigmoid_tcgen05(const void* q, const void* k_pool, const void* v_pool, void* out, float* scratch,
                                             const int* tile_seg, const int* tile_row0, const int* seg_q_start, const int* seg_q_len,
                                             const int* seg_pos0, const int* block_table, const int* seg_slot, int table_width, int tiles,
                                             int heads, int kv_heads, int dim, int vdim, int page_size, int pool_pages, float scale,
                                             const float* r1, const float* r2, const float* pb, const float* talk, int ctas, int max_tiles, int max_rows,
                                             int* error_word, cudaStream_t stream) {
  if (tiles == 0) return MLR_OK;
  if (tiles < 0 || page_size <= 0 || table_width <= 0 || pool_pages <= 0 || ctas <= 0 || max_tiles <= 0 || max_rows <= 0 || scratch == nullptr ||
      error_word == nullptr || ((r1 == nullptr) != (r2 == nullptr)))
    return MLR_BAD_SIZE;
  if (!mlr_attention_sigmoid_tcgen05_fits(heads, kv_heads, dim, vdim, page_size)) return MLR_TOO_LARGE;
  const long long pool_rows = (long long)pool_pages * kv_heads * page_size;
  if (tiles > mlr_attention_sigmoid_tcgen05_most()) return MLR_TOO_LARGE;
  if (pool_rows >= (1ll << 31) || (long long)tiles * max_tiles >= (1ll << 31)) return MLR_TOO_LARGE;
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (!aligned(q) || !aligned(k_pool) || !aligned(v_pool) || !aligned(out) || !aligned(scratch)) return MLR_BAD_ALIGNMENT;
  SgArgs a;
  a.q = (const bf16*)q; a.out = (bf16*)out; a.partial = scratch;
  a.slot_rows = max_rows < SG_ROWS ? max_rows : SG_ROWS;
  a.before = reinterpret_cast<int*>(scratch + 2ll * ctas * a.slot_rows * heads * vdim);
  a.tile_seg = tile_seg; a.tile_row0 = tile_row0; a.seg_q_start = seg_q_start; a.seg_q_len = seg_q_len; a.seg_pos0 = seg_pos0;
  a.block_table = block_table; a.seg_slot = seg_slot; a.r1 = r1; a.r2 = r2; a.pb = pb; a.talk = talk;
  a.table_width = table_width; a.tiles = tiles; a.heads = heads; a.kv_heads = kv_heads; a.page_size = page_size;
  a.page_shift = 0;
  while ((1 << a.page_shift) < page_size) ++a.page_shift;
  a.pool_rows = (int)pool_rows; a.scale = scale; a.error_word = error_word;
  // Entries of up to two key tiles that run together anyway are not cut: the second launch costs more than a tile.
  a.whole = max_tiles <= 2 && tiles <= ctas;
  if (a.whole) ctas = tiles;
  const bool cut = !a.whole && max_tiles > 1;
  if (dim == 64 && vdim == 64) return sg_launch<64, 64>(a, k_pool, v_pool, ctas, cut, stream);
  if (dim == 64 && vdim == 128) return sg_launch<64, 128>(a, k_pool, v_pool, ctas, cut, stream);
  if (dim == 128 && vdim == 64) return sg_launch<128, 64>(a, k_pool, v_pool, ctas, cut, stream);
  return sg_launch<128, 128>(a, k_pool, v_pool, ctas, cut, stream);
}
