// y[M,N] = x[M,K] * W[N,K]^T (+ bias[N]) on the CUDA cores, float32 multiply-add throughout.
//
// This is the matrix product of the true 32-bit path (no TF32) for weights that linear_split.cu does not take, and the fallback
// of the bfloat16 path for shapes the tensor-core kernel refuses.  Weights keep the checkpoint's
// [out, in] layout, as the reference's F.linear calls do (qwen_model_runner.py:88-102,183,215-217).
//
// Every output element is a chain of fmaf over k in ascending order (for long k of narrow outputs up to four such
// chains, cut at places that N and K alone decide, added in order), whatever M, the tile shape or the position of the
// row in the batch: results do not depend on how tokens are batched.  Any M, N, K is accepted.
#include "copy_async.cuh"

namespace mlr {

// Bound by the multiply-add pipes and the shared memory that feeds them (and, for a handful of rows, by the stream of
// weights).  Both operand tiles lie in shared memory as they lie in memory, rows of BK entries along k at a pitch of
// BK + 4, filled by asynchronous copies STAGES - 1 k blocks ahead; a thread reads four (or two) entries of k per load, and
// the rows that one such load of a warp touches (4 rows of x, 8 rows of W) fall into different banks.  A thread holds
// TM x TN outputs, rows 4 apart and columns 8 apart; a warp 4*TM x 8*TN.
// Measured (B200, 600 rows, K 896 -> 9,728, the gate, 4,864 -> 896): 1,458 us with 4 x 4 outputs per thread read one
// number at a time and no copy under the arithmetic, 494 us now; products of many rows reach 41 of 74 TFLOP/s (11 before).
// A thread tile of 8 x 16 in 128 x 128 CTAs was no faster (39 TFLOP/s).
constexpr int STAGES = 4;

template <int BM, int BN, int BK>
constexpr size_t simt_shared() { return (size_t)STAGES * (BM + BN) * (BK + 4) * sizeof(float); }

// Rows row0 .. row0 + ROWS - 1, entries k0 .. k0 + BK - 1 of a row-major [rows, K] operand; what lies outside becomes zero.
template <typename TIn, int ROWS, int BK, int THREADS, bool VEC>
__device__ __forceinline__ void fetch_tile(float* tile, const TIn* src, int row0, int rows, int k0, int end_k, int K) {
  constexpr int PITCH = BK + 4;
  if constexpr (VEC) {          // float32 rows of whole 16-byte pieces
#pragma unroll
    for (int i = 0; i < (ROWS * (BK / 4) + THREADS - 1) / THREADS; ++i) {
      const int idx = threadIdx.x + i * THREADS;
      if (ROWS * (BK / 4) % THREADS != 0 && idx >= ROWS * (BK / 4)) break;
      const int r = idx / (BK / 4), c = (idx % (BK / 4)) * 4;
      float* dst = tile + r * PITCH + c;
      if (row0 + r < rows && k0 + c < end_k)
        copy_async_16(dst, reinterpret_cast<const float*>(src) + (size_t)(row0 + r) * K + k0 + c);
      else
        *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {
    for (int idx = threadIdx.x; idx < ROWS * BK; idx += THREADS) {
      const int r = idx / BK, c = idx % BK;
      tile[r * PITCH + c] = (row0 + r < rows && k0 + c < end_k) ? to_float(src[(size_t)(row0 + r) * K + k0 + c]) : 0.f;
    }
  }
}

template <int N>
__device__ __forceinline__ void load_entries(float (&v)[N], const float* src) {
  if constexpr (N == 4) {
    const float4 q = *reinterpret_cast<const float4*>(src);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else {
    const float2 q = *reinterpret_cast<const float2*>(src);
    v[0] = q.x, v[1] = q.y;
  }
}

template <typename TIn, typename TOut, int BM, int BN, int TM, int TN, int BK, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), BM * BN >= 64 * 128 ? 3 : 4)
linear_simt_kernel(const TIn* x, const TIn* __restrict__ w, const TIn* __restrict__ bias,
                   TOut* __restrict__ y, float* __restrict__ partial, int M, int N, int K, int part_k) {
  constexpr int THREADS = (BM / TM) * (BN / TN), PITCH = BK + 4;
  constexpr int WARPS_N = BN / (8 * TN);
  static_assert(BM % (4 * TM) == 0 && BN % (8 * TN) == 0 && THREADS % 32 == 0, "warps cover 4*TM x 8*TN outputs");
  extern __shared__ __align__(16) float shared[];
  float* a_tiles = shared;
  float* b_tiles = shared + STAGES * BM * PITCH;
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int row = (warp / WARPS_N) * 4 * TM + (lane >> 3), col = (warp % WARPS_N) * 8 * TN + (lane & 7);
  const bool live = m0 + (warp / WARPS_N) * 4 * TM < M;      // some row of this warp exists
  const int first_k = blockIdx.z * part_k, end_k = min(K, first_k + part_k);      // this CTA's part of every sum
  const int blocks = (end_k - first_k + BK - 1) / BK;

  auto fetch = [&](int block) {
    if (block < blocks) {
      fetch_tile<TIn, BM, BK, THREADS, VEC>(a_tiles + (block % STAGES) * BM * PITCH, x, m0, M, first_k + block * BK, end_k, K);
      fetch_tile<TIn, BN, BK, THREADS, VEC>(b_tiles + (block % STAGES) * BN * PITCH, w, n0, N, first_k + block * BK, end_k, K);
    }
    copy_async_commit();
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);

  for (int block = 0; block < blocks; ++block) {
    copy_async_wait<STAGES - 2>();
    __syncthreads();      // block's tiles are there for all, and all are done with the tiles before
    fetch(block + STAGES - 1);
    if (!live) continue;
    const float* a_tile = a_tiles + (block % STAGES) * BM * PITCH + row * PITCH;
    const float* b_tile = b_tiles + (block % STAGES) * BN * PITCH + col * PITCH;
    // 64 outputs per thread leave registers for two entries of k at a time, fewer outputs for four
    constexpr int KV = TM * TN >= 64 ? 2 : 4;
#pragma unroll
    for (int k = 0; k < BK; k += KV) {
      float b[TN][KV];
#pragma unroll
      for (int j = 0; j < TN; ++j) load_entries<KV>(b[j], b_tile + 8 * j * PITCH + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        float a[KV];
        load_entries<KV>(a, a_tile + 4 * i * PITCH + k);
#pragma unroll
        for (int e = 0; e < KV; ++e)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[e], b[j][e], acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + row + 4 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + col + 8 * j;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (partial != nullptr) {
        partial[((size_t)blockIdx.z * M + gm) * N + gn] = v;
        continue;
      }
      if (bias != nullptr) v += to_float(bias[gn]);
      y[(size_t)gm * N + gn] = from_float<TOut>(v);
    }
  }
}

// The parts of every sum in the order of k, then the bias.
template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256)
linear_simt_add_kernel(const float* partial, const TIn* __restrict__ bias, TOut* __restrict__ y, long long count, int N, int parts) {
  pdl_trigger();
  pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= count) return;
  float v = partial[i];
  for (int p = 1; p < parts; ++p) v += partial[p * count + i];
  if (bias != nullptr) v += to_float(bias[i % N]);
  y[i] = from_float<TOut>(v);
}

// Parts of a sum over k.  Long sums of narrow outputs have few CTAs, each with a long chain of dependent steps; they
// are cut into up to four parts of at least 1,024 entries, a rule on N and K alone, so that an output's additions keep
// their order whatever the number of rows.  Wide outputs (a vocabulary) have CTAs enough.
inline int simt_parts(int N, int K) { return N > 16384 ? 1 : K / 1024 < 1 ? 1 : K / 1024 > 4 ? 4 : K / 1024; }

// Rows whose parts are in scratch at a time, whole tiles of them: the parts of many rows and columns would be several copies of a large
// output (4,096 rows of 16,384 in two parts 537 MB).  At most 128 MB of them; an output's additions keep their order.  Measured in us, all
// rows together / within 64 MB / 128 MB: [M, N, K] = [4096, 3584, 4100] 2,874 / 3,144 / 2,930, [4096, 16384, 2048] 6,442 / 6,688 / 6,561,
// [2048, 3584, 18944] 6,465 / 6,942 / 6,458 (whose parts are 117 MB): each block's last CTAs leave SMs idle.
inline int simt_block_rows(int M, int N, int K) {
  constexpr long long SCRATCH = 32ll << 20;      // numbers
  const int parts = simt_parts(N, K);
  if (parts == 1 || (long long)parts * M * N <= SCRATCH) return M;
  const long long most = SCRATCH / ((long long)parts * N) / 64 * 64;      // N is at most 16,384: 512 and more
  const long long blocks = (M + most - 1) / most;
  return (int)(((M + blocks - 1) / blocks + 63) / 64 * 64);
}

template <typename TIn, typename TOut, int BM, int BN, int TM, int TN, int BK>
int linear_simt_tiles(const void* x, const void* w, const void* bias, void* y, float* partial, int M, int N, int K, bool vec,
                      cudaStream_t stream) {
  auto kernel = linear_simt_kernel<TIn, TOut, BM, BN, TM, TN, BK, false>;
  if constexpr (sizeof(TIn) == 4) {
    if (vec) kernel = linear_simt_kernel<TIn, TOut, BM, BN, TM, TN, BK, true>;
  }
  constexpr size_t shared = simt_shared<BM, BN, BK>();
  if (shared > 48 * 1024) {
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (err != cudaSuccess) return (int)err;
  }
  const int parts = simt_parts(N, K);
  const int part_k = ((K + parts - 1) / parts + 63) / 64 * 64;
  launch_kernel(kernel, dim3((N + BN - 1) / BN, (M + BM - 1) / BM, parts), dim3((BM / TM) * (BN / TN)), shared, stream,
                (const TIn*)x, (const TIn*)w, (const TIn*)bias, (TOut*)y, parts > 1 ? partial : nullptr, M, N, K, part_k);
  int status = launch_status();
  if (status != MLR_OK || parts == 1) return status;
  const long long count = (long long)M * N;
  launch_kernel(linear_simt_add_kernel<TIn, TOut>, dim3((unsigned)((count + 255) / 256)), dim3(256), 0, stream,
                (const float*)partial, (const TIn*)bias, (TOut*)y, count, N, parts);
  return launch_status();
}

// The tile of a product.  Per step of k the busiest SM spends on its CTAs `work` cycles each (measured with many rows:
// 71, 69, 44 and 20 multiply-adds per cycle and SM from the largest tile to the smallest: the more outputs a thread has,
// the fewer loads per multiply-add), but per round of the CTAs it holds `together` no less than the `step` cycles that one CTA
// alone takes.  The cheapest wins: many rows get 64 x 128 or 64 x 64 (within a few percent of one another), a few dozen
// rows or few columns smaller tiles that keep all SMs busy, a handful of rows 16 x 16, whose CTAs only stream weights.
// Times in us at [N, K] = [9728, 896] / [896, 4864], tiles from large to small: 16 rows 89 38 32 37 / 86 48 22 29, 200 rows
// 153 132 150 276 / 150 94 103 143, 1,500 rows 645 664 1017 2010 / 361 370 522 1017.
// Whole products before these tiles and copies / now, from a flushed L2: 1 and 8 rows [9728, 896] 145 150 / 19 27, [896, 4864] 678 710 / 16 20,
// a head of [151936, 896] 483 493 / 145 150; bfloat16 and 32-bit operands of odd lengths, which come by plain loads: 1, 64 and 600 rows
// [4864, 897] 133 193 299 / 35 74 250 and 152 219 301 / 37 102 279, [2000, 2002] 305 453 406 / 68 145 307 and 346 510 434 / 68 201 379.
struct SimtTile {
  int m, n, together;
  float work, step;
};
constexpr SimtTile SIMT_TILES[] = {{64, 128, 3, 115.f, 137.f}, {64, 64, 4, 59.f, 76.f}, {32, 32, 8, 23.f, 35.f}, {16, 16, 8, 13.f, 30.f}};

inline int simt_plan(int M, int N, int K) {
  int best = 0;
  float best_cost = 0.f;
  for (int i = 0; i < 4; ++i) {
    const SimtTile& t = SIMT_TILES[i];
    const long long ctas = (long long)((M + t.m - 1) / t.m) * ((N + t.n - 1) / t.n) * simt_parts(N, K);
    const long long per_sm = (ctas + sm_count() - 1) / sm_count();                       // CTAs the busiest SM gets
    const float work = per_sm * t.work, chain = (per_sm + t.together - 1) / t.together * t.step;
    const float cost = work > chain ? work : chain;
    if (i == 0 || cost < best_cost) {
      best = i;
      best_cost = cost;
    }
  }
  return best;
}

template <typename TIn, typename TOut>
int linear_simt_block(const void* x, const void* w, const void* bias, void* y, float* partial, int M, int N, int K,
                      cudaStream_t stream) {
  const bool vec = K % 4 == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0;
  switch (simt_plan(M, N, K)) {
    case 0: return linear_simt_tiles<TIn, TOut, 64, 128, 8, 8, 16>(x, w, bias, y, partial, M, N, K, vec, stream);
    case 1: return linear_simt_tiles<TIn, TOut, 64, 64, 4, 8, 32>(x, w, bias, y, partial, M, N, K, vec, stream);
    case 2: return linear_simt_tiles<TIn, TOut, 32, 32, 2, 4, 32>(x, w, bias, y, partial, M, N, K, vec, stream);
    default: return linear_simt_tiles<TIn, TOut, 16, 16, 1, 2, 64>(x, w, bias, y, partial, M, N, K, vec, stream);
  }
}

template <typename TIn, typename TOut>
int linear_simt_launch(const void* x, const void* w, const void* bias, void* y, float* partial, int M, int N, int K,
                       cudaStream_t stream) {
  const int block = simt_block_rows(M, N, K);
  for (int row = 0; row < M; row += block) {
    const int status = linear_simt_block<TIn, TOut>((const TIn*)x + (size_t)row * K, w, bias, (TOut*)y + (size_t)row * N, partial,
                                                    M - row < block ? M - row : block, N, K, stream);
    if (status != MLR_OK) return status;
  }
  return MLR_OK;
}

}  // namespace mlr

using namespace mlr;

MLR_DEFINE_PDL_SWITCH

// How many parts a product's sums over k are taken in; with more than one mlr_linear_simt needs float32 scratch
// [parts, rows, N] in `partial`, for the rows it takes at a time.
MLR_EXPORT int mlr_linear_simt_parts(int N, int K) { return N <= 0 || K <= 0 ? 1 : mlr::simt_parts(N, K); }
MLR_EXPORT int mlr_linear_simt_block_rows(int M, int N, int K) { return M <= 0 || N <= 0 || K <= 0 ? M : mlr::simt_block_rows(M, N, K); }

// in_dtype: storage of x, w and bias.  out_dtype: storage of y (float32 output from bfloat16
// inputs is used for logits).
MLR_EXPORT int mlr_linear_simt(const void* x, const void* w, const void* bias, void* y, int M, int N,
                               int K, float* partial, int in_dtype, int out_dtype, cudaStream_t stream) {
  if (M == 0) return MLR_OK;
  if (M < 0 || N <= 0 || K <= 0) return MLR_BAD_SIZE;
  if ((M + 15) / 16 > 65535) return MLR_TOO_LARGE;
  if (partial == nullptr && simt_parts(N, K) > 1) return MLR_BAD_SIZE;
  if (in_dtype == MLR_F32 && out_dtype == MLR_F32)
    return linear_simt_launch<float, float>(x, w, bias, y, partial, M, N, K, stream);
  if (in_dtype == MLR_BF16 && out_dtype == MLR_BF16)
    return linear_simt_launch<bf16, bf16>(x, w, bias, y, partial, M, N, K, stream);
  if (in_dtype == MLR_BF16 && out_dtype == MLR_F32)
    return linear_simt_launch<bf16, float>(x, w, bias, y, partial, M, N, K, stream);
  return MLR_BAD_DTYPE;
}
