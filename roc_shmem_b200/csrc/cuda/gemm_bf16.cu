// gemm_bf16.cu — stand-alone tcgen05 bf16 GEMM:  C[M,N] = op(A) · op(B)^T, each operand
// K-major (activations, a torch Linear weight) or MN-major (as a gradient product finds it),
// fp32 accumulation in TMEM, bf16 output through TMA stores (split tiles and a ragged last
// column: direct stores); CTA pairs (cta_group::2) on tiles of
// 256 rows and 128 to 512 columns, see gemm_pair.cuh and pair_plan.h.  This is the compute core
// that the fused all-gather→GEMM and GEMM→reduce-scatter kernels build on; it has
// no counterpart in the reference, which contains no GEMM.  Problems with few rows of A
// take the weight-streaming kernel of gemm_skinny.cuh instead (plan_skinny says when).
#include <atomic>
#include <utility>

#include "gemm_pair.cuh"
#include "gemm_skinny.cuh"
#include "pair_plan.h"
#include "prefetch_plan.h"
#include "tma_host.h"

using namespace bshmem;
using namespace bshmem::gemm2;

namespace {

struct PlainParams {
  CoreParams core;
  CUtensorMap map_a, map_b, map_c;
  CUtensorMap map_b2, map_c2;  // B rows of a second accumulator (wide form), output boxes of 32 columns
  __nv_bfloat16* out;          // split form: the result, written directly
  long long ldc;
  int turned;                  // A and B have changed places, the maps of C are for its transpose
};

// One policy per operand layout.  K-major (kAmn / kBmn false): A is stored [M][K], one 128-row x 64 box per CTA and stage.
// MN-major (true): A is stored [K][M], as a gradient GEMM finds it; a stage holds two 64-wide column blocks of 64 reduction
// rows (8 KiB each, 128-byte swizzle), which the tensor core reads through MN-major descriptors — no transposed copy.
// Rows and columns beyond the matrix, the reduction included, are zero-filled by TMA.
enum Form { NARROW, WIDE, SPLIT };
template <bool kAmn, bool kBmn, int kForm>
struct PlainBf16 : PolicyDefaults {
  using Params = PlainParams;
  static constexpr bool kSplit = kForm == SPLIT, kWide = kForm == WIDE, kVarCols = !kSplit, kHalfChunks = !kSplit;
  static constexpr uint32_t kIdesc = kIdescBf16 | (kAmn ? 1u << 15 : 0u) | (kBmn ? 1u << 16 : 0u);
  static constexpr uint32_t kBlock = 64 * BK_BYTES;           // one 64 (MN) x 64 (K) block
  static constexpr uint32_t kKStepA = kAmn ? 2048 : UMMA_K_BYTES, kKStepB = kBmn ? 2048 : UMMA_K_BYTES;
  __device__ static __forceinline__ uint64_t desc_a0(uint32_t a0) { return kAmn ? ptx::umma_desc_sw128_ex(a0, kBlock, 1024) : ptx::umma_desc_sw128(a0); }
  __device__ static __forceinline__ uint64_t desc_b0(uint32_t b0) { return kBmn ? ptx::umma_desc_sw128_ex(b0, kBlock, 1024) : ptx::umma_desc_sw128(b0); }
  __device__ static __forceinline__ void load_stage(const Params&, const CUtensorMap* ma, const CUtensorMap* mb, uint32_t a_smem,
                                                    uint32_t b_smem, uint32_t bar, int kb, int a_row, int b_row, int, int, int) {
    if constexpr (kAmn) {
      ptx::tma_load_2d(a_smem, ma, bar, a_row, kb * BK);
      ptx::tma_load_2d(a_smem + kBlock, ma, bar, a_row + 64, kb * BK);
    } else {
      ptx::tma_load_2d(a_smem, ma, bar, kb * BK, a_row);
    }
    if constexpr (kBmn) {
      ptx::tma_load_2d(b_smem, mb, bar, b_row, kb * BK);
      ptx::tma_load_2d(b_smem + kBlock, mb, bar, b_row + 64, kb * BK);
    } else {
      ptx::tma_load_2d(b_smem, mb, bar, kb * BK, b_row);
    }
  }
  // MN-major column blocks are loaded whole, also where the CTA's half of an accumulator ends inside the second one
  __device__ static __forceinline__ void load_b(const Params& p, const CUtensorMap* mb, uint32_t b_smem, uint32_t bar, int kb, int b_row, int, int, int) {
    if constexpr (kBmn) {
      ptx::tma_load_2d(b_smem, mb, bar, b_row, kb * BK);
      ptx::tma_load_2d(b_smem + kBlock, mb, bar, b_row + 64, kb * BK);
    } else {
      ptx::tma_load_2d(b_smem, &p.map_b2, bar, kb * BK, b_row);
    }
  }
  __device__ static __forceinline__ int acc_cols(const Params& p, int a) { return kVarCols ? p.core.acc_cols[a] : BN; }
  __device__ static __forceinline__ uint32_t stage_tx(const Params& p) {
    if constexpr (kBmn || !kVarCols) return kWide ? WIDE_STAGE_BYTES : STAGE_BYTES;
    return A_STAGE_BYTES + (uint32_t)(p.core.acc_cols[0] + (kWide ? p.core.acc_cols[1] : 0)) / 2 * BK_BYTES;
  }
  __device__ static __forceinline__ int b_row(const Params& p, int, int n_blk) {
    return n_blk * (acc_cols(p, 0) + (kWide ? acc_cols(p, 1) : 0));
  }
  __device__ static __forceinline__ const CoreParams& core(const Params& p) { return p.core; }
  __device__ static __forceinline__ const CUtensorMap* map_a(const Params& p) { return &p.map_a; }
  __device__ static __forceinline__ const CUtensorMap* map_b(const Params& p) { return &p.map_b; }
  __device__ static __forceinline__ void tile_coords(const Params& p, int tile, int* m_blk, int* n_blk) {
    raster_coords(p.core, tile, m_blk, n_blk);
  }
  __device__ static __forceinline__ void out_target(const Params& p, int row, int col, const CUtensorMap** map, int* x, int* y) {
    *map = (row < p.core.M && col < p.core.N) ? &p.map_c : nullptr;
    *x = p.turned ? row : col;
    *y = p.turned ? col : row;
  }
  __device__ static __forceinline__ void out_target_half(const Params& p, int row, int col, const CUtensorMap** map, int* x, int* y) {
    *map = (row < p.core.M && col < p.core.N) ? &p.map_c2 : nullptr;
    *x = p.turned ? row : col;
    *y = p.turned ? col : row;
  }
  static constexpr bool kTurns = kVarCols;
  __device__ static __forceinline__ bool turned(const Params& p) { return p.turned; }
  static constexpr bool kRaggedCols = kVarCols;
  __device__ static __forceinline__ bool ragged_chunk(const Params& p, int col) { return (p.core.N & 7) && col < p.core.N && col + EPI_COLS > p.core.N; }
  __device__ static __forceinline__ void store_ragged(const Params& p, int row, int col, const uint32_t (&w)[32], int cols) {
    if (row >= p.core.M) return;
    uint16_t* dst = reinterpret_cast<uint16_t*>(p.out + row * p.ldc + col);
#pragma unroll
    for (int j = 0; j < 64; ++j)
      if (j < cols && col + j < p.core.N) dst[j] = (uint16_t)(w[j / 2] >> 16 * (j & 1));
  }
  // 16 columns of a row: one 32-byte sector, as far as the matrix goes (N need not be a multiple of 8 when B is K-major)
  __device__ static __forceinline__ void store_row16(const Params& p, int row, int col, const float4 (&v)[4]) {
    if (row >= p.core.M) return;
    __nv_bfloat16* dst = p.out + row * p.ldc + col;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 a = v[2 * h], b = v[2 * h + 1];
      const int left = p.core.N - col - 8 * h;
      if (left >= 8) {
        *reinterpret_cast<uint4*>(dst + 8 * h) = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
      } else {
        const float f[7] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z};
#pragma unroll
        for (int j = 0; j < 7; ++j)
          if (j < left) dst[8 * h + j] = __float2bfloat16_rn(f[j]);
      }
    }
  }
};

template <bool kAmn, bool kBmn>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1) gemm_bf16_kernel(const __grid_constant__ PlainParams prm) {
  extern __shared__ uint8_t smem_raw[];
  gemm_mainloop<PlainBf16<kAmn, kBmn, NARROW>>(prm, smem_raw);
}
template <bool kAmn, bool kBmn>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1) gemm_bf16_wide_kernel(const __grid_constant__ PlainParams prm) {
  extern __shared__ uint8_t smem_raw[];
  gemm_mainloop<PlainBf16<kAmn, kBmn, WIDE>>(prm, smem_raw);
}
template <bool kAmn, bool kBmn>                       // cluster size at launch: 2 * split
__global__ void __launch_bounds__(NUM_THREADS, 1) gemm_bf16_split_kernel(const __grid_constant__ PlainParams prm) {
  extern __shared__ uint8_t smem_raw[];
  gemm_mainloop<PlainBf16<kAmn, kBmn, SPLIT>>(prm, smem_raw);
}
using PlainKernel = void (*)(PlainParams);
constexpr PlainKernel kPlainKernels[2][2] = {{gemm_bf16_kernel<false, false>, gemm_bf16_kernel<false, true>},
                                             {gemm_bf16_kernel<true, false>, gemm_bf16_kernel<true, true>}};
constexpr PlainKernel kWideKernels[2][2] = {{gemm_bf16_wide_kernel<false, false>, gemm_bf16_wide_kernel<false, true>},
                                            {gemm_bf16_wide_kernel<true, false>, gemm_bf16_wide_kernel<true, true>}};
constexpr PlainKernel kSplitKernels[2][2] = {{gemm_bf16_split_kernel<false, false>, gemm_bf16_split_kernel<false, true>},
                                             {gemm_bf16_split_kernel<true, false>, gemm_bf16_split_kernel<true, true>}};

template <bool kWmn>
__global__ void __launch_bounds__(skinny::NUM_THREADS) gemm_skinny_kernel(const __grid_constant__ skinny::Params prm) {
  extern __shared__ uint8_t smem_raw[];
  skinny::body<kWmn>(prm, smem_raw);
}

int* g_err_dev[64] = {};
int g_pairs[64] = {};
int g_sms[64] = {};
int g_quads[64] = {}, g_octs[64] = {};       // clusters of two / four CTA pairs the device holds at once

int ensure_device_state(int dev) {
  if (g_err_dev[dev]) return 0;
  int sms = 0;
  BSHMEM_CUDA_TRY(cudaMalloc(&g_err_dev[dev], sizeof(int)));
  BSHMEM_CUDA_TRY(cudaMemset(g_err_dev[dev], 0, sizeof(int)));
  BSHMEM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  for (auto& row : kPlainKernels)
    for (PlainKernel k : row) BSHMEM_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
  for (auto& row : kWideKernels)
    for (PlainKernel k : row) BSHMEM_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
  for (auto& row : kSplitKernels)
    for (PlainKernel k : row) BSHMEM_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
  g_pairs[dev] = max_resident_pairs(kPlainKernels[0][0], sms);
  g_quads[dev] = max_resident_clusters(kSplitKernels[0][0], sms, 4);
  g_octs[dev] = max_resident_clusters(kSplitKernels[0][0], sms, 8);
  g_sms[dev] = sms;
  BSHMEM_CUDA_TRY(cudaFuncSetAttribute(gemm_skinny_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)skinny::SMEM_FULL));
  BSHMEM_CUDA_TRY(cudaFuncSetAttribute(gemm_skinny_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)skinny::SMEM_FULL));
  return 0;
}

// How many clusters of `split` one-per-SM skinny CTAs the device holds at once (clusters do not span GPCs, so eight CTAs
// per cluster fill fewer SMs than two).
int skinny_clusters(int dev, int split) {
  static std::atomic<int> cache[64][4] = {};
  std::atomic<int>& slot = cache[dev][split == 1 ? 0 : split == 2 ? 1 : split == 4 ? 2 : 3];
  int n = slot.load(std::memory_order_relaxed);
  if (n) return n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(8 * g_sms[dev]));
  cfg.blockDim = dim3(skinny::NUM_THREADS);
  cfg.dynamicSmemBytes = skinny::SMEM_FULL;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_skinny_kernel<false>, &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = g_sms[dev] / split; }
  slot.store(n, std::memory_order_relaxed);
  return n;
}

struct SkinnyPlan {
  int split;       // 0: leave the problem to the 256x256 tiles
  bool half;
};
// Split the reduction as far as all clusters still run at once and every CTA keeps four k-blocks.  Times in us, K x N:
//  - up to 64 tokens two CTAs per SM: 3584x8192, 16 tokens: split 1 / 2 / 4 / 8 = 17.8 / 14.3 / 13.7 / 18.0 (64 tiles:
//    256 CTAs at split 4, two waves at 8); 14336x4096: 60.6 / 34.1 / 23.7 / 22.5
//  - 65 to 128 tokens one CTA per SM with six stages, because a stage grows to 32 KiB (3584x8192, 128 tokens: 15.8
//    against 17.2 for two CTAs of three stages), unless the tiles alone nearly fill the chip and only half-size CTAs
//    can split (4096x14336: 25.8 against 27.9)
//  - above, only while the reduction can be split (3584x8192, 256 tokens: 19.8 against 24.7 for 256x256 tiles; 4096x14336
//    unsplit: 38.0 against 31.6), and beyond 208 tokens only by four or more: split in two, a CTA loads all tokens for half of
//    the reduction, a CTA pair on 256x256 tiles half of them.  Where the lines cross depends on how the tiles fill the chip,
//    few-token form against pairs at 176 / 208 / 224 / 240 / 256 tokens:
//      8192x7168  30.2-31.8   32.1-33.3   33.3-34.4   37.1-34.8   38.7-35.7
//      6168x4784  29.1-29.7   30.9-28.0   32.2-27.7   33.4-28.1   35.1-28.1
//      3584x8192  16.4-18.8   17.4-19.0   17.3-18.9   18.7-18.9   20.0-19.0
//      4096x6144  18.3-21.6   17.7-19.9   17.9-19.9   19.4-19.7   20.0-19.8
//    208 gives up to 10 % away at 192 and 208 tokens for the second and about as much at 224 for the last two; split in four,
//    14336x4096, 256 tokens: 33.6 against 42.9
//  - above 64 tokens a short reduction leaves a CTA few k-blocks to hide the exchange of its parts behind, and a CTA pair on one wave of
//    tiles of 128 columns needs about 0.16 us per k-block whatever the tokens.  The lines cross at 88 + 4.5 tokens per k-block, for every
//    N that makes one wave (1024 to 8192), few-token form against pairs:  8 k-blocks 112 / 128 / 256 tokens 6.1-5.7 / 6.2-5.8 / 8.1-5.8;
//    16: 144 / 160 / 256  7.3-7.1 / 7.8-7.1 / 9.7-7.1;  24: 192 / 224 / 256  8.8-8.4 / 9.6-8.4 / 10.4-8.5;  32: 224 / 256  9.5-9.6 /
//    10.2-9.6;  40: 256  10.3-10.8.  The pairs' sum is one chain, see below: 256 x 8192 x 2048, 0.11 % not the nearest bf16, split 0.06 %
SkinnyPlan plan_skinny(int M, int N, int K, int dev) {
  if (M > skinny::MAX_TOKENS) return {0, false};
  const int tiles = (N + skinny::ROWS - 1) / skinny::ROWS, kb = (K + skinny::BK - 1) / skinny::BK;
  if (M > 64 && kb <= 32 && 2 * M >= 176 + 9 * kb && (N + 127) / 128 <= g_pairs[dev]) return {0, false};
  auto best = [&](bool half) {
    int s = 1;
    while (s < 8 && kb >= 8 * s && (half ? tiles * s <= g_sms[dev] : tiles <= skinny_clusters(dev, 2 * s))) s *= 2;
    return s;
  };
  if (M <= 64) return {best(true), true};
  const int full = best(false);
  if (full == 2 && M > 208 && kb >= 32 && (N + BN - 1) / BN <= g_quads[dev]) return {0, false};
  if (full > 1) return {full, false};
  if (M <= 128) return {best(true), true};
  return {0, false};
}

// Few tokens: weight-streaming kernel (gemm_skinny.cuh).
int launch_skinny(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, bool w_mn, cudaStream_t st,
                  int dev, unsigned long long timeout_ns, const SkinnyPlan& plan) {
  if (reinterpret_cast<uintptr_t>(C) & 15) { host::last_error() = "gemm: the output must be 16-byte aligned"; return 1; }
  skinny::Params p;
  p.out = static_cast<__nv_bfloat16*>(C);
  p.ldo = ldc;
  p.M = M; p.N = N; p.K = K;
  p.nt = (M + 15) / 16 * 16;
  p.timeout_ns = timeout_ns;
  p.err = g_err_dev[dev];
  const uint32_t budget = (plan.half ? skinny::SMEM_HALF : skinny::SMEM_FULL) - skinny::CTRL_BYTES - 1024;
  p.stages = (int)(budget / skinny::stage_bytes(p.nt));
  if (p.stages > skinny::MAX_STAGES) p.stages = skinny::MAX_STAGES;
  p.tmem_cols = 32;
  while (p.tmem_cols < (uint32_t)p.nt) p.tmem_cols *= 2;
  p.split = plan.split;
  p.prefetch = skinny::prefetch_blocks(M, 2ll * ldb, (K + skinny::BK - 1) / skinny::BK / plan.split);
  if (p.prefetch > p.stages) p.prefetch = p.stages;
  const int tiles = (N + skinny::ROWS - 1) / skinny::ROWS;
  int rc = w_mn ? host::make_tmap_2d(&p.map_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, B, K, N, ldb, skinny::BK, 64)
                : host::make_tmap_2d(&p.map_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, B, N, K, ldb, skinny::ROWS, skinny::BK);
  if (rc) return rc;
  rc = host::make_tmap_2d(&p.map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, M, K, lda, p.nt, skinny::BK);
  if (rc) return rc;
  // a split tile is parked over the stages as nt x 512 bytes: at most 128 KiB, over four stages of 48 KiB
  if (p.stages < 2 || (p.split > 1 && (uint32_t)p.stages * skinny::stage_bytes(p.nt) < (uint32_t)p.nt * skinny::ROWS * 4)) {
    host::last_error() = "gemm: internal error, the split tile does not fit the stages";
    return 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * p.split));
  cfg.blockDim = dim3(skinny::NUM_THREADS);
  cfg.dynamicSmemBytes = skinny::smem_bytes(p.nt, p.stages);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.split; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.split > 1 ? 2 : 1;
  BSHMEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, w_mn ? gemm_skinny_kernel<true> : gemm_skinny_kernel<false>, p));
  return 0;
}

}  // namespace

extern "C" {

const char* bshmem_gemm_last_error() { return host::last_error().c_str(); }

// C = op(A) · op(B)^T with a reduction of K.  a_mn = 0: A is [M, K] row-major (lda elements); a_mn = 1: A is [K, M] (the
// reduction runs over its rows).  Likewise B: [N, K] or, with b_mn, [K, N].  C: [M, N] (ldc).  All bf16.
// lda, ldb, ldc, and K (M, N) where it is the contiguous extent of an operand, must be multiples of 8 and the bases
// 16-byte aligned (TMA).  The kernel runs as CTA pairs (clusters of two); max_ctas <= 1 uses every pair the device can
// hold.  timeout_ms bounds every in-kernel wait.
int bshmem_gemm_bf16_ex(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int a_mn, int b_mn,
                        void* stream, int max_ctas, int timeout_ms) {
  if (M <= 0 || N <= 0 || K <= 0) { host::last_error() = "gemm: empty problem"; return 1; }
  if ((!(a_mn && b_mn) && K % 8) || (a_mn && M % 8) || (b_mn && N % 8) || (lda % 8) || (ldb % 8) || (ldc % 8)) {
    host::last_error() = "gemm: K and leading dimensions must be multiples of 8";
    return 1;
  }
  int dev = 0;
  BSHMEM_CUDA_TRY(cudaGetDevice(&dev));
  int rc = ensure_device_state(dev);
  if (rc) return rc;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned long long timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 2000) * 1000000ull;
  if (max_ctas <= 1 && !a_mn) {        // an explicit limit on the CTAs keeps the persistent kernel
    const SkinnyPlan plan = plan_skinny(M, N, K, dev);
    if (plan.split) return launch_skinny(A, B, C, M, N, K, lda, ldb, ldc, b_mn != 0, st, dev, timeout_ns, plan);
  }
  int pairs = g_pairs[dev];
  if (max_ctas > 1 && max_ctas / 2 < pairs) pairs = max_ctas / 2;
  if (pairs < 1) { host::last_error() = "gemm: the device holds no CTA pair of this kernel"; return 1; }
  // Few tiles: split each over the two or four pairs of a cluster while all clusters run at once.  Parking and adding the
  // parts costs about 4 us, what a pair needs for 14 k-blocks.  Where tiles of 128 columns make one wave they are the better answer up
  // to deeper reductions, in every layout (us, 32 / 40 / 48 / 56 / 64 k-blocks): 512 x 2048 10.9 / 12.9 / 14.6 / 16.3 / 18.0, split in
  // two 12.9 / 14.2 / 15.5 / 16.6 / 17.8; 768 x 1024 9.6 / 11.9 / 13.7 / 15.6 / 17.2, split in four 11.1 / 12.0 / 12.9 / 13.7 / 14.4.
  // No wider tile is better than these then: 512 x 2048 x 1536, both operands MN-major, by 128 / 160 / 192 / 224 / 256 columns
  // 9.3 / 10.1 / 10.4 / 11.4 / 13.0.  The unsplit sum is one chain of up to 59 k-blocks in tensor memory, which truncates, where the split one adds two
  // or four shorter chains: of normal inputs 0.12 % of the bf16 results are not the nearest to the sum in 64 bits, split in two 0.06 %
  // (768 x 1024 x 2560: 0.14 %, split in four 0.04 %; every product of 128 k-blocks 0.46 %); the 2-norm of the error differs in the seventh digit.
  const int kb = (K + BK - 1) / BK;
  PlainParams p;
  p.core.split = 1;
  const long long row_blocks = (M + BM - 1) / BM;
  const bool one_wave = row_blocks * ((N + 127) / 128) <= pairs;
  if (max_ctas <= 1) {
    const long long tiles = row_blocks * ((N + BN - 1) / BN);
    if (tiles <= g_octs[dev] && kb >= (one_wave ? 41 : 24)) p.core.split = 4;
    else if (tiles <= g_quads[dev] && kb >= (one_wave ? 60 : 32)) p.core.split = 2;
  }
  // Tiles have 256 rows, but their columns come in steps of 32: where that leaves less of them empty, A and B change places and C is
  // stored transposed (its TMA boxes are cut off on 16 bytes, so N is a multiple of 8); the bits are the same.  us before, with tiles of
  // two accumulators from 352 columns on, and now, with those from 288: 264 x 8192 x 3584 22.9 and 18.9, 320 x 7168 x 8192 52.5 and 40.5,
  // 640 x 4096 x 14336 86 and 62, 1152 x 8192 x 3584 69 and 58.  Not for an MN-major A, which would be loaded like an MN-major B
  // (see plan_width), nor narrow tiles of two accumulators for such a B: 264 x 14336 x 4096 so took 63, as it is 50.  A threshold of 3 %,
  // about what the estimates are good for.
  auto plan = [&](int rows, int cols, bool mn) { return plan_width((rows + BM - 1) / BM, cols, K, pairs, 32, mn, true, 512, 0, mn ? 352 : 288); };
  Width w = p.core.split > 1 ? Width{{BN, 0}} : one_wave ? Width{{128, 0}} : plan(M, N, b_mn != 0);
  p.turned = 0;
  if (p.core.split == 1 && !one_wave && !a_mn && N % 8 == 0) {
    const Width t = plan(N, M, false);
    if (t.cost < 0.97 * w.cost) {
      w = t;
      p.turned = 1;
      std::swap(A, B);
      std::swap(M, N);
      std::swap(lda, ldb);
      std::swap(a_mn, b_mn);
    }
  }
  const int width = w.cols[0] + w.cols[1];
  p.core.acc_cols[0] = w.cols[0];
  p.core.acc_cols[1] = w.cols[1];
  p.core.M = M; p.core.N = N; p.core.K = K;
  p.core.num_m_blocks = (M + BM - 1) / BM;
  p.core.num_n_blocks = (N + width - 1) / width;
  // row blocks that are worked on side by side: wide tiles are fewer (8192 x 8192 x 3584 by 512 columns: 4, 8, 12, 16 row blocks
  // 365, 355, 352, 350 us)
  p.core.group_m = w.cols[1] ? 16 : 8;
  p.core.timeout_ns = timeout_ns;
  p.core.err = g_err_dev[dev];
  const auto bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  rc = a_mn ? host::make_tmap_2d(&p.map_a, bf, 2, A, K, M, lda, 64, 64) : host::make_tmap_2d(&p.map_a, bf, 2, A, M, K, lda, CTA_M, 64);
  if (rc) return rc;
  rc = b_mn ? host::make_tmap_2d(&p.map_b, bf, 2, B, K, N, ldb, 64, 64) : host::make_tmap_2d(&p.map_b, bf, 2, B, N, K, ldb, w.cols[0] / 2, 64);
  if (rc) return rc;
  if (w.cols[1] && !b_mn) rc = host::make_tmap_2d(&p.map_b2, bf, 2, B, N, K, ldb, w.cols[1] / 2, 64);
  if (rc) return rc;
  if ((w.cols[0] | w.cols[1]) & 63)
    rc = p.turned ? host::make_tmap_2d(&p.map_c2, bf, 2, C, N, M, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_NONE)
                  : host::make_tmap_2d(&p.map_c2, bf, 2, C, M, N, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
  if (rc) return rc;
  rc = p.turned ? host::make_tmap_2d(&p.map_c, bf, 2, C, N, M, ldc, EPI_COLS, 32, CU_TENSOR_MAP_SWIZZLE_NONE)
                : host::make_tmap_2d(&p.map_c, bf, 2, C, M, N, ldc, 32, EPI_COLS);
  if (rc) return rc;
  const int tiles = p.core.num_m_blocks * p.core.num_n_blocks;
  p.out = static_cast<__nv_bfloat16*>(C);
  p.ldc = ldc;
  if (tiles < pairs) pairs = tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pairs * p.core.split));
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)(2 * p.core.split); attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.core.split > 1 ? 2 : 1;
  const auto& kernels = p.core.split > 1 ? kSplitKernels : w.cols[1] ? kWideKernels : kPlainKernels;
  BSHMEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernels[a_mn ? 1 : 0][b_mn ? 1 : 0], p));
  return 0;
}

int bshmem_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                     void* stream, int max_ctas, int timeout_ms) {
  return bshmem_gemm_bf16_ex(A, B, C, M, N, K, lda, ldb, ldc, 0, 0, stream, max_ctas, timeout_ms);
}

// Reads (and clears) the device error word of the current device: 0 = no bounded wait ran out.
int bshmem_gemm_error_site(int clear) {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || !g_err_dev[dev]) return 0;
  cudaMemcpy(&v, g_err_dev[dev], sizeof(int), cudaMemcpyDeviceToHost);
  if (clear && v) cudaMemset(g_err_dev[dev], 0, sizeof(int));
  return v;
}

}  // extern "C"
