// moe_gemm.cu — grouped (per-expert) tcgen05 GEMM for the MoE layer.  The K-major forms (gate/up, down and the two
// data-gradient GEMMs) and the weight-gradient form on token-major operands run on the CTA-pair main loop of gemm_pair.cuh
// (cta_group::2, the epilogue of one tile overlaps the MMAs of the next), few rows per expert on the grouped form of
// gemm_skinny.cuh; the ragged-K form runs on the single-CTA main loop of gemm_core.cuh, as does the weight-gradient form on a
// device that holds no CTA pair of it.
//
//   C_g = A_g · B_g^T  for every local expert g, bf16 operands, K-major but for the weight gradient's:
//     rows mode   A: [G][cap rows][K]   B: [G][N][K]    C: [G][cap][N]
//                 the row count of group g is read from device memory (tokens that arrived),
//                 so no host synchronisation is needed between dispatch and the GEMM;
//     ragged-K    A: [G][M][cap]        B: [G][N][cap]  C: [G][M][N]
//                 the reduction length of group g is the device-side token count (weight
//                 gradients over transposed, zero-padded activations).
//   Optional gated epilogue (SwiGLU fused: interleaved gate/up columns → silu(g)·u) and an
//   optional wait on the dispatch arrival words before the first A load.
// There is no grouped GEMM in the reference; the layout conventions are those of
// moe_kernels.cu.
#include <cstdlib>

#include "gemm_pair.cuh"
#include "gemm_skinny.cuh"
#include "moe_common.h"
#include "pair_plan.h"
#include "tma_host.h"

using namespace bshmem;
using namespace bshmem::gemm;

namespace {

struct GroupedParams {
  CoreParams core;                 // N = output columns of the accumulator, K = full reduction length
  CUtensorMap map_a, map_b, map_c;
  CUtensorMap map_b2;              // CTA pairs: B rows of a tile's second accumulator
  const int* rows;                 // [G] valid rows per group (rows mode) or null (all `fixed_rows`)
  const int* klen;                 // [G] reduction length per group (ragged-K mode) or null
  int G, fixed_rows;
  int a_blocks_per_group;          // 256-row blocks between consecutive groups in A and C
  int b_rows_per_group;            // rows between consecutive groups in B
  int k_rows_per_group;            // token rows between consecutive groups of A and B (transposed-operand mode)
  int tn3d;                        // transposed-operand mode: maps are 3-D column-block views, one copy per operand
  int group_m;
  int P;                           // arrival wait: number of words, 0 = no wait
  const unsigned long long* arrive;
  const int* expected;
  __nv_bfloat16* act;              // training forward: activations [G * rows, N / 2] next to the pre-activations C
  long long ld_act;
  const __nv_bfloat16* gu;         // SwiGLU backward: saved pre-activations [G * rows, 2 N]
  long long ld_gu;
};

template <bool kGatedEpi>
struct Grouped : PolicyDefaults {
  using Params = GroupedParams;
  static constexpr int kElemBytes = 2;
  static constexpr uint32_t kIdesc = ptx::umma_idesc(1, 1, UMMA_M, UMMA_N);
  static constexpr bool kGated = kGatedEpi;
  __device__ static __forceinline__ const CoreParams& core(const Params& p) { return p.core; }
  __device__ static __forceinline__ const CUtensorMap* map_a(const Params& p) { return &p.map_a; }
  __device__ static __forceinline__ const CUtensorMap* map_b(const Params& p) { return &p.map_b; }
  __device__ static __forceinline__ int group_rows(const Params& p, int g) { return p.rows ? p.rows[g] : p.fixed_rows; }
  __device__ static __forceinline__ int num_tiles(const Params& p) {
    int t = 0;
    for (int g = 0; g < p.G; ++g) t += ((group_rows(p, g) + BM - 1) / BM) * p.core.num_n_blocks;
    return t;
  }
  // m_blk is a virtual block index: group * a_blocks_per_group + block inside the group
  __device__ static __forceinline__ void tile_coords(const Params& p, int tile, int* m_blk, int* n_blk) {
    int g = 0, mb_g = 0;
    for (; g < p.G; ++g) {
      mb_g = (group_rows(p, g) + BM - 1) / BM;
      int tg = mb_g * p.core.num_n_blocks;
      if (tile < tg) break;
      tile -= tg;
    }
    coords_in_group(p, g, mb_g, tile, m_blk, n_blk);
  }
  // tile number `tile` of group g, which has `blocks` row blocks
  __device__ static __forceinline__ void coords_in_group(const Params& p, int g, int blocks, int tile, int* m_blk, int* n_blk) {
    const int per = p.group_m * p.core.num_n_blocks;
    const int sg = tile / per, first = sg * p.group_m;
    const int rows = min(p.group_m, blocks - first);
    const int in = tile - sg * per;
    *m_blk = g * p.a_blocks_per_group + first + in % rows;
    *n_blk = in / rows;
  }
  __device__ static __forceinline__ int a_row(const Params&, int m_blk) { return m_blk * BM; }
  __device__ static __forceinline__ int b_row(const Params& p, int m_blk, int n_blk) {
    return (m_blk / p.a_blocks_per_group) * p.b_rows_per_group + n_blk * BN;
  }
  __device__ static __forceinline__ int num_kb(const Params& p, int m_blk, int bk) {
    int k = p.klen ? p.klen[m_blk / p.a_blocks_per_group] : p.core.K;
    int n = (k + bk - 1) / bk;
    return n < 1 ? 1 : n;     // an empty group still runs one (all-zero) k-block so that C becomes 0
  }
  __device__ static __forceinline__ bool a_ready(const Params& p, int, Guard& g) {
    for (int s = 0; s < p.P; ++s)
      if (!wait_ge<true>(p.arrive + s, (unsigned long long)p.expected[s], g, ERR_PEER_SIGNAL)) return false;
    if (p.P) ptx::fence_proxy_async_all();   // peer stores (generic proxy) before the TMA reads
    return true;
  }
  __device__ static __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    ptx::umma_f16(d, a, b, idesc, acc);
  }
  __device__ static __forceinline__ uint32_t pack(uint32_t lo, uint32_t hi, const Params&, int, int) {
    return pack_bf16(__uint_as_float(lo), __uint_as_float(hi));
  }
  __device__ static __forceinline__ void out_target(const Params& p, int row, int col, const CUtensorMap** map, int* x, int* y) {
    *map = &p.map_c;       // rows beyond a group's count are scratch inside the group's own region
    *x = col;
    *y = row;
  }
};

// Weight-gradient flavour: C_g[M, N] = A_g^T · B_g with A_g stored [tokens_g][M] and B_g stored [tokens_g][N]
// (the token-major activations as they are), i.e. both operands MN-major; the reduction runs over the
// ragged token dimension.  A stage holds, per operand, four 64-wide MN blocks of 64 tokens each (8 KiB per
// block, 128-byte swizzle): inside a block 8 tokens form one 1 KiB swizzle atom (SBO), blocks are 8 KiB apart
// (LBO).  Tokens in [count, next multiple of 64) of every group must be zero (bshmem_moe_zero_pad_rows).
struct GroupedTN : Grouped<false> {
  static constexpr uint32_t kIdesc = ptx::umma_idesc_mn_major(1, 1, UMMA_M, UMMA_N);
  static constexpr uint32_t kBlock = 64 * BK_BYTES;            // one 64 (MN) x 64 (tokens) block: 8 KiB
  // the "row" values handed to load_stage are the tile's block indices; the token row comes from the group
  __device__ static __forceinline__ int a_row(const Params&, int m_blk) { return m_blk; }
  __device__ static __forceinline__ int b_row(const Params&, int, int n_blk) { return n_blk; }
  __device__ static __forceinline__ void load_stage(const Params& p, const CUtensorMap* ma, const CUtensorMap* mb, uint32_t a_smem,
                                                    uint32_t b_smem, uint32_t bar, int k_elem, int m_blk, int n_blk) {
    const int g = m_blk / p.a_blocks_per_group;
    const int tok = g * p.k_rows_per_group + k_elem;
    const int m0 = (m_blk - g * p.a_blocks_per_group) * BM, n0 = n_blk * BN;
    if (p.tn3d) {                  // one 32 KiB copy per operand: {64, 64 tokens, 4 column blocks}
      ptx::tma_load_3d(a_smem, ma, bar, 0, tok, m0 / 64);
      ptx::tma_load_3d(b_smem, mb, bar, 0, tok, n0 / 64);
      return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      ptx::tma_load_2d(a_smem + i * kBlock, ma, bar, m0 + i * 64, tok);
      ptx::tma_load_2d(b_smem + i * kBlock, mb, bar, n0 + i * 64, tok);
    }
  }
  // one MMA consumes 16 tokens = two swizzle atoms (2 KiB) of every MN block
  __device__ static __forceinline__ uint64_t desc_a(uint32_t a0, int half, int k) {
    return ptx::umma_desc_sw128_ex(a0 + half * 2 * kBlock + k * 2048, kBlock, 1024);
  }
  __device__ static __forceinline__ uint64_t desc_b(uint32_t b0, int k) { return ptx::umma_desc_sw128_ex(b0 + k * 2048, kBlock, 1024); }
};

__global__ void __launch_bounds__(NUM_THREADS, 1) grouped_gemm_kernel(const __grid_constant__ GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  gemm_mainloop<Grouped<false>>(prm, smem_raw);
}
__global__ void __launch_bounds__(NUM_THREADS, 1) grouped_gemm_gated_kernel(const __grid_constant__ GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  gemm_mainloop<Grouped<true>>(prm, smem_raw);
}
__global__ void __launch_bounds__(NUM_THREADS, 1) grouped_gemm_tn_kernel(const __grid_constant__ GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  gemm_mainloop<GroupedTN>(prm, smem_raw);
}

// ---- the K-major rows mode on CTA pairs ---------------------------------------------------------------------------
// Same tile schedule (a tile is 256 rows of one group x 256 accumulator columns) and the same parameters; each CTA of
// the pair loads 128 rows of the A block and half of an accumulator's rows of B.  A tile has one accumulator or, in the
// wide form, two (see gemm_pair.cuh); grouped_width chooses.
namespace g2 = bshmem::gemm2;

constexpr int kTableGroups = 64;

template <bool kGatedEpi, bool kWideTile>
struct GroupedPair : g2::PolicyDefaults {
  using Params = GroupedParams;
  using Base = Grouped<kGatedEpi>;
  static constexpr bool kGated = kGatedEpi, kWide = kWideTile, kVarCols = true;
  __device__ static __forceinline__ int acc_cols(const Params& p, int a) { return p.core.acc_cols[a]; }
  __device__ static __forceinline__ int tile_cols(const Params& p) { return p.core.acc_cols[0] + (kWide ? p.core.acc_cols[1] : 0); }
  __device__ static __forceinline__ uint32_t stage_tx(const Params& p) { return g2::A_STAGE_BYTES + (uint32_t)tile_cols(p) / 2 * g2::BK_BYTES; }
  __device__ static __forceinline__ void load_b(const Params& p, const CUtensorMap*, uint32_t b_smem, uint32_t bar, int kb, int b_row, int, int, int) {
    ptx::tma_load_2d(b_smem, &p.map_b2, bar, kb * g2::BK, b_row);
  }
  __device__ static __forceinline__ const CoreParams& core(const Params& p) { return p.core; }
  __device__ static __forceinline__ const CUtensorMap* map_a(const Params& p) { return &p.map_a; }
  __device__ static __forceinline__ const CUtensorMap* map_b(const Params& p) { return &p.map_b; }
  // First tile of every group, in shared memory: walking the groups' counts in global memory took every role of the CTA
  // 1.5 us per tile with 64 groups.
  static constexpr bool kTileTable = true;
  __device__ static __forceinline__ int* tile_starts() {
    __shared__ int starts[kTableGroups + 1];
    return starts;
  }
  __device__ static __forceinline__ int group_blocks(const Params& p, int g) { return (Base::group_rows(p, g) + g2::BM - 1) / g2::BM; }
  __device__ static __forceinline__ void fill_tile_table(const Params& p) {
    if (p.G > kTableGroups || threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    int before = 0;
    for (int g0 = 0; g0 < p.G; g0 += 32) {
      const int mine = g0 + lane < p.G ? group_blocks(p, g0 + lane) * p.core.num_n_blocks : 0;
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      if (g0 + lane < p.G) tile_starts()[g0 + lane] = before + incl - mine;
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) tile_starts()[p.G] = before;
  }
  __device__ static __forceinline__ int num_tiles(const Params& p) { return p.G > kTableGroups ? Base::num_tiles(p) : tile_starts()[p.G]; }
  __device__ static __forceinline__ void tile_coords(const Params& p, int tile, int* m_blk, int* n_blk) {
    if (p.G > kTableGroups) return Base::tile_coords(p, tile, m_blk, n_blk);
    const int* starts = tile_starts();
    int g = 0, end = p.G;                 // starts[g] <= tile < starts[end]; an empty group starts where the next one does
    while (end - g > 1) {
      const int mid = (g + end) >> 1;
      if (starts[mid] <= tile) g = mid; else end = mid;
    }
    Base::coords_in_group(p, g, (starts[g + 1] - starts[g]) / p.core.num_n_blocks, tile - starts[g], m_blk, n_blk);
  }
  __device__ static __forceinline__ int a_row(const Params&, int m_blk) { return m_blk * g2::BM; }
  __device__ static __forceinline__ int b_row(const Params& p, int m_blk, int n_blk) {
    return (m_blk / p.a_blocks_per_group) * p.b_rows_per_group + n_blk * tile_cols(p);
  }
  // runs in the producer lane of BOTH CTAs: each loads its own half of the block
  __device__ static __forceinline__ bool a_ready(const Params& p, int, Guard& g) {
    for (int s = 0; s < p.P; ++s)
      if (!wait_ge<true>(p.arrive + s, (unsigned long long)p.expected[s], g, g2::ERR_PEER_SIGNAL)) return false;
    if (p.P) ptx::fence_proxy_async_all();   // peer stores (generic proxy) before the TMA reads
    return true;
  }
  // whether row `row` of C belongs to its group's rows (those behind them are scratch inside the group's own region)
  __device__ static __forceinline__ bool live(const Params& p, int row) {
    const int per = p.a_blocks_per_group * g2::BM, g = row / per;
    return row - g * per < Base::group_rows(p, g);
  }
  __device__ static __forceinline__ void out_target(const Params& p, int row, int col, const CUtensorMap** map, int* x, int* y) {
    *map = live(p, row) ? &p.map_c : nullptr;        // 32 rows: none of them is the group's, nothing to write
    *x = col;
    *y = row;
  }
};

// Training forward of the gated MLP: C keeps the interleaved gate / up pre-activations for the backward pass, and the
// activations silu(gate) * up are written in the same epilogue, from the rounded values that C holds (a pass of its own
// over C reads 2 and writes 1 of the 3 x 940 MB at 32768 rows x 14336: 440 us).
template <bool kWideTile>
struct GroupedPairAct : GroupedPair<false, kWideTile> {
  using Params = GroupedParams;
  static constexpr bool kStoreAct = true;
  // a lane owns a row: 64 consecutive bytes
  __device__ static __forceinline__ void store_act(const Params& p, int row, int col, const float (&f)[64]) {
    if (!GroupedPairAct::live(p, row)) return;
    uint4* dst = reinterpret_cast<uint4*>(p.act + row * p.ld_act + col / 2);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float h[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float gate = __bfloat162float(__float2bfloat16_rn(f[j * 8 + 2 * q + e])), up = __bfloat162float(__float2bfloat16_rn(f[32 + j * 8 + 2 * q + e]));
          h[e] = gate / (1.f + __expf(-gate)) * up;
        }
        w[q] = pack_bf16(h[0], h[1]);
      }
      dst[j] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
};

// Backward through the activations: the accumulator is d_h = d_y · W2; the epilogue reads the saved pre-activations and
// writes the gradients of the gate / up pre-activations, so that d_h never goes to memory (written and read again it was
// 1.9 of the 4.7 GB that the separate pass moved in 700 us).
struct GroupedPairSwigluBwd : GroupedPair<false, false> {
  static constexpr bool kSwigluBwd = true;
  __device__ static __forceinline__ void swiglu_grad(const Params& p, int row, int col, const float (&d)[32], float (&o)[64]) {
    const uint4* src = reinterpret_cast<const uint4*>(p.gu + row * p.ld_gu + 2 * col);
    const bool used = live(p, row);
    uint4 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = used ? src[j] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&v[j]);
      const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&v[4 + j]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 gf = __bfloat1622float2(gh[q]), uf = __bfloat1622float2(uh[q]);
        const float dx = __bfloat162float(__float2bfloat16_rn(d[j * 8 + 2 * q])), dy = __bfloat162float(__float2bfloat16_rn(d[j * 8 + 2 * q + 1]));
        const float sx = 1.f / (1.f + __expf(-gf.x)), sy = 1.f / (1.f + __expf(-gf.y));
        // d silu(g)/dg = s * (1 + g * (1 - s))
        o[j * 8 + 2 * q] = dx * uf.x * sx * (1.f + gf.x * (1.f - sx));
        o[j * 8 + 2 * q + 1] = dy * uf.y * sy * (1.f + gf.y * (1.f - sy));
        o[32 + j * 8 + 2 * q] = dx * (gf.x * sx);
        o[32 + j * 8 + 2 * q + 1] = dy * (gf.y * sy);
      }
    }
  }
};

// Weight-gradient flavour on CTA pairs: both operands MN-major (token-major activations as they are), ragged
// reduction over the group's tokens.  Per CTA and stage, each operand is two 64-wide MN blocks of 64 tokens (8 KiB per
// block, 128-byte swizzle), i.e. the CTA's 128 of the tile's 256 rows / columns.  One accumulator has always 256 columns here (128
// would load as much), fixed at compile time: with a width of its own this form took 2 to 6 % longer (8 groups of 2048 x 4096, 4096
// tokens: 462 us against 446).
template <bool kWideTile>
struct GroupedPairTN : GroupedPair<false, kWideTile> {
  using Params = GroupedParams;
  static constexpr bool kVarCols = kWideTile;
  __device__ static __forceinline__ int acc_cols(const Params& p, int a) { return kWideTile ? p.core.acc_cols[a] : g2::BN; }
  __device__ static __forceinline__ int tile_cols(const Params& p) { return kWideTile ? p.core.acc_cols[0] + p.core.acc_cols[1] : g2::BN; }
  static constexpr uint32_t kIdesc = ptx::umma_idesc_mn_major(1, 1, g2::BM, g2::BN);
  static constexpr uint32_t kBlock = 64 * g2::BK_BYTES;         // one 64 (MN) x 64 (tokens) block: 8 KiB
  static constexpr uint32_t kKStepA = 2048, kKStepB = 2048;     // one MMA consumes 16 tokens = two swizzle atoms
  __device__ static __forceinline__ uint64_t desc_a0(uint32_t a0) { return ptx::umma_desc_sw128_ex(a0, kBlock, 1024); }
  __device__ static __forceinline__ uint64_t desc_b0(uint32_t b0) { return ptx::umma_desc_sw128_ex(b0, kBlock, 1024); }
  __device__ static __forceinline__ int num_kb(const Params& p, int m_blk) {
    const int n = (p.klen[m_blk / p.a_blocks_per_group] + 63) / 64;
    return n < 1 ? 1 : n;     // an empty group still runs one (all-zero) k-block so that C becomes 0
  }
  __device__ static __forceinline__ bool a_ready(const Params&, int, Guard&) { return true; }
  // every row of a gradient is live (asking costs 8 % where a tile has one or two k-blocks)
  __device__ static __forceinline__ void out_target(const Params& p, int row, int col, const CUtensorMap** map, int* x, int* y) {
    *map = &p.map_c;
    *x = col;
    *y = row;
  }
  __device__ static __forceinline__ void load_stage(const Params& p, const CUtensorMap* ma, const CUtensorMap* mb, uint32_t a_smem,
                                                    uint32_t b_smem, uint32_t bar, int kb, int, int, int m_blk, int n_blk, int rank) {
    const int g = m_blk / p.a_blocks_per_group;
    const int tok = g * p.k_rows_per_group + kb * 64;
    const int m0 = (m_blk - g * p.a_blocks_per_group) * g2::BM + rank * g2::CTA_M;
    load_columns(p, ma, a_smem, bar, m0, tok);
    load_columns(p, mb, b_smem, bar, n_blk * GroupedPairTN::tile_cols(p) + rank * (acc_cols(p, 0) / 2), tok);
  }
  // the second accumulator has 256 columns, or 128: the CTA's 64 are then loaded together with the 64 next to them
  __device__ static __forceinline__ void load_b(const Params& p, const CUtensorMap* mb, uint32_t b_smem, uint32_t bar, int kb, int, int m_blk,
                                                int n_blk, int rank) {
    const int tok = m_blk / p.a_blocks_per_group * p.k_rows_per_group + kb * 64;
    load_columns(p, mb, b_smem, bar, n_blk * GroupedPairTN::tile_cols(p) + p.core.acc_cols[0] + rank * (p.core.acc_cols[1] / 2), tok);
  }
  __device__ static __forceinline__ uint32_t stage_tx(const Params&) { return kWideTile ? g2::WIDE_STAGE_BYTES : g2::STAGE_BYTES; }
  __device__ static __forceinline__ void load_columns(const Params& p, const CUtensorMap* map, uint32_t smem, uint32_t bar, int col, int tok) {
    if (p.tn3d) return ptx::tma_load_3d(smem, map, bar, 0, tok, col / 64);       // one 16 KiB copy: {64, 64 tokens, 2 column blocks}
    ptx::tma_load_2d(smem, map, bar, col, tok);
    ptx::tma_load_2d(smem + kBlock, map, bar, col + 64, tok);
  }
};

template <bool kWide>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(g2::NUM_THREADS, 1) grouped_gemm_pair_kernel(const __grid_constant__ GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  g2::gemm_mainloop<GroupedPair<false, kWide>>(prm, smem_raw);
}
template <bool kWide>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(g2::NUM_THREADS, 1) grouped_gemm_pair_gated_kernel(const __grid_constant__ GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  g2::gemm_mainloop<GroupedPair<true, kWide>>(prm, smem_raw);
}
template <bool kWide>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(g2::NUM_THREADS, 1) grouped_gemm_pair_act_kernel(const __grid_constant__ GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  g2::gemm_mainloop<GroupedPairAct<kWide>>(prm, smem_raw);
}
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(g2::NUM_THREADS, 1) grouped_gemm_pair_swiglu_bwd_kernel(const __grid_constant__ GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  g2::gemm_mainloop<GroupedPairSwigluBwd>(prm, smem_raw);
}
template <bool kWide>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(g2::NUM_THREADS, 1) grouped_gemm_pair_tn_kernel(const __grid_constant__ GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  g2::gemm_mainloop<GroupedPairTN<kWide>>(prm, smem_raw);
}
using PairKernel = void (*)(GroupedParams);
enum PairForm { ROWS_PLAIN, ROWS_GATED, ROWS_ACT, ROWS_SWIGLU_BWD, PAIR_TN };
// [form][wide]
constexpr PairKernel kPairKernels[][2] = {{grouped_gemm_pair_kernel<false>, grouped_gemm_pair_kernel<true>},
                                          {grouped_gemm_pair_gated_kernel<false>, grouped_gemm_pair_gated_kernel<true>},
                                          {grouped_gemm_pair_act_kernel<false>, grouped_gemm_pair_act_kernel<true>},
                                          {grouped_gemm_pair_swiglu_bwd_kernel, nullptr},
                                          {grouped_gemm_pair_tn_kernel<false>, grouped_gemm_pair_tn_kernel<true>}};

// Few rows per group (decode): weight-streaming tiles, see gemm_skinny.cuh.
template <bool kGated>
__global__ void __launch_bounds__(skinny::NUM_THREADS) grouped_gemm_few_kernel(const __grid_constant__ skinny::GroupedParams prm) {
  extern __shared__ uint8_t smem_raw[];
  skinny::grouped_body<kGated>(prm, smem_raw);
}

// Zero the token rows [count_g, next multiple of 64) — rows [0, 64) of an empty group — of every group of up to four
// [G][cap][cols] bf16 buffers.
struct PadBuffers {
  __nv_bfloat16* buf[4];
  int cols[4];
};
__global__ void zero_pad_rows_kernel(PadBuffers pb, const int* counts, int cap) {
  ptx::grid_dependency_wait();
  const int g = blockIdx.y;
  const int c = __ldcg(counts + g);
  int end = c == 0 ? 64 : (c + 63) / 64 * 64;      // an empty group still feeds one (all-zero) block to the GEMM
  if (end > cap) end = cap;
  const int cols = pb.cols[blockIdx.z];
  const int vec_per_row = cols / 8;
  const long long n = (long long)(end - c) * vec_per_row;
  uint4* base = reinterpret_cast<uint4*>(pb.buf[blockIdx.z] + ((size_t)g * cap + c) * cols);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    base[i] = make_uint4(0, 0, 0, 0);
}

int* g_err_dev[64] = {};
int g_sms[64] = {};
int g_pairs[64] = {};

int ensure(int dev) {
  if (g_err_dev[dev]) return 0;
  BSHMEM_CUDA_TRY(cudaMalloc(&g_err_dev[dev], sizeof(int)));
  BSHMEM_CUDA_TRY(cudaMemset(g_err_dev[dev], 0, sizeof(int)));
  BSHMEM_CUDA_TRY(cudaDeviceGetAttribute(&g_sms[dev], cudaDevAttrMultiProcessorCount, dev));
  BSHMEM_CUDA_TRY(cudaFuncSetAttribute(grouped_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
  BSHMEM_CUDA_TRY(cudaFuncSetAttribute(grouped_gemm_gated_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
  BSHMEM_CUDA_TRY(cudaFuncSetAttribute(grouped_gemm_tn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
  for (auto& form : kPairKernels)
    for (PairKernel k : form)
      if (k) BSHMEM_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g2::SMEM_BYTES));
  BSHMEM_CUDA_TRY(cudaFuncSetAttribute(grouped_gemm_few_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)skinny::SMEM_FULL));
  BSHMEM_CUDA_TRY(cudaFuncSetAttribute(grouped_gemm_few_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)skinny::SMEM_FULL));
  g_pairs[dev] = g2::max_resident_pairs(kPairKernels[ROWS_PLAIN][0], g_sms[dev]);
  return 0;
}

// Widths for a launch on CTA pairs (plan_width).  The host knows the row blocks exactly where all groups have `rows` rows; with
// counts on the device (`counted`) they are an estimate (group_rows).  In the wide form the epilogue of one accumulator delays that of the other, and the tensor
// cores wait for both: with the activations in it, some 8000 cycles per tile (32768 x 28672 by 512 columns, 4096 deep: 6.48 ms, by
// 256: 6.07; 8192 x 7168, 8192 deep, where 448 columns save half a wave: 0.74 against 0.77), with their derivative more
// (32768 x 14336, 4096 deep: 3.86 against 3.34 ms; 8192 x 3584, 8192 deep: 477 against 444 us).  Groups of one row block stream
// weights and gain nothing (training step of 1240 tokens, 64 experts of 1024, hidden 2048: 779 us, 791 with wide tiles).
// The gated form delays by less, which shows with counted groups: sustained, by 256 and by 512 columns, 8 groups of 750 rows, 8192 columns,
// 2048 deep 180 and 190 us, of 1366 rows 323 and 333, of 2250 rows 485 and 477; 28672 columns, 4096 deep, 750 rows 1263 and 1225, 1931 rows
// 2894 and 2850.  4000 cycles put the line near 2500 deep.
// In the weight gradients wide tiles pay at shorter reductions than in the plain product: 750 tokens, 8 groups of 2048 x 4096 102.6 and 94.3
// us, 64 of 2048 x 2048 437 and 373, one of 4096 x 3584 25.2 and 24.2; 375 tokens 62.4 and 62.4, 251 and 234, 16.6 and 16.4.  They are
// planned as if they were 256 deeper, which puts the line near 600.
g2::Width grouped_width(PairForm form, int G, int rows, bool counted, int N, int K, int pairs) {
  return g2::plan_width(G * ((rows + BM - 1LL) / BM), N, form == PAIR_TN ? K + 256 : K, pairs, form == ROWS_GATED || form == PAIR_TN ? 128 : 64, form == PAIR_TN, !counted,
                        form == ROWS_SWIGLU_BWD || (counted && rows <= BM) ? BN : 2 * BN, form == ROWS_ACT ? 8000 : form == ROWS_GATED && counted ? 4000 : 0);
}

// A launch of the CTA-pair kernels that may overlap the tail of the stream's previous kernel.
int launch_pairs(PairKernel kernel, const GroupedParams& p, int pairs, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pairs));
  cfg.blockDim = dim3(g2::NUM_THREADS);
  cfg.dynamicSmemBytes = g2::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BSHMEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p));
  return 0;
}

}  // namespace

extern "C" {

const char* bshmem_moe_gemm_last_error() { return host::last_error().c_str(); }

// Grouped GEMM.  A: [G * a_rows_per_group, K] (lda), B: [G * b_rows_per_group, K] (ldb), C: [G * a_rows_per_group, N_out] (ldc).
//   rows_dev   per-group valid row counts on the device (`fixed_rows`: about how many they are, 0 → not known; any counts are right), or
//              null → every group has `fixed_rows` rows
//   klen_dev   per-group reduction lengths on the device, or null → K
//   gated      1: accumulator columns are interleaved gate/up, C gets N/2 columns of silu(gate)*up
//   arrive/expected/P  optional arrival words to wait for before the first load (P = 0: none)
static int grouped_gemm_rows(PairForm form, const void* A, const void* B, void* C, int G, int a_rows_per_group, int b_rows_per_group, int N,
                             int K, int lda, int ldb, int ldc, const int* rows_dev, int fixed_rows, const int* klen_dev, const void* arrive,
                             const int* expected, int P, void* stream, int timeout_ms, int max_ctas, void* act, int ld_act, const void* gu,
                             int ld_gu) {
  if (G < 1 || a_rows_per_group % BM || N % BN || K % 8 || lda % 8 || ldb % 8 || ldc % 8) {
    host::last_error() = "grouped gemm: needs rows-per-group % 256 == 0, N % 256 == 0, K and leading dimensions % 8 == 0";
    return 1;
  }
  int dev = 0;
  BSHMEM_CUDA_TRY(cudaGetDevice(&dev));
  int rc = ensure(dev);
  if (rc) return rc;
  GroupedParams p;
  memset(&p, 0, sizeof(p));
  p.core.M = G * a_rows_per_group; p.core.N = N; p.core.K = K;
  p.core.num_m_blocks = p.core.M / BM; p.core.num_n_blocks = N / BN;
  p.core.group_m = 16;
  p.core.timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 4000) * 1000000ull;
  p.core.err = g_err_dev[dev];
  p.rows = rows_dev; p.klen = klen_dev; p.G = G; p.fixed_rows = fixed_rows > 0 ? fixed_rows : a_rows_per_group;
  p.a_blocks_per_group = a_rows_per_group / BM;
  p.b_rows_per_group = b_rows_per_group;
  p.group_m = 16;
  p.P = P; p.arrive = static_cast<const unsigned long long*>(arrive); p.expected = expected;
  // K-major rows mode with a uniform reduction length: CTA pairs; a ragged reduction length (legacy weight-gradient
  // form on transposed copies) stays on the single-CTA loop
  const bool pair = klen_dev == nullptr && g_pairs[dev] > 0, gated = form == ROWS_GATED;
  if (!pair && (form == ROWS_ACT || form == ROWS_SWIGLU_BWD)) { host::last_error() = "grouped gemm: this form needs CTA pairs"; return 1; }
  p.act = static_cast<__nv_bfloat16*>(act); p.ld_act = ld_act;
  p.gu = static_cast<const __nv_bfloat16*>(gu); p.ld_gu = ld_gu;
  int pairs = g_pairs[dev];
  if (max_ctas > 1 && max_ctas / 2 < pairs) pairs = max_ctas / 2;
  const g2::Width w = pair ? grouped_width(form, G, rows_dev ? g2::group_rows(a_rows_per_group, fixed_rows) : p.fixed_rows, rows_dev != nullptr, N, K, pairs) : g2::Width{{BN, 0}};
  if (pair) {
    p.core.acc_cols[0] = w.cols[0]; p.core.acc_cols[1] = w.cols[1];
    p.core.num_n_blocks = (N + w.cols[0] + w.cols[1] - 1) / (w.cols[0] + w.cols[1]);
  }
  const int box_rows_a = pair ? g2::CTA_M : BM, box_rows_b = pair ? w.cols[0] / 2 : BN;
  rc = host::make_tmap_2d(&p.map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, (uint64_t)G * a_rows_per_group, K, lda, box_rows_a, 64);
  if (rc) return rc;
  rc = host::make_tmap_2d(&p.map_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, B, (uint64_t)G * b_rows_per_group, K, ldb, box_rows_b, 64);
  if (rc) return rc;
  if (w.cols[1]) rc = host::make_tmap_2d(&p.map_b2, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, B, (uint64_t)G * b_rows_per_group, K, ldb, w.cols[1] / 2, 64);
  if (rc) return rc;
  rc = host::make_tmap_2d(&p.map_c, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, C, (uint64_t)G * a_rows_per_group,
                          form == ROWS_GATED ? N / 2 : form == ROWS_SWIGLU_BWD ? 2 * N : N, ldc, 32, EPI_COLS);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (pair) {
    return launch_pairs(kPairKernels[form][w.cols[1] ? 1 : 0], p, pairs, st);
  } else {
    int ctas = g_sms[dev];
    if (max_ctas > 0 && max_ctas < ctas) ctas = max_ctas;
    if (gated) grouped_gemm_gated_kernel<<<ctas, NUM_THREADS, SMEM_BYTES, st>>>(p);
    else grouped_gemm_kernel<<<ctas, NUM_THREADS, SMEM_BYTES, st>>>(p);
  }
  BSHMEM_CUDA_TRY(cudaGetLastError());
  return 0;
}

int bshmem_moe_grouped_gemm(const void* A, const void* B, void* C, int G, int a_rows_per_group, int b_rows_per_group, int N, int K,
                            int lda, int ldb, int ldc, const int* rows_dev, int fixed_rows, const int* klen_dev, int gated,
                            const void* arrive, const int* expected, int P, void* stream, int timeout_ms, int max_ctas) {
  return grouped_gemm_rows(gated ? ROWS_GATED : ROWS_PLAIN, A, B, C, G, a_rows_per_group, b_rows_per_group, N, K, lda, ldb, ldc, rows_dev,
                           fixed_rows, klen_dev, arrive, expected, P, stream, timeout_ms, max_ctas, nullptr, 0, nullptr, 0);
}

// Training forward of the gated MLP: C [G * a_rows_per_group, N] keeps the interleaved gate / up pre-activations, act
// [.., N / 2] (ld_act % 8 == 0) gets silu(gate) * up.
int bshmem_moe_grouped_gemm_act(const void* A, const void* B, void* C, void* act, int G, int a_rows_per_group, int N, int K, int lda, int ldb,
                                int ldc, int ld_act, const int* rows_dev, const void* arrive, const int* expected, int P, void* stream,
                                int timeout_ms, int about_rows) {
  if (!act || ld_act % 8) { host::last_error() = "grouped gemm (act): needs an activation buffer, leading dimension % 8 == 0"; return 1; }
  return grouped_gemm_rows(ROWS_ACT, A, B, C, G, a_rows_per_group, N, N, K, lda, ldb, ldc, rows_dev, rows_dev ? about_rows : 0, nullptr, arrive, expected, P, stream,
                           timeout_ms, 0, act, ld_act, nullptr, 0);
}

// Backward of the same: d_h = A · B^T (N columns) goes through SwiGLU's derivative at the saved pre-activations gu
// [.., 2 N] (ld_gu % 8 == 0); C [.., 2 N] gets their gradients.
int bshmem_moe_grouped_gemm_swiglu_bwd(const void* A, const void* B, const void* gu, void* C, int G, int a_rows_per_group, int N, int K,
                                       int lda, int ldb, int ld_gu, int ldc, const int* rows_dev, const void* arrive, const int* expected,
                                       int P, void* stream, int timeout_ms, int about_rows) {
  if (!gu || ld_gu % 8) { host::last_error() = "grouped gemm (swiglu): needs the pre-activations, leading dimension % 8 == 0"; return 1; }
  return grouped_gemm_rows(ROWS_SWIGLU_BWD, A, B, C, G, a_rows_per_group, N, N, K, lda, ldb, ldc, rows_dev, rows_dev ? about_rows : 0, nullptr, arrive, expected, P,
                           stream, timeout_ms, 0, nullptr, 0, gu, ld_gu);
}

// The same product for few rows per group (up to about 128; more are taken in chunks, reading the weights again).
// max_rows and max_active are the largest group and the number of groups with rows as far as the host knows them (the tokens
// and the token-expert entries of a decode step); they choose chunk, split and grid, and the product is right for any counts
// on the device: larger groups are taken in more chunks, and more tiles than clusters are not split.  Up to 64 groups, a_rows_per_group and N multiples of 256; rows of
// C beyond a group's count are not written.
// us, 8 groups, N x K = 28672 x 4096 gated: 8 rows each 285 against 380 for the 256-row tiles (weights at the measured copy
// rate: 288), 64 rows 315 / 375, 100 rows 325 / 373, 128 rows 410 / 380 (some groups have more than the chunk of 128 rows
// then and read their weights twice).
int bshmem_moe_grouped_gemm_few(const void* A, const void* B, void* C, int G, int a_rows_per_group, int N, int K, int lda, int ldb, int ldc,
                                const int* rows_dev, int max_rows, int max_active, int gated, const void* arrive, const int* expected, int P,
                                void* stream, int timeout_ms) {
  if (G < 1 || G > skinny::MAX_GROUPS || a_rows_per_group < BM || a_rows_per_group % BM || N % BN || K % 8 || lda % 8 || ldb % 8 || ldc % 8 || !rows_dev || max_rows < 1) {
    host::last_error() = "grouped gemm (few rows): needs 1 to 64 groups, rows-per-group % 256 == 0, N % 256 == 0, K and leading dimensions % 8 == 0";
    return 1;
  }
  int dev = 0;
  BSHMEM_CUDA_TRY(cudaGetDevice(&dev));
  int rc = ensure(dev);
  if (rc) return rc;
  skinny::GroupedParams p;
  p.out = static_cast<__nv_bfloat16*>(C);
  p.ldo = ldc;
  p.rows = rows_dev;
  p.G = G; p.cap = a_rows_per_group; p.N = N; p.K = K;
  if (max_rows > a_rows_per_group) max_rows = a_rows_per_group;
  p.nt_cap = max_rows >= 128 ? 128 : (max_rows + 15) / 16 * 16;
  // Two CTAs per SM.  An SM does not get more than about 45 GB/s out of HBM however many stages it keeps in flight, so
  // where the tiles cannot occupy the chip (two groups with one row, N x K = 4096 x 14336: 64 tiles, 2.1 TB/s) each is
  // split over a cluster while at least eight k-blocks remain per CTA.
  if (max_active < 1 || max_active > G) max_active = G;
  const long long tiles = (long long)max_active * (N / skinny::ROWS) * ((max_rows + p.nt_cap - 1) / p.nt_cap);
  const int kb = (K + skinny::BK - 1) / skinny::BK;
  p.split = 1;
  while (p.split < 8 && tiles * p.split <= g_sms[dev] && kb >= 16 * p.split) p.split *= 2;
  const uint32_t fixed = 1024 + skinny::GROUP_CTRL_BYTES + (gated ? skinny::GROUP_XCHG_BYTES : 0);
  p.ring_bytes = (skinny::SMEM_HALF - fixed) & ~1023u;          // also holds a split tile's 512 bytes per token
  p.xbox = max_rows <= 16 ? 16 : 32;     // a copy of 16 rows takes the copy unit as long as one of 32
  p.tmem_cols = 32;
  while (p.tmem_cols < 2u * p.nt_cap) p.tmem_cols *= 2;
  p.P = P; p.arrive = static_cast<const unsigned long long*>(arrive); p.expected = expected;
  p.timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 4000) * 1000000ull;
  p.err = g_err_dev[dev];
  rc = host::make_tmap_2d(&p.map_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, B, (uint64_t)G * N, K, ldb, skinny::ROWS, skinny::BK);
  if (rc) return rc;
  rc = host::make_tmap_2d(&p.map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, (uint64_t)G * a_rows_per_group, K, lda, p.xbox, skinny::BK);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.split > 1 ? tiles * p.split : 2 * g_sms[dev]));
  cfg.blockDim = dim3(skinny::NUM_THREADS);
  cfg.dynamicSmemBytes = p.ring_bytes + fixed;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.split; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.split > 1 ? 2 : 1;
  BSHMEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, gated ? grouped_gemm_few_kernel<true> : grouped_gemm_few_kernel<false>, p));
  return 0;
}

// Weight-gradient GEMM on token-major operands: C_g[M, N] = A_g^T · B_g for every group.
//   A: [G * cap, M] (lda), B: [G * cap, N] (ldb), C: [G * M, N] (ldc); the number of tokens of group g is
//   klen_dev[g] (<= cap; about_len: about how many they are, 0: not known).  Token rows [klen, next multiple of 64) must be zero in A and B.
int bshmem_moe_grouped_gemm_tn(const void* A, const void* B, void* C, int G, int cap, int M, int N, int lda, int ldb, int ldc,
                               const int* klen_dev, void* stream, int timeout_ms, int max_ctas, int about_len) {
  if (G < 1 || M % BM || N % BN || cap % 64 || lda % 8 || ldb % 8 || ldc % 8 || !klen_dev) {
    host::last_error() = "grouped gemm (transposed operands): needs M % 256 == 0, N % 256 == 0, capacity % 64 == 0, leading dimensions % 8 == 0";
    return 1;
  }
  int dev = 0;
  BSHMEM_CUDA_TRY(cudaGetDevice(&dev));
  int rc = ensure(dev);
  if (rc) return rc;
  GroupedParams p;
  memset(&p, 0, sizeof(p));
  p.core.M = G * M; p.core.N = N; p.core.K = cap;
  p.core.num_m_blocks = p.core.M / BM; p.core.num_n_blocks = N / BN;
  p.core.group_m = 16;
  p.core.timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 4000) * 1000000ull;
  p.core.err = g_err_dev[dev];
  p.rows = nullptr; p.klen = klen_dev; p.G = G; p.fixed_rows = M;
  p.a_blocks_per_group = M / BM;
  p.k_rows_per_group = cap;
  p.group_m = 16;
  // CTA pairs (a CTA then loads two 64-wide column blocks per operand and stage instead of four); the single-CTA loop
  // only if the device cannot hold a pair of this kernel
  const bool pair = g_pairs[dev] > 0;
  const uint32_t blocks = pair ? 2 : 4;
  int pairs = g_pairs[dev];
  if (max_ctas > 1 && max_ctas / 2 < pairs) pairs = max_ctas / 2;
  // the reduction is a group's tokens
  g2::Width w = pair ? grouped_width(PAIR_TN, G, M, false, N, g2::group_rows(cap, about_len), pairs) : g2::Width{{BN, 0}};
  if (!w.cols[1]) w.cols[0] = BN;      // what the form with one accumulator has
  if (pair) {
    p.core.acc_cols[0] = w.cols[0]; p.core.acc_cols[1] = w.cols[1];
    p.core.num_n_blocks = (N + w.cols[0] + w.cols[1] - 1) / (w.cols[0] + w.cols[1]);
  }
  // preferred: one 3-D copy per operand and stage; if the driver refuses that view, boxes of 64 MN-elements
  // (128 bytes, the swizzle span) by 64 tokens, one per column block
  static const bool no3d = getenv("B200SHMEM_TN_2D") != nullptr;
  p.tn3d = 0;
  if (!no3d && host::make_tmap_colblocks_3d(&p.map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, A, (uint64_t)G * cap, M, lda, 64, blocks) == 0 &&
      host::make_tmap_colblocks_3d(&p.map_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, B, (uint64_t)G * cap, N, ldb, 64, blocks) == 0)
    p.tn3d = 1;
  if (!p.tn3d) {
    rc = host::make_tmap_2d(&p.map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, (uint64_t)G * cap, M, lda, 64, 64);
    if (rc) return rc;
    rc = host::make_tmap_2d(&p.map_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, B, (uint64_t)G * cap, N, ldb, 64, 64);
    if (rc) return rc;
  }
  rc = host::make_tmap_2d(&p.map_c, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, C, (uint64_t)G * M, N, ldc, 32, EPI_COLS);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (pair) {
    return launch_pairs(kPairKernels[PAIR_TN][w.cols[1] ? 1 : 0], p, pairs, st);
  } else {
    int ctas = g_sms[dev];
    if (max_ctas > 0 && max_ctas < ctas) ctas = max_ctas;
    grouped_gemm_tn_kernel<<<ctas, NUM_THREADS, SMEM_BYTES, st>>>(p);
  }
  BSHMEM_CUDA_TRY(cudaGetLastError());
  return 0;
}

// Up to four [G][cap][cols] bf16 buffers (null: none), cols % 8 == 0: zero rows [counts[g], next multiple of 64) of every
// group.  One launch for all: four in a row took 12 us of a backward pass.
int bshmem_moe_zero_pad_rows(void* b0, int cols0, void* b1, int cols1, void* b2, int cols2, void* b3, int cols3, const int* counts_dev, int G,
                             int cap, void* stream) {
  PadBuffers pb;
  memset(&pb, 0, sizeof(pb));
  void* bufs[4] = {b0, b1, b2, b3};
  const int cols[4] = {cols0, cols1, cols2, cols3};
  int n = 0;
  for (int i = 0; i < 4; ++i) {
    if (!bufs[i]) continue;
    if (cols[i] % 8) { host::last_error() = "zero_pad_rows: cols % 8 != 0"; return 1; }
    pb.buf[n] = static_cast<__nv_bfloat16*>(bufs[i]);
    pb.cols[n++] = cols[i];
  }
  if (G < 1 || n == 0) { host::last_error() = "zero_pad_rows: nothing to do"; return 1; }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(8, (unsigned)G, (unsigned)n);
  cfg.blockDim = dim3(256);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BSHMEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, zero_pad_rows_kernel, pb, counts_dev, cap));
  return 0;
}

int bshmem_moe_gemm_error_site(int clear) {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || !g_err_dev[dev]) return 0;
  cudaMemcpy(&v, g_err_dev[dev], sizeof(int), cudaMemcpyDeviceToHost);
  if (clear && v) cudaMemset(g_err_dev[dev], 0, sizeof(int));
  return v;
}

int* bshmem_moe_gemm_error_word() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || ensure(dev)) return nullptr;
  return g_err_dev[dev];
}

}  // extern "C"
