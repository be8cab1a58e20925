// gemm_skinny.cuh — tcgen05 GEMM for few tokens on sm_100a:  C[M,N] = X[M,K] · W[N,K]^T with M up to 256.
//
// With few rows the product reads the weight matrix once and does little else, so the tile follows the weights: a tile
// is 128 weight rows (the M dimension of the MMA) times all tokens of the chunk (its N dimension, 16 to 256 in steps
// of 16), and the accumulator is the transposed result.  The 256x256 tiles of gemm_pair.cuh would give N / 256 tiles
// (32 for 8192 columns, on 148 SMs), multiply padding rows for 94 % of the time at M = 16 and put 32 KiB of token rows
// into every stage.
//
// What bounds it is the weight stream from HBM; what matters is bytes in flight on every SM.  Up to 64 tokens two CTAs
// share an SM, each with its own ring of 16 KiB weight blocks (5 or 6 stages, about 190 KiB in flight per SM).  Where
// N / 128 tiles do not fill the chip, a cluster of S = 2, 4 or 8 CTAs splits the reduction of a tile: each CTA sums its
// share of K in tensor memory, parks the fp32 partial tile in its shared memory, and after one cluster barrier every
// CTA adds the S partials of its share of the tokens (fixed order: reproducible bits) and writes bf16.  No workspace,
// no atomics, nothing to clear between calls.
//
//   warp 0      TMA producer: {128 weight rows, nt token rows} x 64 of K per stage, plain loads of local memory
//   warp 1      MMA issuer: tcgen05.mma.cta_group::1 M128 x N=nt x K16
//   warps 2-5   epilogue
// Producer and issuer are loops of their whole warp, one elected lane issues (see ptx::elect_one); from a lane in a branch of its own,
// us: 16 x 3584 x 8192 13.05 (now 12.81), 64 x 4096 x 4096 10.8 (10.5), 100 x 2048 x 2048 7.4 (7.0), 128 x 8192 x 8192 28.5 (27.8); the grouped
// form, 32 tokens on 8 experts of 14336: 452.5 (448.7).
// Every wait is bounded (see gemm_core.cuh).  The reference has no GEMM, hence no counterpart.
#pragma once
#include "gemm_pair.cuh"

namespace bshmem {
namespace skinny {

using gemm::Guard;
using gemm::mbar_wait;
using gemm::pack_bf16;
using gemm2::cluster_ctarank;
using gemm2::cluster_sync_all;
using gemm2::ld_cluster_f4;
using gemm2::mapa;
using gemm2::warp_wait;

constexpr int ROWS = 128;                          // weight rows of a tile
constexpr int BK = 64;                             // bf16 elements per k-block: one 128-byte swizzle atom
constexpr int MAX_TOKENS = 256;
constexpr int MAX_STAGES = 8;                     // of the dense form; the grouped form: MAX_GROUP_STAGES
constexpr int NUM_EPI_WARPS = 4;
constexpr int NUM_THREADS = 32 * (2 + NUM_EPI_WARPS);
constexpr uint32_t W_STAGE_BYTES = ROWS * BK * 2;  // 16 KiB
constexpr uint32_t CTRL_BYTES = 256;               // barriers, tensor-memory address, abort flag
// shared memory of a CTA: two CTAs per SM as long as a stage is small, else one
constexpr uint32_t SMEM_HALF = 112u << 10, SMEM_FULL = 227u << 10;

enum ErrSite : int { ERR_PRODUCER_EMPTY = 301, ERR_MMA_FULL = 302, ERR_EPI_FULL = 303 };

struct Params {
  CUtensorMap map_w, map_x;      // weights [N, K] or [K, N], tokens [M, K]: boxes {64, 128} or {64, 64}, and {64, nt}
  __nv_bfloat16* out;            // [M, N]
  long long ldo;
  int M, N, K;
  int nt;                        // tokens of the MMA: M rounded up to 16
  int stages;
  int split;                     // CTAs of a cluster that share a tile's reduction (1, 2, 4 or 8)
  int prefetch;                  // weight blocks a CTA prefetches into L2 (see prefetch_plan.h), at most `stages`
  uint32_t tmem_cols;
  unsigned long long timeout_ns;
  int* err;
};

__host__ __device__ constexpr uint32_t stage_bytes(int nt) { return W_STAGE_BYTES + (uint32_t)nt * BK * 2; }
__host__ __device__ constexpr uint32_t smem_bytes(int nt, int stages) { return stages * stage_bytes(nt) + CTRL_BYTES + 1024; }

__device__ __forceinline__ float ld_cluster_f1(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

struct Smem {
  uint32_t base, stage, ctrl;    // 1024-byte aligned base, bytes of a stage, control block
  uint8_t* gen;                  // generic pointer to the control block
  __device__ __forceinline__ uint32_t w(int s) const { return base + s * stage; }
  __device__ __forceinline__ uint32_t x(int s) const { return base + s * stage + W_STAGE_BYTES; }
  __device__ __forceinline__ uint32_t full(int s) const { return ctrl + 8 * s; }
  __device__ __forceinline__ uint32_t empty(int s) const { return ctrl + 8 * (MAX_STAGES + s); }
  __device__ __forceinline__ uint32_t acc_full() const { return ctrl + 8 * (2 * MAX_STAGES); }
  __device__ __forceinline__ uint32_t tmem_slot() const { return ctrl + 8 * (2 * MAX_STAGES + 1); }
  __device__ __forceinline__ volatile int* abort_flag() const { return reinterpret_cast<volatile int*>(gen + 8 * (2 * MAX_STAGES + 2)); }
};

}  // namespace skinny
}  // namespace bshmem

namespace bshmem {
namespace skinny {

// Sum of the S partial tiles over the tokens of this CTA: one warp per token, four weight rows per lane, kTok tokens at a
// time so that S * kTok loads of the other CTAs' shared memory are in flight (one after the other they cost M = 256,
// S = 8 more than the product itself).
template <int S>
__device__ __forceinline__ void add_partials(const Params& p, uint32_t base, int rank, int warp, int lane, int n0) {
  constexpr int kTok = 8 / S < 1 ? 1 : 8 / S, kStep = S * (NUM_THREADS / 32);
  uint32_t src[S];
#pragma unroll
  for (int q = 0; q < S; ++q) src[q] = mapa(base + lane * 16, q);
  for (int t0 = rank + warp * S; t0 < p.M; t0 += kTok * kStep) {
    float4 v[kTok][S];
#pragma unroll
    for (int u = 0; u < kTok; ++u)
#pragma unroll
      for (int q = 0; q < S; ++q)                    // past the last token: read the last one again, drop it below
        v[u][q] = ld_cluster_f4(src[q] + min(t0 + u * kStep, p.M - 1) * (ROWS * 4));
#pragma unroll
    for (int u = 0; u < kTok; ++u) {
      const int t = t0 + u * kStep;
#pragma unroll
      for (int q = 1; q < S; ++q) { v[u][0].x += v[u][q].x; v[u][0].y += v[u][q].y; v[u][0].z += v[u][q].z; v[u][0].w += v[u][q].w; }
      if (t >= p.M) continue;
      __nv_bfloat16* dst = p.out + (long long)t * p.ldo + n0 + lane * 4;
      const int left = p.N - n0 - lane * 4;           // columns from here on; what lies behind them is not ours
      if (left >= 4) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v[u][0].x, v[u][0].y), pack_bf16(v[u][0].z, v[u][0].w));
      } else {
        const float f[3] = {v[u][0].x, v[u][0].y, v[u][0].z};
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (j < left) dst[j] = __float2bfloat16_rn(f[j]);
      }
    }
  }
}

// One tile per cluster of p.split CTAs: grid = tiles * split.
// kWmn: the weights are stored [K][N] (the data gradient's operand): a stage is two 64-wide column blocks of 64 reduction
// rows, read through an MN-major descriptor.
template <bool kWmn>
__device__ __forceinline__ void body(const Params& p, uint8_t* smem_raw) {
  Smem L;
  {
    const uint32_t r = ptx::smem_u32(smem_raw);
    L.base = (r + 1023u) & ~1023u;
    L.stage = stage_bytes(p.nt);
    L.ctrl = L.base + p.stages * L.stage;
    L.gen = smem_raw + (L.ctrl - r);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = p.split;
  const int rank = split > 1 ? (int)cluster_ctarank() : 0;
  const int n0 = (int)(blockIdx.x / split) * ROWS;
  const int kb_all = (p.K + BK - 1) / BK;
  const int kb0 = kb_all * rank / split, kb1 = kb_all * (rank + 1) / split;
  Guard g{p.err, L.abort_flag(), p.timeout_ns};

  if (threadIdx.x == 0) {
    *L.abort_flag() = 0;
    for (int s = 0; s < p.stages; ++s) { ptx::mbar_init(L.full(s), 1); ptx::mbar_init(L.empty(s), 1); }
    ptx::mbar_init(L.acc_full(), 1);
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&p.map_w);
    ptx::prefetch_tensormap(&p.map_x);
  }
  if (warp == 1) {
    ptx::tmem_alloc(L.tmem_slot(), p.tmem_cols);
    ptx::tmem_relinquish();
  }
  // This CTA's weights start on their way to L2 while the previous kernel of the stream still runs.  They may not be read yet, it could
  // be writing them, but a prefetch reads nothing.
  if (warp == 2 && lane == 0)
    for (int kb = kb0; kb < min(kb1, kb0 + p.prefetch); ++kb) {
      if constexpr (kWmn) {
        ptx::tma_prefetch_2d(&p.map_w, n0, kb * BK);
        ptx::tma_prefetch_2d(&p.map_w, n0 + 64, kb * BK);
      } else {
        ptx::tma_prefetch_2d(&p.map_w, kb * BK, n0);
      }
    }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(L.tmem_slot()));
  // the set-up above overlaps the previous kernel of the stream; operands and output belong to it until it is done
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  bool ok = true;
  if (warp == 0) {
    const bool leader = ptx::elect_one();
    int s = 0; uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!warp_wait(L.empty(s), ph ^ 1, g, ERR_PRODUCER_EMPTY)) break;
      if (leader) {
        ptx::mbar_arrive_expect_tx(L.full(s), L.stage);
        if constexpr (kWmn) {
          ptx::tma_load_2d(L.w(s), &p.map_w, L.full(s), n0, kb * BK);
          ptx::tma_load_2d(L.w(s) + W_STAGE_BYTES / 2, &p.map_w, L.full(s), n0 + 64, kb * BK);
        } else {
          ptx::tma_load_2d(L.w(s), &p.map_w, L.full(s), kb * BK, n0);
        }
        ptx::tma_load_2d(L.x(s), &p.map_x, L.full(s), kb * BK, 0);
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    const bool leader = ptx::elect_one();
    int s = 0; uint32_t ph = 0;
    const uint32_t idesc = ptx::umma_idesc(1, 1, ROWS, (uint32_t)p.nt) | (kWmn ? 1u << 15 : 0u);
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!warp_wait(L.full(s), ph, g, ERR_MMA_FULL)) { ok = false; break; }
      ptx::tc_fence_after();
      if (leader) {
        const uint64_t dw = kWmn ? ptx::umma_desc_sw128_ex(L.w(s), W_STAGE_BYTES / 2, 1024) : ptx::umma_desc_sw128(L.w(s));
        const uint64_t dx = ptx::umma_desc_sw128(L.x(s));
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) ptx::umma_f16(tmem, dw + (kWmn ? 128 : 2) * k, dx + 2 * k, idesc, (kb > kb0 || k) ? 1u : 0u);
        ptx::umma_commit(L.empty(s));
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    if (ok && leader) ptx::umma_commit(L.acc_full());
  } else {
    ok = mbar_wait(L.acc_full(), 0, g, ERR_EPI_FULL);
    ptx::tc_fence_after();
    if (ok) {
      const int quarter = warp & 3;                  // tensor-memory lanes = weight rows 32 * quarter ..
      const int row = quarter * 32 + lane;
      const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16);
      if (split == 1) {
        __nv_bfloat16* out = p.out + n0 + row;
        const bool live = n0 + row < p.N;
        for (int c = 0; c < p.nt; c += 16) {
          uint32_t v[16];
          ptx::tmem_ld_32x32b_x16(taddr + c, v);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j)               // 32 lanes = 64 consecutive bytes of a token's row
            if (live && c + j < p.M) out[(long long)(c + j) * p.ldo] = __float2bfloat16_rn(__uint_as_float(v[j]));
        }
      } else {
        // partial tile as [token][weight row] floats over the (drained) stages: all loads have landed and all MMAs
        // have read them once the accumulator is complete
        const uint32_t dst = L.base + row * 4;
        for (int c = 0; c < p.nt; c += 16) {
          uint32_t v[16];
          ptx::tmem_ld_32x32b_x16(taddr + c, v);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + (c + j) * (ROWS * 4)), "r"(v[j]) : "memory");
        }
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (split > 1) {
    cluster_sync_all();
    // every CTA adds the partials of the tokens rank, rank + split, ...
    if (!*L.abort_flag() && n0 + lane * 4 < p.N) {
      if (split == 2) add_partials<2>(p, L.base, rank, warp, lane, n0);
      else if (split == 4) add_partials<4>(p, L.base, rank, warp, lane, n0);
      else add_partials<8>(p, L.base, rank, warp, lane, n0);
    }
    cluster_sync_all();                                  // nobody's shared memory goes away while it is being read
  }
  if (*L.abort_flag()) {
    // let copies and MMAs that are still in flight land before shared and tensor memory go away
    const unsigned long long t0 = ptx::globaltimer();
    while (ptx::globaltimer() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, p.tmem_cols);
  }
}

}  // namespace skinny
}  // namespace bshmem

// ---- grouped form: few tokens per group (the experts of a decode step) -----------------------------------------------
//   C_g[rows_g, N] = X_g[rows_g, K] · W_g[N, K]^T  for every group g, the row counts read on the device.
// Persistent CTAs over (group, chunk of up to 128 tokens, 128 weight rows); groups without rows cost nothing.  Two
// accumulators, so that the epilogue of a tile overlaps the loads and MMAs of the next.  The stage size follows the
// largest group of the call: 16 KiB of weights plus 128 bytes per token, as many stages as fit.
// Gated: the weight rows are 32 gate rows followed by the matching 32 up rows, i.e. alternating quarters of the tensor
// memory; the up warps hand their values to the gate warps through shared memory, 16 tokens at a time, and the gate warps
// write silu(gate) * up.
// Split (few active groups with few weight rows): as in the dense form, a cluster shares one tile and adds its parts
// through distributed shared memory; a CTA has no second tile then.  The counts on the device decide whether that holds: with
// more tiles than clusters the CTAs take whole tiles, each on its own.
namespace bshmem {
namespace skinny {

constexpr int MAX_GROUPS = 64, MAX_GROUP_STAGES = 12;
constexpr uint32_t GROUP_XCHG_BYTES = 2 * 2 * 16 * 32 * 4;             // two warp pairs x two buffers x 16 tokens x 32 columns
constexpr uint32_t GROUP_CTRL_BYTES = 8 * (2 * MAX_GROUP_STAGES + 6) + 16 + 4 * MAX_GROUPS;

struct GroupedParams {
  CUtensorMap map_w, map_x;      // weights [G * N, K] box {64, 128}; tokens [G * cap, K] box {64, xbox}
  __nv_bfloat16* out;            // [G * cap, N] or gated [G * cap, N / 2]
  long long ldo;
  const int* rows;
  int G, cap, N, K;
  int xbox;                      // token rows per TMA box: 16 or 32
  uint32_t ring_bytes;           // shared memory of the stages
  uint32_t tmem_cols;            // two accumulators
  int nt_cap;                    // tokens per chunk that the tensor memory holds (multiple of 16, at most 128)
  int split;                     // > 1: clusters of that many CTAs share the reduction of a tile while each has one at most
  int P;                         // arrival words to wait for before the first token load (0: none)
  const unsigned long long* arrive;
  const int* expected;
  unsigned long long timeout_ns;
  int* err;
};

enum GroupErrSite : int { ERR_G_PRODUCER_EMPTY = 311, ERR_G_MMA_FULL = 312, ERR_G_MMA_ACC = 313, ERR_G_EPI_FULL = 314, ERR_G_ARRIVE = 315 };

struct GroupedSmem {
  uint32_t base, ctrl;
  uint8_t* gen;
  __device__ __forceinline__ uint32_t full(int s) const { return ctrl + 8 * s; }
  __device__ __forceinline__ uint32_t empty(int s) const { return ctrl + 8 * (MAX_GROUP_STAGES + s); }
  __device__ __forceinline__ uint32_t acc_full(int a) const { return ctrl + 8 * (2 * MAX_GROUP_STAGES + a); }
  __device__ __forceinline__ uint32_t acc_empty(int a) const { return ctrl + 8 * (2 * MAX_GROUP_STAGES + 2 + a); }
  __device__ __forceinline__ uint32_t tmem_slot() const { return ctrl + 8 * (2 * MAX_GROUP_STAGES + 4); }
  __device__ __forceinline__ volatile int* abort_flag() const { return reinterpret_cast<volatile int*>(gen + 8 * (2 * MAX_GROUP_STAGES + 5)); }
  __device__ __forceinline__ int* rows() const { return reinterpret_cast<int*>(gen + 8 * (2 * MAX_GROUP_STAGES + 6)); }
};

// Walks the tiles first, first + step, ...: weight blocks fastest, then chunks, then groups.
struct GroupedTiles {
  const int* rows;
  int G, nb, chunk;              // groups, weight blocks per group, tokens per chunk
  int tile, step, g, base;       // base: index of the first tile of group g
  __device__ __forceinline__ bool next(int* group, int* n_blk, int* tok0, int* ntok) {
    for (; g < G; ++g) {
      const int r = rows[g], n = (r + chunk - 1) / chunk * nb;
      if (tile < base + n) {
        const int in = tile - base, c = in / nb;
        *group = g; *n_blk = in - c * nb; *tok0 = c * chunk; *ntok = min(chunk, r - c * chunk);
        tile += step;
        return true;
      }
      base += n;
    }
    return false;
  }
};

template <bool kGated>
__device__ __forceinline__ void grouped_body(const GroupedParams& p, uint8_t* smem_raw) {
  GroupedSmem L;
  uint32_t xchg;
  {
    const uint32_t r = ptx::smem_u32(smem_raw);
    L.base = (r + 1023u) & ~1023u;
    xchg = L.base + p.ring_bytes;
    L.ctrl = xchg + (kGated ? GROUP_XCHG_BYTES : 0);
    L.gen = smem_raw + (L.ctrl - r);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Guard g{p.err, L.abort_flag(), p.timeout_ns};
  if (threadIdx.x == 0) {
    *L.abort_flag() = 0;
    for (int s = 0; s < MAX_GROUP_STAGES; ++s) { ptx::mbar_init(L.full(s), 1); ptx::mbar_init(L.empty(s), 1); }
    for (int a = 0; a < 2; ++a) { ptx::mbar_init(L.acc_full(a), 1); ptx::mbar_init(L.acc_empty(a), NUM_EPI_WARPS); }
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&p.map_w);
    ptx::prefetch_tensormap(&p.map_x);
  }
  if (warp == 1) {
    ptx::tmem_alloc(L.tmem_slot(), p.tmem_cols);
    ptx::tmem_relinquish();
  }
  ptx::grid_dependency_wait();
  for (int i = threadIdx.x; i < p.G; i += NUM_THREADS) L.rows()[i] = __ldcg(p.rows + i);
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(L.tmem_slot()));
  int most = 1, tiles = 0;
  for (int i = lane; i < p.G; i += 32) {
    most = max(most, L.rows()[i]);
    tiles += (L.rows()[i] + p.nt_cap - 1) / p.nt_cap * (p.N / ROWS);
  }
  most = __reduce_max_sync(0xffffffffu, most);
  tiles = __reduce_add_sync(0xffffffffu, tiles);
  // A cluster has room for the parts of one tile.  The host chose the split from the counts it expected; where the real ones
  // make more tiles than there are clusters, every CTA of the grid (all read the same counts) walks whole tiles on its own.
  const int split = p.split > 1 && tiles <= (int)gridDim.x / p.split ? p.split : 1;
  const int nt_max = min((most + 15) / 16 * 16, p.nt_cap);
  const uint32_t stage = W_STAGE_BYTES + (uint32_t)((nt_max + p.xbox - 1) / p.xbox * p.xbox) * BK * 2;
  const int stages = min((int)(p.ring_bytes / stage), MAX_GROUP_STAGES);
  const int kb_all = (p.K + BK - 1) / BK;
  const int rank = split > 1 ? (int)cluster_ctarank() : 0;
  const int kb0 = kb_all * rank / split, kb1 = kb_all * (rank + 1) / split;
  GroupedTiles it{L.rows(), p.G, p.N / ROWS, p.nt_cap, (int)blockIdx.x / split, (int)gridDim.x / split, 0, 0};
  struct { int grp, n_blk, tok0, ntok; } split_tile = {0, 0, 0, 0};
  bool mine = false;                                 // split form: there is a tile for this cluster
  if (split > 1) {
    GroupedTiles probe = it;
    mine = probe.next(&split_tile.grp, &split_tile.n_blk, &split_tile.tok0, &split_tile.ntok);
  }
  int grp, n_blk, tok0, ntok;

  if (warp == 0) {
    const bool leader = ptx::elect_one();
    int s = 0; uint32_t ph = 0;
    bool ok = true;
    if (leader) {
      for (int q = 0; q < p.P && ok; ++q) ok = gemm::wait_ge<true>(p.arrive + q, (unsigned long long)p.expected[q], g, ERR_G_ARRIVE);
      if (p.P) ptx::fence_proxy_async_all();         // peer stores (generic proxy) before the TMA reads
    }
    ok = __all_sync(0xffffffffu, ok);
    while (ok && it.next(&grp, &n_blk, &tok0, &ntok)) {
      const int boxes = (ntok + p.xbox - 1) / p.xbox;
      const uint32_t box_bytes = (uint32_t)p.xbox * BK * 2;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!warp_wait(L.empty(s), ph ^ 1, g, ERR_G_PRODUCER_EMPTY)) { ok = false; break; }
        if (leader) {
          const uint32_t w = L.base + s * stage, x = w + W_STAGE_BYTES;
          ptx::mbar_arrive_expect_tx(L.full(s), W_STAGE_BYTES + boxes * box_bytes);
          ptx::tma_load_2d(w, &p.map_w, L.full(s), kb * BK, grp * p.N + n_blk * ROWS);
          for (int b = 0; b < boxes; ++b)
            ptx::tma_load_2d(x + b * box_bytes, &p.map_x, L.full(s), kb * BK, grp * p.cap + tok0 + b * p.xbox);
        }
        if (++s == stages) { s = 0; ph ^= 1; }
      }
    }
    if (leader) ptx::grid_launch_dependents();
  } else if (warp == 1) {
    const bool leader = ptx::elect_one();
    int s = 0; uint32_t ph = 0, acc_ph = 0;
    bool ok = true;
    for (int ord = 0; ok && it.next(&grp, &n_blk, &tok0, &ntok); ++ord) {
      const int acc = ord & 1;
      if (!warp_wait(L.acc_empty(acc), ((acc_ph >> acc) & 1) ^ 1, g, ERR_G_MMA_ACC)) break;
      acc_ph ^= 1u << acc;
      ptx::tc_fence_after();
      const uint32_t idesc = ptx::umma_idesc(1, 1, ROWS, (uint32_t)((ntok + 15) / 16 * 16));
      const uint32_t d = tmem + acc * p.nt_cap;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!warp_wait(L.full(s), ph, g, ERR_G_MMA_FULL)) { ok = false; break; }
        ptx::tc_fence_after();
        if (leader) {
          const uint64_t dw = ptx::umma_desc_sw128(L.base + s * stage), dx = ptx::umma_desc_sw128(L.base + s * stage + W_STAGE_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) ptx::umma_f16(d, dw + 2 * k, dx + 2 * k, idesc, (kb > kb0 || k) ? 1u : 0u);
          ptx::umma_commit(L.empty(s));
        }
        if (++s == stages) { s = 0; ph ^= 1; }
      }
      if (ok && leader) ptx::umma_commit(L.acc_full(acc));
    }
  } else {
    const int quarter = warp & 3;
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    uint32_t acc_ph = 0;
    uint32_t vote = 1;
    uint32_t turn = 0;                               // exchange buffer of the next 16 tokens
    for (int ord = 0; it.next(&grp, &n_blk, &tok0, &ntok); ++ord) {
      const int acc = ord & 1;
      bool ok = mbar_wait(L.acc_full(acc), (acc_ph >> acc) & 1, g, ERR_G_EPI_FULL);
      if constexpr (kGated) {
        // a gate and an up warp meet at barriers below: both go on or both leave
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, %2, 64, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(vote) : "r"((uint32_t)ok), "r"(1 + (quarter >> 1)) : "memory");
        ok = vote != 0;
      }
      if (!ok) break;
      acc_ph ^= 1u << acc;
      ptx::tc_fence_after();
      const uint32_t taddr = lanes + acc * p.nt_cap;
      if (split > 1) {
        // [token][weight row] floats over the drained stages
        const uint32_t dst = L.base + (quarter * 32 + lane) * 4;
        for (int c = 0; c < ntok; c += 16) {
          uint32_t v[16];
          ptx::tmem_ld_32x32b_x16(taddr + c, v);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + (c + j) * (ROWS * 4)), "r"(v[j]) : "memory");
        }
        break;
      }
      __nv_bfloat16* out = p.out + ((long long)grp * p.cap + tok0) * p.ldo + (kGated ? n_blk * (ROWS / 2) + (quarter >> 1) * 32 : n_blk * ROWS + quarter * 32) + lane;
      for (int c = 0; c < ntok; c += 16) {
        uint32_t v[16];
        ptx::tmem_ld_32x32b_x16(taddr + c, v);
        ptx::tmem_ld_wait();
        if constexpr (!kGated) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j < ntok) out[(long long)(c + j) * p.ldo] = __float2bfloat16_rn(__uint_as_float(v[j]));
        } else {
          // buffer `turn` is free: the gate warp read it before it came to the barrier of the previous 16 tokens
          const uint32_t buf = xchg + (((quarter >> 1) * 2 + turn) * 16 * 32 + lane) * 4;
          if (quarter & 1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) asm volatile("st.shared.u32 [%0], %1;" ::"r"(buf + j * 128), "r"(v[j]) : "memory");
          }
          asm volatile("bar.sync %0, 64;" ::"r"(1 + (quarter >> 1)) : "memory");
          if (!(quarter & 1)) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              float u;
              asm volatile("ld.shared.f32 %0, [%1];" : "=f"(u) : "r"(buf + j * 128) : "memory");
              const float gate = __uint_as_float(v[j]);
              if (c + j < ntok) out[(long long)(c + j) * p.ldo] = __float2bfloat16_rn(gate / (1.f + __expf(-gate)) * u);
            }
          }
          turn ^= 1;
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(L.acc_empty(acc));
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (split > 1) {
    cluster_sync_all();
    if (mine && !*L.abort_flag()) {
      // one warp per token; a lane's sum over the parts of weight row r of token t
      auto sum = [&](int t, int r) {
        float f = 0.f;
#pragma unroll 4
        for (int q = 0; q < split; ++q) f += ld_cluster_f1(mapa(L.base + (t * ROWS + r) * 4, q));
        return f;
      };
      for (int t = rank + warp * split; t < split_tile.ntok; t += split * (NUM_THREADS / 32)) {
        __nv_bfloat16* out = p.out + ((long long)split_tile.grp * p.cap + split_tile.tok0 + t) * p.ldo;
        if constexpr (kGated) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float gate = sum(t, h * 64 + lane), u = sum(t, h * 64 + 32 + lane);
            out[split_tile.n_blk * (ROWS / 2) + h * 32 + lane] = __float2bfloat16_rn(gate / (1.f + __expf(-gate)) * u);
          }
        } else {
#pragma unroll
          for (int h = 0; h < 4; ++h) out[split_tile.n_blk * ROWS + h * 32 + lane] = __float2bfloat16_rn(sum(t, h * 32 + lane));
        }
      }
    }
    cluster_sync_all();                                  // nobody's shared memory goes away while it is being read
  }
  if (*L.abort_flag()) {
    const unsigned long long t0 = ptx::globaltimer();
    while (ptx::globaltimer() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, p.tmem_cols);
  }
}

}  // namespace skinny
}  // namespace bshmem
