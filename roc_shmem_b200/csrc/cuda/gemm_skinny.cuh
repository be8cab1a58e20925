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
// Every wait is bounded (see gemm_core.cuh).  The reference has no GEMM, hence no counterpart.
#pragma once
#include "gemm_core.cuh"

namespace bshmem {
namespace skinny {

using gemm::Guard;
using gemm::mbar_wait;
using gemm::pack_bf16;

constexpr int ROWS = 128;                          // weight rows of a tile
constexpr int BK = 64;                             // bf16 elements per k-block: one 128-byte swizzle atom
constexpr int MAX_TOKENS = 256;
constexpr int MAX_STAGES = 8;
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
  uint32_t tmem_cols;
  unsigned long long timeout_ns;
  int* err;
};

__host__ __device__ constexpr uint32_t stage_bytes(int nt) { return W_STAGE_BYTES + (uint32_t)nt * BK * 2; }
__host__ __device__ constexpr uint32_t smem_bytes(int nt, int stages) { return stages * stage_bytes(nt) + CTRL_BYTES + 1024; }

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  // volatile keeps it behind the cluster barrier; without a memory clobber a run of them stays together
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
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
  for (int q = 0; q < S; ++q) src[q] = map_rank(base + lane * 16, q);
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
      if (t < p.M)
        *reinterpret_cast<uint2*>(p.out + (long long)t * p.ldo + n0 + lane * 4) =
            make_uint2(pack_bf16(v[u][0].x, v[u][0].y), pack_bf16(v[u][0].z, v[u][0].w));
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
  const int rank = split > 1 ? (int)cluster_rank() : 0;
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
    if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(L.empty(s), ph ^ 1, g, ERR_PRODUCER_EMPTY)) break;
        ptx::mbar_arrive_expect_tx(L.full(s), L.stage);
        if constexpr (kWmn) {
          ptx::tma_load_2d(L.w(s), &p.map_w, L.full(s), n0, kb * BK);
          ptx::tma_load_2d(L.w(s) + W_STAGE_BYTES / 2, &p.map_w, L.full(s), n0 + 64, kb * BK);
        } else {
          ptx::tma_load_2d(L.w(s), &p.map_w, L.full(s), kb * BK, n0);
        }
        ptx::tma_load_2d(L.x(s), &p.map_x, L.full(s), kb * BK, 0);
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      const uint32_t idesc = ptx::umma_idesc(1, 1, ROWS, (uint32_t)p.nt) | (kWmn ? 1u << 15 : 0u);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(L.full(s), ph, g, ERR_MMA_FULL)) { ok = false; break; }
        ptx::tc_fence_after();
        const uint64_t dw = kWmn ? ptx::umma_desc_sw128_ex(L.w(s), W_STAGE_BYTES / 2, 1024) : ptx::umma_desc_sw128(L.w(s));
        const uint64_t dx = ptx::umma_desc_sw128(L.x(s));
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) ptx::umma_f16(tmem, dw + (kWmn ? 128 : 2) * k, dx + 2 * k, idesc, (kb > kb0 || k) ? 1u : 0u);
        ptx::umma_commit(L.empty(s));
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
      if (ok) ptx::umma_commit(L.acc_full());
    }
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
    cluster_sync();
    // every CTA adds the partials of the tokens rank, rank + split, ...
    if (!*L.abort_flag() && n0 + lane * 4 < p.N) {
      if (split == 2) add_partials<2>(p, L.base, rank, warp, lane, n0);
      else if (split == 4) add_partials<4>(p, L.base, rank, warp, lane, n0);
      else add_partials<8>(p, L.base, rank, warp, lane, n0);
    }
    cluster_sync();                                  // nobody's shared memory goes away while it is being read
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
