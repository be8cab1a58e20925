// gemm_fp8_pair.cuh — the plain block-scaled fp8 product (gemm_fp8.cu) on CTA PAIRS (cta_group::2): 256 x 256 tiles.
// CTA r of a pair loads rows [128r, 128r+128) of A and half of the rows of B, 32 KiB per k-block instead of the 48 of a CTA by itself,
// and promotes its 128 rows.  A k-block's product is made in two halves of 128 columns (M256 N128), so that the 512 TMEM columns hold
// four of them: a half's life (its MMAs, commit, promotion, release) may take two k-blocks' time without holding up the MMAs.
//   warp 0       TMA producer (each CTA for its own operands): A, B and, four k-blocks at a time, the rows' scales
//   warp 1       first CTA: MMA issuer.  second CTA: relay of "my stage is full" (see gemm_pair.cuh)
//   warps 2-3    idle: a warpgroup hands registers on as a whole
//   warps 4-11   promotion, 32 rows x 128 columns each (warps 4-7 the first half of a product)
// Reductions are whole groups of four k-blocks, unrolled: buffers, barriers and parities are constants then.
// What bounds it: a promotion warp's chain of loads and FMAs, 720 cycles per k-block (the MMAs: 512; a CTA by itself 905), and the power
// cap behind it (1.48 GHz instead of 1.6 in a short loop, 1.24 instead of 1.35 in a long one).  4096 x 7168 x 8192: 218 -> 187 us in
// the kernel, 236 -> 207 us per product, 273 -> 238 in a loop of a second.  Tried on the way, cycles per k-block: sixteen promotion
// warps of 64 columns that copy their own scales 1150; eight that wait for a product, then load it 1230; the same with the next product asked for and
// its first columns loaded ahead of the last FMAs 790; products of 256 columns in two buffers 770; 32 columns per load (spills) 790 to 1390.
#pragma once
#include "gemm_pair.cuh"

namespace {

constexpr int PSTAGES = 5, PEPI_WARPS = 8, PFIRST_EPI = 4, PTHREADS = 32 * (PFIRST_EPI + PEPI_WARPS);
constexpr int PCOLS = 128, PCHUNK = 16;                 // columns a warp promotes, and how many of them a load brings
constexpr int PGROUP = 4, PGROUPS = 4;                  // k-blocks whose scales travel together, and groups in the ring
constexpr uint32_t PA_BYTES = 128 * 128, PSTAGE_BYTES = 2 * PA_BYTES, PSCALE_BYTES = 128 * 4;
constexpr uint32_t PSMEM_TILES = PSTAGES * PSTAGE_BYTES + PEPI_WARPS * FEPI_BYTES + PGROUPS * PGROUP * PSCALE_BYTES;
constexpr uint32_t PSMEM_BYTES = PSMEM_TILES + 256 + 1024;
constexpr int PREGS_LAUNCH = 168, PREGS_FEW = 40, PREGS_MANY = 232;
static_assert(128 * PREGS_FEW + 32 * PEPI_WARPS * PREGS_MANY <= PTHREADS * PREGS_LAUNCH, "what some give up is what the others take");

enum : int { ERR_F8P_EMPTY = 131, ERR_F8P_PART_EMPTY = 132, ERR_F8P_FULL = 133, ERR_F8P_RELAY = 134, ERR_F8P_PART = 135, ERR_F8P_SCALE = 136 };

struct PSmem {
  uint32_t base;
  uint8_t* gen;
  __device__ __forceinline__ uint32_t a(int s) const { return base + s * PSTAGE_BYTES; }
  __device__ __forceinline__ uint32_t b(int s) const { return base + s * PSTAGE_BYTES + PA_BYTES; }
  __device__ __forceinline__ uint32_t epi(int w) const { return base + PSTAGES * PSTAGE_BYTES + w * FEPI_BYTES; }
  __device__ __forceinline__ uint32_t scales(uint32_t group) const {
    return base + PSTAGES * PSTAGE_BYTES + PEPI_WARPS * FEPI_BYTES + (group % PGROUPS) * (PGROUP * PSCALE_BYTES);
  }
  __device__ __forceinline__ uint32_t bar(int i) const { return base + PSMEM_TILES + 8 * i; }
  __device__ __forceinline__ uint32_t full(int s) const { return bar(s); }
  __device__ __forceinline__ uint32_t empty(int s) const { return bar(PSTAGES + s); }
  __device__ __forceinline__ uint32_t part_full(int b, int half) const { return bar(2 * PSTAGES + 2 * b + half); }
  __device__ __forceinline__ uint32_t part_empty(int b, int half) const { return bar(2 * PSTAGES + 4 + 2 * b + half); }
  __device__ __forceinline__ uint32_t scale_full(uint32_t group) const { return bar(2 * PSTAGES + 8 + group % PGROUPS); }
  __device__ __forceinline__ uint32_t tmem_slot() const { return bar(2 * PSTAGES + 8 + PGROUPS); }
  __device__ __forceinline__ volatile int* abort_flag() const {
    return reinterpret_cast<volatile int*>(gen + PSMEM_TILES + 8 * (2 * PSTAGES + 8 + PGROUPS) + 8);
  }
};
static_assert(8 * (2 * PSTAGES + 8 + PGROUPS) + 16 <= 256, "barriers");

__device__ __forceinline__ void umma2_f8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// PCHUNK columns of a warp's rows.  The wait names the registers of the load it is for: what uses them cannot move in front of it.
__device__ __forceinline__ void chunk_load(uint32_t taddr, uint32_t (&r)[PCHUNK]) {
  ptx::tmem_ld_32x32b_x16(taddr, r);
}
__device__ __forceinline__ void chunk_wait(uint32_t (&r)[PCHUNK]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

__global__ void __launch_bounds__(PTHREADS, 1) gemm_fp8_pair_kernel(const __grid_constant__ Fp8Params prm) {
  extern __shared__ uint8_t smem_raw[];
  PSmem L;
  {
    uint32_t r = ptx::smem_u32(smem_raw);
    L.base = (r + 1023u) & ~1023u;
    L.gen = smem_raw + (L.base - r);
  }
  const CoreParams& cp = prm.core;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = gemm2::cluster_ctarank();
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int num_kb = cp.K / FBK;
  Guard g{cp.err, L.abort_flag(), cp.timeout_ns};

  if (threadIdx.x == 0) {
    *L.abort_flag() = 0;
    for (int s = 0; s < PSTAGES; ++s) { ptx::mbar_init(L.full(s), rank == 0 ? 2 : 1); ptx::mbar_init(L.empty(s), 1); }
    for (int i = 0; i < 4; ++i) {
      ptx::mbar_init(L.part_full(i >> 1, i & 1), 1);
      ptx::mbar_init(L.part_empty(i >> 1, i & 1), PEPI_WARPS);      // a half's four warps in both CTAs
    }
    for (int i = 0; i < PGROUPS; ++i) ptx::mbar_init(L.scale_full(i), 1);
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&prm.map_a);
    ptx::prefetch_tensormap(&prm.map_b);
  }
  if (warp == 1) {
    gemm2::tmem_alloc2(L.tmem_slot(), TMEM_COLS);
    gemm2::tmem_relinquish2();
  }
  ptx::tc_fence_before();
  __syncthreads();
  gemm2::cluster_sync_all();
  ptx::tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(L.tmem_slot()));
  ptx::grid_dependency_wait();

  if (warp < PFIRST_EPI) {
    regs_dec<PREGS_FEW>();
    const bool leader = ptx::elect_one();
    int s = 0; uint32_t ph = 0;
    bool ok = true;
    if (warp == 0) {
      // ------------------------------ TMA producer ------------------------------
      uint32_t group = 0;
      for (int tile = prm.first_tile + pair; tile < prm.end_tile && ok; tile += num_pairs) {
        int m_blk, n_blk;
        raster_coords(cp, tile, &m_blk, &n_blk);
        const int a_row = m_blk * 256 + (int)rank * 128, b_row = n_blk * 256 + (int)rank * 64;
        const float* sa = prm.sa + min(a_row, cp.M - 128);        // rows behind the matrix: scales that exist, results that nobody stores
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!gemm2::warp_wait(L.empty(s), ph ^ 1, g, ERR_F8P_EMPTY)) { ok = false; break; }
          if (leader) {
            ptx::mbar_arrive_expect_tx(L.full(s), PSTAGE_BYTES);
            ptx::tma_load_2d(L.a(s), &prm.map_a, L.full(s), kb * FBK, a_row);
            ptx::tma_load_2d(L.b(s), &prm.map_b, L.full(s), kb * FBK, b_row);
            ptx::tma_load_2d(L.b(s) + 64 * FBK, &prm.map_b, L.full(s), kb * FBK, b_row + 128);
            if (kb % PGROUP == 0) {
              // The slot's last group was read before the products were released that had to be for this stage to be free: PGROUPS *
              // PGROUP k-blocks are more than the stages and the two products on their way.
              ptx::mbar_arrive_expect_tx(L.scale_full(group), PGROUP * PSCALE_BYTES);
              for (int i = 0; i < PGROUP; ++i)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(L.scales(group) + i * PSCALE_BYTES), "l"(sa + (size_t)(kb + i) * cp.M), "r"(PSCALE_BYTES), "r"(L.scale_full(group))
                             : "memory");
              ++group;
            }
          }
          if (++s == PSTAGES) { s = 0; ph ^= 1; }
        }
      }
      if (leader) ptx::grid_launch_dependents();
    } else if (warp == 1 && rank == 0) {
      // ------------------------------ MMA issuer ---------------------------------
      const uint64_t da0 = ptx::umma_desc_sw128(L.a(0)), db0 = ptx::umma_desc_sw128(L.b(0));
      constexpr uint32_t kIdesc = ptx::umma_idesc(0, 0, 256, 128);
      for (int tile = prm.first_tile + pair; tile < prm.end_tile && ok; tile += num_pairs)
        for (int kb0 = 0; kb0 < num_kb && ok; kb0 += PGROUP)
#pragma unroll 1
          for (int i = 0; i < PGROUP; ++i) {
            const uint32_t buf = i & 1, drained = ((i >> 1) & 1) ^ 1;      // products alternate between two buffers, tiles are whole groups
            const uint64_t da = da0 + (uint64_t)((s * PSTAGE_BYTES) >> 4), db = db0 + (uint64_t)((s * PSTAGE_BYTES) >> 4);
            const uint32_t d = tmem_base + buf * 256;
            // Asked ahead by every lane, and agreed on where it is needed: lanes need not see the same, and the waits are the whole warp's.
            // One vote for the first two: 222 us for 4096 x 7168 x 8192, as without votes; a vote each 224.5, a reduction of all three 235.
            const bool there = ptx::mbar_test(L.full(s), ph);
            const bool free0 = ptx::mbar_test(L.part_empty(buf, 0), drained), free1 = ptx::mbar_test(L.part_empty(buf, 1), drained);
            if (!__all_sync(0xffffffffu, there && free0) &&
                !(gemm2::warp_wait(L.full(s), ph, g, ERR_F8P_FULL) && gemm2::warp_wait(L.part_empty(buf, 0), drained, g, ERR_F8P_PART_EMPTY))) { ok = false; break; }
            ptx::tc_fence_after();
            auto multiply = [&](int h) {
#pragma unroll
              for (int k = 0; k < FBK / UMMA_K_BYTES; ++k)
                umma2_f8(d + 128 * h, da + ((k * UMMA_K_BYTES) >> 4), db + ((h * 64 * FBK + k * UMMA_K_BYTES) >> 4), kIdesc, k != 0);
              gemm2::umma2_commit_both(L.part_full(buf, h), 0);
            };
            if (leader) multiply(0);
            if (!__all_sync(0xffffffffu, free1) && !gemm2::warp_wait(L.part_empty(buf, 1), drained, g, ERR_F8P_PART_EMPTY)) { ok = false; break; }
            ptx::tc_fence_after();
            if (leader) {
              multiply(1);
              gemm2::umma2_commit_both(L.empty(s), 0);
            }
            if (++s == PSTAGES) { s = 0; ph ^= 1; }
          }
    } else if (warp == 1) {
      // ------------------------------ relay (second CTA) --------------------------
      for (int tile = prm.first_tile + pair; tile < prm.end_tile && ok; tile += num_pairs)
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!gemm2::warp_wait(L.full(s), ph, g, ERR_F8P_RELAY)) { ok = false; break; }
          if (leader) gemm2::mbar_arrive_cluster(gemm2::mapa(L.full(s), 0));
          if (++s == PSTAGES) { s = 0; ph ^= 1; }
        }
    }
  } else {
    regs_inc<PREGS_MANY>();
    // ------------------------------ promotion + epilogue -------------------------
    const int ew = warp - PFIRST_EPI, quarter = warp & 3, half = ew >> 2;
    const uint32_t tmem0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + half * PCOLS;
    const uint32_t released0 = gemm2::mapa(L.part_empty(0, half), 0);
    const int sb_stride = cp.N / 128;
    const uint32_t made0 = L.part_full(0, half), my_scales = (quarter * 32 + lane) * 4;
    uint32_t group = 0;
    bool ok = true;
    for (int tile = prm.first_tile + pair; tile < prm.end_tile && ok; tile += num_pairs) {
      int m_blk, n_blk;
      raster_coords(cp, tile, &m_blk, &n_blk);
      const float* sb = prm.sb + n_blk * 2 + half;
      float2 acc[PCOLS / 2];
#pragma unroll
      for (int i = 0; i < PCOLS / 2; ++i) acc[i] = make_float2(0.f, 0.f);
      // the weight's scale is one value per k-block: 32 of them across the warp's lanes, the next 32 on their way
      auto sb_load = [&](int kb) -> float { return kb + lane < num_kb ? __ldg(sb + (size_t)(kb + lane) * sb_stride) : 0.f; };
      float sb_now = 0.f, sb_next = sb_load(0);
      uint32_t v[2][PCHUNK];
      if (!gemm2::warp_wait(made0, 0, g, ERR_F8P_PART)) break;
      ptx::tc_fence_after();
      chunk_load(tmem0, v[0]);
#pragma unroll 1
      for (int kb0 = 0; kb0 < num_kb && ok; kb0 += PGROUP, ++group) {
        if ((kb0 & 31) == 0) { sb_now = sb_next; sb_next = sb_load(kb0 + 32); }
        if (!gemm2::warp_wait(L.scale_full(group), (group / PGROUPS) & 1, g, ERR_F8P_SCALE)) { ok = false; break; }
        float sc[PGROUP];
#pragma unroll
        for (int i = 0; i < PGROUP; ++i)
          sc[i] = ptx::ld_shared_f32(L.scales(group) + i * PSCALE_BYTES + my_scales) * __shfl_sync(0xffffffffu, sb_now, (kb0 & 31) + i);
#pragma unroll
        for (int i = 0; i < PGROUP; ++i) {
          const uint32_t buf = i & 1, next = (i + 1) & 1, next_parity = ((i + 1) >> 1) & 1;
          const bool more = i + 1 < PGROUP || kb0 + PGROUP < num_kb;
          const float2 scale = make_float2(sc[i], sc[i]);
          bool seen = false;
#pragma unroll
          for (int c = 0; c < PCOLS / PCHUNK; ++c) {
            // the next columns, of this product or the next, are on their way while these are added
            chunk_wait(v[c & 1]);
            if (c + 1 < PCOLS / PCHUNK) {
              chunk_load(tmem0 + buf * 256 + (c + 1) * PCHUNK, v[(c + 1) & 1]);
              if (c + 2 == PCOLS / PCHUNK) seen = ptx::mbar_test(made0 + 16 * next, next_parity);
            } else {
              ptx::tc_fence_before();          // everything is read: the half may be overwritten
              __syncwarp();
              if (lane == 0) gemm2::mbar_arrive_cluster(released0 + 16 * buf);
              if (more) {
                if (!__all_sync(0xffffffffu, seen) && !gemm2::warp_wait(made0 + 16 * next, next_parity, g, ERR_F8P_PART)) { ok = false; break; }
                ptx::tc_fence_after();
                chunk_load(tmem0 + next * 256, v[0]);
              }
            }
            const uint32_t* x = v[c & 1];
#pragma unroll
            for (int j = 0; j < PCHUNK / 2; ++j)
              acc[c * (PCHUNK / 2) + j] =
                  __ffma2_rn(scale, make_float2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1])), acc[c * (PCHUNK / 2) + j]);
          }
          if (!ok) break;
        }
      }
      if (!ok) break;
#pragma unroll
      for (int h = 0; h < PCOLS / 64; ++h) {
        if (lane == 0) ptx::tma_wait_group_read<0>();       // the previous store has read the buffer
        __syncwarp();
        f8_stage_chunk(L.epi(ew), lane, acc + 32 * h);
        const int row0 = m_blk * 256 + (int)rank * 128 + quarter * 32;
        if (lane == 0 && row0 < cp.M) {
          ptx::tma_store_2d(&prm.map_c, L.epi(ew), n_blk * FBN + half * PCOLS + 64 * h, row0);
          ptx::tma_commit_group();
        }
      }
    }
    if (lane == 0) ptx::tma_wait_group<0>();
    __syncwarp();
  }

  // ------------------------------ teardown ---------------------------------------
  ptx::tc_fence_before();
  __syncthreads();
  if (*L.abort_flag()) {
    unsigned long long t0 = ptx::globaltimer();
    while (ptx::globaltimer() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  gemm2::cluster_sync_all();
  if (warp == 1) {
    ptx::tc_fence_after();
    gemm2::tmem_dealloc2(tmem_base, TMEM_COLS);
  }
}

}  // namespace
