// gemm_pair.cuh — persistent tcgen05 GEMM main loop on CTA PAIRS (cta_group::2) for
// sm_100a:  C[M,N] = A[M,K] · B[N,K]^T, bf16 operands, fp32 accumulation in TMEM.
//
// A thread-block cluster of two CTAs (two SMs of one TPC) owns an output tile of 256 rows and up to 256 columns:
//   CTA r of the pair loads A rows [128r, 128r+128) and B rows [128r, 128r+128) of the
//   tile — 32 KiB per stage and CTA, plain (non-multicast) TMA loads from this GPU's own
//   memory — and holds the accumulator of its 128 output rows x 256 columns in its TMEM.
//   One thread of the pair's first CTA issues tcgen05.mma.cta_group::2 (M256 N256 K16);
//   the tensor cores of both SMs read both CTAs' shared memory.
// An accumulator is 256 TMEM columns, so the 512 columns hold TWO: the epilogue of tile
// i (tcgen05.ld -> bf16 -> swizzled smem -> TMA store, possibly to another GPU) runs
// while the tensor cores already work on tile i+1.  That is the point of this core: the
// single-CTA 256x256 loop (gemm_core.cuh) has to drain both of its accumulators before
// the next tile can start, which exposes the epilogue — and everything the epilogue
// waits for, e.g. NVLink stores — on the critical path.
//
//   warp 0      TMA producer (each CTA for its own halves), 6-stage ring
//   warp 1      first CTA: MMA issuer.  second CTA: relay — waits for its own stage to
//               fill, then arrives on the first CTA's `full` barrier of that stage, which
//               expects two arrivals (a load without the cta_group qualifier can only
//               signal a barrier of the CTA it writes to)
//   warps 2-9   epilogue: warp w drains TMEM lanes 32*(w%4).., columns 128*(w>=6)..
// Producer, issuer and relay are loops of their whole warp; one elected lane issues (see ptx::elect_one): a k-block then takes the 512
// cycles of its MMAs, where from a lane in a branch of its own the issue and the wait took 565.  Long launches gain less, since the power cap
// takes the clock down: 8192 x 8192 x 3584 341 -> 339 us, training of 1000 x 8192 -> 7168 296 -> 290, the 8192-token MLP step 3387 -> 3333.
//
// tcgen05.commit (with its cluster-multicast form, a barrier arrival, not a load) hands
// stages and accumulators back to BOTH CTAs.
// Wide form (policy with kWide): a tile takes both accumulators, up to 512 columns.  Its A rows are loaded once for all of
// them, a quarter less traffic from L2 per product, and read once from shared memory: the MMAs of a k-block go to the two
// accumulators in turn, and the second of each two takes A from the collector buffer.  What is moved counts because a long
// launch runs at the clock that the power cap leaves: 8192 x 8192 x 3584 went from 367 to 350 us (1.31 -> 1.38 PFLOP/s).  The
// epilogue still overlaps the MMAs: at a tile's ends WIDE_BATCH k-blocks go into one accumulator first, then into the
// other, so that each has the time of a batch to be drained.
// Split form (policy with kSplit, for problems with fewer than about half as many tiles as the chip has pairs): the
// cluster is S = 2 or 4 pairs that share one tile.  Each pair sums its share of K; then every CTA parks its fp32
// accumulator (128 x 256, 128 KiB) over its drained ring, and after one cluster barrier CTA (pair j, half r) adds the S
// parked halves r over columns [256 j / S, 256 (j + 1) / S) in pair order and writes them: a reduce-scatter through
// distributed shared memory, without workspace or atomics.
//
// Every wait is bounded by a %globaltimer deadline; on expiry the CTA records a site
// code in the error word and all roles leave their loops; both CTAs always reach the
// closing cluster barrier before TMEM is released.  Every load is a plain tiled TMA
// load of one CTA.  The reference has no GEMM, hence no counterpart.
#pragma once
#include "gemm_core.cuh"

namespace bshmem {
namespace gemm2 {

using gemm::CoreParams;
using gemm::Guard;
using gemm::guard_fail;
using gemm::pack_bf16;
using gemm::raster_coords;

constexpr int BM = 256, BN = 256;                 // tile of the CTA pair
constexpr int CTA_M = 128, CTA_NLOAD = 128;       // rows of A / of B one CTA loads
constexpr int BK_BYTES = 128;
constexpr int BK = 64;                            // bf16 elements per k-block
constexpr int STAGES = 6;
constexpr int UMMA_K_BYTES = 32;
constexpr int NUM_EPI_WARPS = 8;
constexpr int NUM_THREADS = 32 * (2 + NUM_EPI_WARPS);
constexpr int EPI_COLS = 64;
constexpr uint32_t A_STAGE_BYTES = CTA_M * BK_BYTES;           // 16 KiB
constexpr uint32_t B_STAGE_BYTES = CTA_NLOAD * BK_BYTES;       // 16 KiB
constexpr uint32_t STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
constexpr uint32_t EPI_BUF_BYTES = 32 * EPI_COLS * 2;          // one warp: 32 rows x 128 B
constexpr uint32_t SMEM_TILES = STAGES * STAGE_BYTES + NUM_EPI_WARPS * EPI_BUF_BYTES;
constexpr uint32_t SMEM_BARS = 512;
constexpr uint32_t SMEM_BYTES = SMEM_TILES + SMEM_BARS + 1024 /*alignment slack*/;
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t ACC_COLS = 256;
// Wide form: a stage holds B rows for both accumulators, and the same shared memory makes four of them.
constexpr int WIDE_STAGES = 4;
constexpr uint32_t WIDE_STAGE_BYTES = A_STAGE_BYTES + 2 * B_STAGE_BYTES;
// k-blocks at a tile's ends that go into one accumulator before the other (at most WIDE_STAGES): one does not cover the drain
// (8192 x 8192 x 3584: 354 us), with two or three (349, 348) the ring keeps a stage on its way, with four (350) none, which a
// reduction of 16 k-blocks notices (7168 x 8192: 108 us; 108, 105, 104 with one, two, three).
constexpr int WIDE_BATCH = 3;
static_assert(WIDE_STAGES * WIDE_STAGE_BYTES == STAGES * STAGE_BYTES, "both forms share one carve-up");
constexpr uint32_t kIdescBf16 = ptx::umma_idesc(1, 1, BM, BN);

enum ErrSite : int {
  ERR_PRODUCER_EMPTY = 201, ERR_MMA_FULL = 202, ERR_MMA_TMEM_EMPTY = 204, ERR_EPI_TMEM_FULL = 205,
  ERR_RELAY_FULL = 206, ERR_A_READY = 207, ERR_PEER_SIGNAL = 208, ERR_PEER_READY = 209, ERR_PEER_DONE = 210
};

// ---- cluster / cta_group::2 PTX --------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory byte in CTA `rank` of this cluster (shared::cluster window).
__device__ __forceinline__ uint32_t mapa(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Waits use the default (CTA-scope) acquire also for barriers the other CTA arrives on: what such an arrival
// announces is shared-memory or tensor-memory traffic of the async proxies (TMA, tcgen05), not generic-proxy
// stores, and a cluster-scope acquire on every poll made the MMA issuer the bottleneck (2.5x slower).
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) { return ptx::mbar_try_wait(bar, parity); }
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  // volatile keeps it behind the cluster barrier; without a memory clobber a run of them stays together
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t smem_result, uint32_t ncols) {   // whole warp, in both CTAs
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma2_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Two MMAs of the same A, one after the other: the first keeps it in the collector buffer, the second reads it from there.
__device__ __forceinline__ void umma2_f16_keep_a(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16.collector::a::fill [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma2_f16_kept_a(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16.collector::a::lastuse [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One commit that arrives on the barrier at this offset in BOTH CTAs of the pair (two single-destination commits
// per k-block cost the issuing thread 6 % of the GEMM's throughput).
__device__ __forceinline__ void umma2_commit_both(uint32_t bar, uint32_t lead) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)(3u << lead)) : "memory");
}

// Host side: how many clusters of `size` CTAs of `kernel` the device can hold at once (one CTA per SM).
template <class Kernel>
inline int max_resident_clusters(Kernel kernel, int sms, int size, int threads = NUM_THREADS, uint32_t smem = SMEM_BYTES) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(sms / size * size), 1, 1);
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)size; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = sms / size; }
  return n < sms / size ? n : sms / size;
}
template <class Kernel> inline int max_resident_pairs(Kernel kernel, int sms) { return max_resident_clusters(kernel, sms, 2); }

__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity, Guard& g, int site) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  unsigned long long t0 = ptx::globaltimer();
  uint32_t it = 0;
  while (!mbar_try_wait_cluster(bar, parity)) {
    if ((++it & 0x3F) == 0) {
      if (*g.abort_flag) return false;
      if (ptx::globaltimer() - t0 > g.timeout_ns) return guard_fail(g, site);
    }
  }
  return true;
}

// The same by a whole warp: one answer for all lanes, so that the warp stays together.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, Guard& g, int site) {
  return __all_sync(0xffffffffu, pair_wait(bar, parity, g, site));
}

// Shared-memory carve-up (shared-window byte addresses).
struct Smem {
  uint32_t base;        // 1024-byte aligned
  uint8_t* gen;         // generic pointer to the same byte
  __device__ __forceinline__ uint32_t epi(int w) const { return base + STAGES * STAGE_BYTES + w * EPI_BUF_BYTES; }
  __device__ __forceinline__ uint8_t* epi_gen(int w) const { return gen + STAGES * STAGE_BYTES + w * EPI_BUF_BYTES; }
  __device__ __forceinline__ uint32_t bars() const { return base + SMEM_TILES; }
  __device__ __forceinline__ uint32_t full(int s) const { return bars() + 8 * s; }
  __device__ __forceinline__ uint32_t empty(int s) const { return bars() + 8 * (2 * STAGES + s); }
  __device__ __forceinline__ uint32_t tmem_full(int a) const { return bars() + 8 * (3 * STAGES + a); }
  __device__ __forceinline__ uint32_t tmem_empty(int a) const { return bars() + 8 * (3 * STAGES + 2 + a); }
  __device__ __forceinline__ uint32_t tmem_slot() const { return bars() + 8 * (3 * STAGES + 4); }
  __device__ __forceinline__ volatile int* abort_flag() const {
    return reinterpret_cast<volatile int*>(gen + SMEM_TILES + 8 * (3 * STAGES + 4) + 8);
  }
  // 8 words of policy scratch per CTA (zeroed at kernel start), e.g. per-tile arrival counters
  __device__ __forceinline__ unsigned int* scratch() const {
    return reinterpret_cast<unsigned int*>(gen + SMEM_TILES + 256);
  }
  // one word of private state per warp, zeroed at kernel start
  __device__ __forceinline__ volatile int* warp_state(int w) const {
    return reinterpret_cast<volatile int*>(gen + SMEM_TILES + 320 + 4 * w);
  }
};

__device__ __forceinline__ Smem carve_smem(uint8_t* raw) {
  Smem L;
  uint32_t r = ptx::smem_u32(raw);
  L.base = (r + 1023u) & ~1023u;
  L.gen = raw + (L.base - r);
  return L;
}

// What an epilogue warp knows about the chunk it is draining.
struct Chunk {
  int m_blk, n_blk;     // tile
  int row0;             // first of the warp's 32 output rows (row of lane l = row0 + l)
  int col0;             // first of the chunk's 64 output columns
  int ordinal;          // how many tiles this CTA pair has finished before this one
  int half;             // which 128-row half of the tile this CTA holds (its rank in the pair)
};

struct PolicyDefaults {
  struct EpiState {};
  // Split form: clusters of 2 * CoreParams::split CTAs, one tile each, output written by store_rows instead of TMA.
  static constexpr bool kSplit = false;
  // Wide form: a tile takes both accumulators, columns [0, acc_cols(0)) and the acc_cols(1) behind them, and load_b loads the
  // second one's rows of B.
  static constexpr bool kWide = false;
  // kVarCols: acc_cols may be less than 256 (a multiple of 64; with kHalfChunks of 32, and out_target_half is asked for a
  // 32-column box where a chunk of 64 does not fit; gated of 128), and columns beyond N are not written.
  static constexpr bool kVarCols = false, kHalfChunks = false;
  template <class Params> __device__ static __forceinline__ int acc_cols(const Params&, int) { return BN; }
  // bytes that the loads of a stage bring into one CTA
  template <class Params> __device__ static __forceinline__ uint32_t stage_tx(const Params&) { return STAGE_BYTES; }
  // Gated epilogue: inside every 64-column chunk of the accumulator, columns 0-31 are gate pre-activations and 32-63
  // the matching up-projections; the epilogue writes silu(gate) * up, i.e. half as many output columns (the two
  // chunks of a warp make one 32 x 64 output box; out_target gets the OUTPUT column).
  static constexpr bool kGated = false;
  // Training forms of the gated MLP, with kVarCols (the accumulator's columns, rounded to bf16, are stored as they are or replaced):
  // kStoreAct: store_act() additionally gets every chunk (32 gate, 32 up) before it is stored, to write silu(gate) * up.
  // kSwigluBwd: the accumulator is the gradient of the activations; each 32 columns of it become 64 columns of output, the
  // gradients of the matching gate and up pre-activations (swiglu_grad), and out_target gets the output column.
  static constexpr bool kStoreAct = false, kSwigluBwd = false;
  // kRaggedCols: the output's width may end inside a 16-byte piece.  A TMA store fills the piece with zeros, over what lies
  // behind the matrix; such a chunk (ragged_chunk) is written by store_ragged instead, element by element.
  static constexpr bool kRaggedCols = false;
  // kTurns, with kVarCols and kHalfChunks: turned(prm) says that the output is stored transposed, element (row, column) of the tile at
  // (column, row) of the matrix.  The maps of out_target and out_target_half then have boxes of 64 and of 32 columns of the tile by
  // 32 rows, without a swizzle.
  static constexpr bool kTurns = false;
  template <class Params> __device__ static __forceinline__ bool turned(const Params&) { return false; }
  // Operand layout.  Default: both operands K-major, one 128-row x 128-byte TMA box per operand, CTA and stage, and
  // shared-memory descriptors that step 32 bytes along K inside the swizzle atom.  A policy with MN-major operands
  // overrides the instruction descriptor, the stage-0 descriptors, the step per MMA and the loads.
  static constexpr uint32_t kIdesc = kIdescBf16;
  static constexpr uint32_t kKStepA = UMMA_K_BYTES, kKStepB = UMMA_K_BYTES;
  __device__ static __forceinline__ uint64_t desc_a0(uint32_t a0) { return ptx::umma_desc_sw128(a0); }
  __device__ static __forceinline__ uint64_t desc_b0(uint32_t b0) { return ptx::umma_desc_sw128(b0); }
  // a_row / b_row: first row this CTA loads (its rank's half included); kb: k-block of the tile
  template <class Params>
  __device__ static __forceinline__ void load_stage(const Params&, const CUtensorMap* ma, const CUtensorMap* mb, uint32_t a_smem,
                                                    uint32_t b_smem, uint32_t bar, int kb, int a_row, int b_row, int, int, int) {
    ptx::tma_load_2d(a_smem, ma, bar, kb * BK, a_row);
    ptx::tma_load_2d(b_smem, mb, bar, kb * BK, b_row);
  }
  // wide form: this CTA's rows of the second accumulator's columns
  template <class Params>
  __device__ static __forceinline__ void load_b(const Params&, const CUtensorMap* mb, uint32_t b_smem, uint32_t bar, int kb, int b_row, int, int, int) {
    ptx::tma_load_2d(b_smem, mb, bar, kb * BK, b_row);
  }
  // k-blocks of the tile's reduction (ragged per group in the grouped weight-gradient GEMM); at least 1
  template <class Params> __device__ static __forceinline__ int num_kb(const Params& p, int) { return (p.core.K + BK - 1) / BK; }
  // first row of the 256-row block of A / of the tile's block of B that tile (m_blk, n_blk) multiplies
  template <class Params> __device__ static __forceinline__ int a_row(const Params&, int m_blk) { return m_blk * BM; }
  template <class Params> __device__ static __forceinline__ int b_row(const Params&, int, int n_blk) { return n_blk * BN; }
  template <class Params> __device__ static __forceinline__ bool a_ready(const Params&, int, Guard&) { return true; }
  template <class Params> __device__ static __forceinline__ int num_tiles(const Params& p) {
    return p.core.num_m_blocks * p.core.num_n_blocks;
  }
  template <class Params> __device__ static __forceinline__ bool idle_work(const Params&, int, int, Guard&, int, volatile int*) { return false; }
  // epilogue warp, accumulator of the tile is complete, before the first chunk; false aborts
  template <class Params, class St> __device__ static __forceinline__ bool tile_begin(const Params&, const Smem&, St&, const Chunk&, int, int, Guard&) { return true; }
  // the warp's 64 accumulators of this chunk (row = lane) may be changed before they are packed and stored;
  // the warp's staging buffer is free to use here (the previous store has finished reading it)
  template <class Params, class St> __device__ static __forceinline__ void adjust(const Params&, const Smem&, St&, const Chunk&, float (&)[64], int, int) {}
  // after the warp issued (not completed) its stores of the tile
  template <class Params, class St> __device__ static __forceinline__ void tile_end(const Params&, const Smem&, St&, const Chunk&, int, int) {}
  // after an epilogue warp's last tile, all of its stores complete
  template <class Params, class St> __device__ static __forceinline__ void epilogue_drain(const Params&, const Smem&, St&, int, int, Guard&) {}
  template <class Params> __device__ static __forceinline__ void tail(const Params&, const Smem&, Guard&) {}
  template <class Params> __device__ static __forceinline__ void prologue(const Params&, Guard&) {}
  // kTileTable: fill_tile_table(prm) runs in every thread before the first tile_coords().
  static constexpr bool kTileTable = false;
  template <class Params> __device__ static __forceinline__ void fill_tile_table(const Params&) {}
};

// Parks 64 bf16 columns of the warp's 32 rows (row = lane) in its staging buffer for a TMA store: eight 16-byte pieces per
// row, piece j at (j ^ (row & 7)) under the 128-byte swizzle.
__device__ __forceinline__ void stage_chunk(uint32_t buf, int lane, const float (&f)[64]) {
  const uint32_t rowbase = buf + lane * 128;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t w0 = pack_bf16(f[j * 8 + 0], f[j * 8 + 1]), w1 = pack_bf16(f[j * 8 + 2], f[j * 8 + 3]);
    const uint32_t w2 = pack_bf16(f[j * 8 + 4], f[j * 8 + 5]), w3 = pack_bf16(f[j * 8 + 6], f[j * 8 + 7]);
    const uint32_t dst = rowbase + ((j ^ (lane & 7)) << 4);
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w0), "r"(w1), "r"(w2), "r"(w3) : "memory");
  }
  ptx::fence_proxy_async_smem();
  __syncwarp();
}

// The same for values that are packed already, two to a word.
__device__ __forceinline__ void stage_packed(uint32_t buf, int lane, const uint32_t (&w)[32]) {
  const uint32_t rowbase = buf + lane * 128;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t dst = rowbase + ((j ^ (lane & 7)) << 4);
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w[4 * j]), "r"(w[4 * j + 1]), "r"(w[4 * j + 2]), "r"(w[4 * j + 3]) : "memory");
  }
  ptx::fence_proxy_async_smem();
  __syncwarp();
}
// The first 32 columns of them, for a store box of 32: four pieces per row, piece j at (j ^ (row / 2 & 3)) under the 64-byte
// swizzle.
__device__ __forceinline__ void stage_packed_half(uint32_t buf, int lane, const uint32_t (&w)[32]) {
  const uint32_t rowbase = buf + lane * 64;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t dst = rowbase + ((j ^ ((lane >> 1) & 3)) << 4);
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w[4 * j]), "r"(w[4 * j + 1]), "r"(w[4 * j + 2]), "r"(w[4 * j + 3]) : "memory");
  }
  ptx::fence_proxy_async_smem();
  __syncwarp();
}

// 64 columns of the warp's 32 rows for a transposed store: column j's 32 values in a row of 64 bytes, two lanes' values to a word.
__device__ __forceinline__ void stage_turned(uint32_t buf, int lane, const uint32_t (&w)[32]) {
  const bool odd = lane & 1;
  const uint32_t at = buf + (odd ? 64 : 0) + (lane >> 1) * 4;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, w[j], 1);
    const uint32_t v = odd ? __byte_perm(other, w[j], 0x7632) : __byte_perm(w[j], other, 0x5410);
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + j * 128), "r"(v) : "memory");
  }
  ptx::fence_proxy_async_smem();
  __syncwarp();
}

// 64 accumulator columns of this warp's 32 rows (row = lane).
__device__ __forceinline__ void load_acc_chunk(uint32_t taddr, float (&f)[64]) {
  uint32_t v[2][32];
  ptx::tmem_ld_32x32b_x32(taddr, v[0]);
  ptx::tmem_ld_32x32b_x32(taddr + 32, v[1]);
  ptx::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 64; ++i) f[i] = __uint_as_float(v[i >> 5][i & 31]);
}

// The same, rounded to bf16 and packed.  Volatile: packed before the next columns are read, so that no more than 64 registers
// hold unpacked ones.
__device__ __forceinline__ void load_acc_packed(uint32_t taddr, uint32_t (&w)[32]) {
  uint32_t v[2][32];
  ptx::tmem_ld_32x32b_x32(taddr, v[0]);
  ptx::tmem_ld_32x32b_x32(taddr + 32, v[1]);
  ptx::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i)
    asm volatile("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[i]) : "f"(__uint_as_float(v[i >> 4][(2 * i + 1) & 31])), "f"(__uint_as_float(v[i >> 4][(2 * i) & 31])));
}

// Split form, behind the cluster barrier: this CTA's share of the sum, 16 columns of a row per thread and step.
template <class P, int S>
__device__ __forceinline__ void split_reduce(const typename P::Params& prm, const Smem& L, uint32_t crank, int m_blk, int n_blk) {
  constexpr int kGroups = BN / S / 16;                       // 16-column groups of the share
  const int half = crank & 1, j0 = crank >> 1;
  uint32_t src[S];
#pragma unroll
  for (int q = 0; q < S; ++q) src[q] = mapa(L.base, 2 * q + half);
  for (int i = threadIdx.x; i < kGroups * CTA_M; i += NUM_THREADS) {
    const int row = i & (CTA_M - 1), col = j0 * (BN / S) + (i / CTA_M) * 16;
    float4 v[S][4];
#pragma unroll
    for (int q = 0; q < S; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) v[q][e] = ld_cluster_f4(src[q] + ((col / 4 + e) * CTA_M + row) * 16);
#pragma unroll
    for (int q = 1; q < S; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) { v[0][e].x += v[q][e].x; v[0][e].y += v[q][e].y; v[0][e].z += v[q][e].z; v[0][e].w += v[q][e].w; }
    P::store_row16(prm, m_blk * BM + half * CTA_M + row, n_blk * BN + col, v[0]);
  }
}

// Policy contract (static __device__ members; P::Params is the kernel's by-value parameter):
//   core(prm) -> const CoreParams&        map_a(prm), map_b(prm) -> const CUtensorMap*
//   tile_coords(prm, tile, &m_blk, &n_blk)     tile = index in the pair's schedule (pair id + k * pairs)
//   a_ready(prm, m_blk, guard)            producer lane, before a tile's first A load (rows of the whole 256-row block)
//   out_target(prm, row, col, &map, &x, &y)    where the 32x64 chunk starting at C[row, col] goes (map may be null)
//   a_row(prm, m_blk), b_row(prm, m_blk, n_blk), kGated                          (defaults in PolicyDefaults)
//   the hooks of PolicyDefaults
template <class P>
__device__ __forceinline__ void gemm_mainloop(const typename P::Params& prm, uint8_t* smem_raw) {
  const CoreParams& cp = P::core(prm);
  const Smem L = carve_smem(smem_raw);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();
  const uint32_t rank = crank & 1, lead = crank & ~1u;   // the pair's first CTA issues the MMAs
  const int S = P::kSplit ? cp.split : 1;
  constexpr int kStages = P::kWide ? WIDE_STAGES : STAGES, kAccs = P::kWide ? 2 : 1;      // accumulators per tile
  constexpr uint32_t kStageBytes = P::kWide ? WIDE_STAGE_BYTES : STAGE_BYTES;
  auto a_smem = [&](int s) { return L.base + s * kStageBytes; };
  auto b_smem = [&](int s) { return L.base + s * kStageBytes + A_STAGE_BYTES; };
  const int cols0 = P::acc_cols(prm, 0), cols1 = P::kWide ? P::acc_cols(prm, 1) : 0;      // of the tile's accumulators
  const int pair = blockIdx.x / (2 * S), num_pairs = gridDim.x / (2 * S);    // split form: index and number of tiles
  // k-blocks of a tile that this pair multiplies
  auto kb_range = [&](int m_blk, int* kb0, int* kb1) {
    const int n = P::num_kb(prm, m_blk), j = P::kSplit ? (int)(crank >> 1) : 0;
    *kb0 = P::kSplit ? n * j / S : 0;
    *kb1 = P::kSplit ? n * (j + 1) / S : n;
  };
  Guard g{cp.err, L.abort_flag(), cp.timeout_ns};

  if (threadIdx.x == 0) {
    *L.abort_flag() = 0;
    for (int w = 0; w < NUM_THREADS / 32; ++w) *L.warp_state(w) = 0;
    for (int i = 0; i < 8; ++i) L.scratch()[i] = 0;
    for (int s = 0; s < kStages; ++s) {
      // first CTA: its own producer's expect_tx arrival plus the relay's arrival for the second CTA's stage
      ptx::mbar_init(L.full(s), rank == 0 ? 2 : 1);
      ptx::mbar_init(L.empty(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(L.tmem_full(a), 1);
      ptx::mbar_init(L.tmem_empty(a), 2 * NUM_EPI_WARPS);     // every epilogue warp of both CTAs
    }
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(P::map_a(prm));
    ptx::prefetch_tensormap(P::map_b(prm));
  }
  if (warp == 1) {
    tmem_alloc2(L.tmem_slot(), TMEM_COLS);
    tmem_relinquish2();
  }
  ptx::tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                 // the peer's barriers exist before anyone arrives on them
  ptx::tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(L.tmem_slot()));
  // launched with programmatic serialization, the set-up above overlaps the previous kernel; without, this is a no-op
  ptx::grid_dependency_wait();
  if (threadIdx.x == 64) P::prologue(prm, g);
  if constexpr (P::kTileTable) {
    P::fill_tile_table(prm);
    __syncthreads();
  }
  const int num_tiles = P::num_tiles(prm);            // may come from device memory: behind the wait

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    const bool leader = ptx::elect_one();
    int s = 0; uint32_t ph = 0;
    bool ok = true;
    const uint32_t tx = P::stage_tx(prm);
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      int m_blk, n_blk, kb0, kb1;
      P::tile_coords(prm, tile, &m_blk, &n_blk);
      if (!__all_sync(0xffffffffu, !leader || P::a_ready(prm, m_blk, g))) break;
      kb_range(m_blk, &kb0, &kb1);
      const int a_row = P::a_row(prm, m_blk) + (int)rank * CTA_M;
      const int b_row = P::b_row(prm, m_blk, n_blk) + (int)rank * (cols0 / 2);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!warp_wait(L.empty(s), ph ^ 1, g, ERR_PRODUCER_EMPTY)) { ok = false; break; }
        if (leader) {
          ptx::mbar_arrive_expect_tx(L.full(s), tx);
          P::load_stage(prm, P::map_a(prm), P::map_b(prm), a_smem(s), b_smem(s), L.full(s), kb, a_row, b_row, m_blk, n_blk, (int)rank);
          if constexpr (P::kWide)
            P::load_b(prm, P::map_b(prm), b_smem(s) + B_STAGE_BYTES, L.full(s), kb,
                      P::b_row(prm, m_blk, n_blk) + cols0 + (int)rank * (cols1 / 2), m_blk, n_blk, (int)rank);
        }
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
    }
    if (leader) ptx::grid_launch_dependents();       // all loads are on their way: the next kernel's blocks may take their places
  } else if (warp == 1) {
    const bool leader = ptx::elect_one();
    if (rank == 0) {
      // ------------------------------ MMA issuer (first CTA) ---------------------------------
      int s = 0; uint32_t ph = 0;
      uint32_t acc_ph = 0;          // bit a = phase of accumulator a
      bool ok = true;
      const uint64_t desc_a0 = P::desc_a0(a_smem(0)), desc_b0 = P::desc_b0(b_smem(0));
      // the instruction's N is the width of the accumulator
      constexpr uint32_t kNoN = ~(0x3Fu << 17);
      const uint32_t idesc0 = P::kVarCols ? (P::kIdesc & kNoN) | (uint32_t)(cols0 >> 3) << 17 : P::kIdesc;
      const uint32_t idesc1 = P::kVarCols ? (P::kIdesc & kNoN) | (uint32_t)(cols1 >> 3) << 17 : P::kIdesc;
      auto wait_acc = [&](int acc) {     // the epilogue warps of both CTAs must have drained it
        if (!warp_wait(L.tmem_empty(acc), ((acc_ph >> acc) & 1) ^ 1, g, ERR_MMA_TMEM_EMPTY)) return false;
        acc_ph ^= 1u << acc;
        ptx::tc_fence_after();
        return true;
      };
      auto wait_stage = [&](int st, uint32_t parity) {
        if (!warp_wait(L.full(st), parity, g, ERR_MMA_FULL)) return false;
        ptx::tc_fence_after();
        return true;
      };
      // What the leader does.  One k-block into one accumulator; which = 1: the second one's rows of B.  Descriptors differ only in
      // the 16-byte-unit start address (low 14 bits; shared memory is < 256 KiB).
      auto multiply = [&](int st, int acc, int which, bool first) {
        const uint64_t da = desc_a0 + (uint64_t)((st * kStageBytes) >> 4);
        const uint64_t db = desc_b0 + (uint64_t)((st * kStageBytes + which * B_STAGE_BYTES) >> 4);
#pragma unroll
        for (int k = 0; k < BK_BYTES / UMMA_K_BYTES; ++k)
          umma2_f16(tmem_base + acc * ACC_COLS, da + (uint64_t)((k * P::kKStepA) >> 4), db + (uint64_t)((k * P::kKStepB) >> 4),
                    which ? idesc1 : idesc0, (!first || k != 0) ? 1u : 0u);
      };
      int ord = 0;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++ord) {
        int m_blk, n_blk, kb0, kb1;
        P::tile_coords(prm, tile, &m_blk, &n_blk);
        kb_range(m_blk, &kb0, &kb1);
        if constexpr (!P::kWide) {
          const int acc = ord & 1;
          if (!wait_acc(acc)) break;                   // drained two tiles ago
          for (int kb = kb0; kb < kb1; ++kb) {
            if (!wait_stage(s, ph)) { ok = false; break; }
            if (leader) {
              multiply(s, acc, 0, kb == kb0);
              umma2_commit_both(L.empty(s), lead);     // stage reusable in both CTAs once these MMAs retire
            }
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
          if (!ok) break;
          if (leader) umma2_commit_both(L.tmem_full(acc), lead);
        } else {
          // `count` stages into accumulator 0, then into accumulator 1, which hands them back.  The first and the last
          // k-blocks of a tile go in batches: while accumulator 1 takes its last k-blocks, the epilogue
          // drains accumulator 0, and while that takes the first ones of the next tile, accumulator 1 is drained.
          auto batch = [&](int count, bool begin, bool end) {
            if (begin && !wait_acc(0)) return false;
            int t = s; uint32_t tph = ph;
            for (int i = 0; i < count; ++i) {
              if (!wait_stage(t, tph)) return false;
              if (leader) multiply(t, 0, 0, begin && i == 0);
              if (++t == kStages) { t = 0; tph ^= 1; }
            }
            if (end && leader) umma2_commit_both(L.tmem_full(0), lead);
            if (begin && !wait_acc(1)) return false;
            for (int i = 0; i < count; ++i) {
              if (leader) {
                multiply(s, 1, 1, begin && i == 0);
                umma2_commit_both(L.empty(s), lead);
              }
              if (++s == kStages) { s = 0; ph ^= 1; }
            }
            if (end && leader) umma2_commit_both(L.tmem_full(1), lead);
            return true;
          };
          // in between, both accumulators take a k-block together: A is read once for the two
          auto multiply_both = [&](int st) {
            const uint64_t da = desc_a0 + (uint64_t)((st * kStageBytes) >> 4), db = desc_b0 + (uint64_t)((st * kStageBytes) >> 4);
#pragma unroll
            for (int k = 0; k < BK_BYTES / UMMA_K_BYTES; ++k) {
              const uint64_t a = da + (uint64_t)((k * P::kKStepA) >> 4), b = db + (uint64_t)((k * P::kKStepB) >> 4);
              umma2_f16_keep_a(tmem_base, a, b, idesc0, 1u);
              umma2_f16_kept_a(tmem_base + ACC_COLS, a, b + (B_STAGE_BYTES >> 4), idesc1, 1u);
            }
          };
          const int n = kb1 - kb0;
          if (n <= WIDE_BATCH) {
            ok = batch(n, true, true);
          } else {
            const int last = min(n - WIDE_BATCH, WIDE_BATCH);
            ok = batch(WIDE_BATCH, true, false);
            for (int i = n - WIDE_BATCH - last; i > 0 && ok; --i) {
              if (!wait_stage(s, ph)) { ok = false; break; }
              if (leader) {
                multiply_both(s);
                umma2_commit_both(L.empty(s), lead);
              }
              if (++s == kStages) { s = 0; ph ^= 1; }
            }
            ok = ok && batch(last, false, true);
          }
        }
      }
    }
    else {
      // ------------------------------ relay (second CTA) --------------------------------------
      int s = 0; uint32_t ph = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        int m_blk, n_blk, kb0, kb1;
        P::tile_coords(prm, tile, &m_blk, &n_blk);
        kb_range(m_blk, &kb0, &kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!warp_wait(L.full(s), ph, g, ERR_RELAY_FULL)) { ok = false; break; }
          if (leader) mbar_arrive_cluster(mapa(L.full(s), lead));
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    // ------------------------------ epilogue (both CTAs) ------------------------------------
    const int ew = warp - 2;               // 0..7
    const int quarter = warp & 3;          // TMEM lanes 32*quarter.. belong to this warp
    const int colhalf = ew >> 2;           // columns 128*colhalf.. of the accumulator
    uint32_t full_ph = 0;           // bit a = phase of accumulator a
    typename P::EpiState st{};
    bool ok = true;
    int ord = 0;                    // accumulators before this one: a tile has kAccs of them
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs)
    for (int part = 0; part < kAccs && ok; ++part, ++ord) {
      const int acc = ord & 1;
      const int cols = part ? cols1 : cols0;
      Chunk ck;
      P::tile_coords(prm, tile, &ck.m_blk, &ck.n_blk);
      ck.ordinal = ord;
      ck.half = (int)rank;
      ck.row0 = P::a_row(prm, ck.m_blk) + (int)rank * CTA_M + quarter * 32;
      ck.col0 = ck.n_blk * (cols0 + cols1) + part * cols0 + colhalf * 128;
      // the tensor core is busy with this tile: do useful work until the accumulator is ready
      while (!mbar_try_wait_cluster(L.tmem_full(acc), ((full_ph >> acc) & 1))) {
        if (!P::idle_work(prm, ew, lane, g, tile, L.warp_state(warp))) {
          if (!pair_wait(L.tmem_full(acc), ((full_ph >> acc) & 1), g, ERR_EPI_TMEM_FULL)) ok = false;
          break;
        }
      }
      if (!ok) break;
      full_ph ^= 1u << acc;
      ptx::tc_fence_after();
      const uint32_t tacc = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * ACC_COLS + colhalf * 128;
      auto acc_done = [&]() {
        // all TMEM reads of this warp are done: hand the accumulator back to the MMA issuer
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa(L.tmem_empty(acc), lead));
      };
      if constexpr (P::kSplit) {
        // [float4 of the row][row]: the lanes' stores and the reading side's loads are consecutive
        const uint32_t dst = L.base + (colhalf * 32 * CTA_M + quarter * 32 + lane) * 16;
#pragma unroll 1
        for (int c = 0; c < 128; c += 32) {
          uint32_t v[32];
          ptx::tmem_ld_32x32b_x32(tacc + c, v);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (c / 4 + j) * CTA_M * 16), "r"(v[4 * j]), "r"(v[4 * j + 1]),
                         "r"(v[4 * j + 2]), "r"(v[4 * j + 3]) : "memory");
        }
        break;                             // one tile per cluster; the rest happens behind the cluster barrier
      }
      if (!P::tile_begin(prm, L, st, ck, ew, lane, g)) { ok = false; break; }
      if constexpr (!P::kVarCols && !P::kGated) {
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          float f[64];
          load_acc_chunk(tacc + c * EPI_COLS, f);
          if (c == 1) acc_done();
          // the previous chunk's TMA store must have finished reading the staging buffer
          if (lane == 0) ptx::tma_wait_group_read<0>();
          __syncwarp();
          Chunk cc = ck;
          cc.col0 = ck.col0 + c * EPI_COLS;
          P::adjust(prm, L, st, cc, f, ew, lane);
          stage_chunk(L.epi(ew), lane, f);
          if (lane == 0) {
            const CUtensorMap* map; int x, y;
            P::out_target(prm, cc.row0, cc.col0, &map, &x, &y);
            if (map != nullptr) ptx::tma_store_2d(map, L.epi(ew), x, y);
            ptx::tma_commit_group();
          }
        }
      } else if constexpr (P::kSwigluBwd || P::kStoreAct) {
        const int left = min(cols - colhalf * 128, 128);        // of this warp, a multiple of 64; may be none
        if (left <= 0) acc_done();
#pragma unroll 1
        for (int c = 0; c * EPI_COLS < left; ++c) {
          float f[64];
          load_acc_chunk(tacc + c * EPI_COLS, f);
          if ((c + 1) * EPI_COLS >= left) acc_done();
          const int col0 = ck.col0 + c * EPI_COLS;
          if (col0 >= cp.N) continue;
          auto store = [&](int col) {                        // the staged 64 columns
            if (lane != 0) return;
            const CUtensorMap* map; int x, y;
            P::out_target(prm, ck.row0, col, &map, &x, &y);
            if (map != nullptr) ptx::tma_store_2d(map, L.epi(ew), x, y);
            ptx::tma_commit_group();
          };
          if constexpr (P::kStoreAct) {
            if (lane == 0) ptx::tma_wait_group_read<0>();    // the previous store has read the staging buffer
            __syncwarp();
            P::store_act(prm, ck.row0 + lane, col0, f);
            stage_chunk(L.epi(ew), lane, f);
            store(col0);
          } else {
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              float d[32], o[64];
#pragma unroll
              for (int i = 0; i < 32; ++i) d[i] = h == 0 ? f[i] : f[32 + i];
              P::swiglu_grad(prm, ck.row0 + lane, col0 + 32 * h, d, o);
              if (lane == 0) ptx::tma_wait_group_read<0>();
              __syncwarp();
              stage_chunk(L.epi(ew), lane, o);
              store(2 * (col0 + 32 * h));
            }
          }
        }
      } else if constexpr (!P::kGated) {
        // In the wide form, where the tensor cores wait for the accumulator, all of the warp's columns are read, rounded and packed
        // before the first are stored; else 64 at a time.
        constexpr int kAtOnce = P::kWide ? 2 : 1;
        const int left = min(cols - colhalf * 128, 128);        // of this warp, a multiple of 32; may be none
        if (left <= 0) acc_done();
#pragma unroll 1
        for (int c0 = 0; c0 * EPI_COLS < left; c0 += kAtOnce) {
          uint32_t w[kAtOnce][32];
          if constexpr (P::kWide) {
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u)
              if (u * EPI_COLS < left) load_acc_packed(tacc + u * EPI_COLS, w[u]);
            acc_done();
          } else {
            float f[64];
            load_acc_chunk(tacc + c0 * EPI_COLS, f);
            if ((c0 + 1) * EPI_COLS >= left) acc_done();
#pragma unroll
            for (int i = 0; i < 32; ++i) w[0][i] = pack_bf16(f[2 * i], f[2 * i + 1]);
          }
#pragma unroll
          for (int u = 0; u < kAtOnce; ++u) {
            const int mine = left - (c0 + u) * EPI_COLS, col0 = ck.col0 + (c0 + u) * EPI_COLS;
            if (mine <= 0 || col0 >= cp.N) continue;
            bool turned = false;
            if constexpr (P::kTurns) turned = P::turned(prm);
            if constexpr (P::kRaggedCols) {
              if (!turned && P::ragged_chunk(prm, col0)) {
                P::store_ragged(prm, ck.row0 + lane, col0, w[u], mine);
                continue;
              }
            }
            if (lane == 0) ptx::tma_wait_group_read<0>();     // the previous store has read the staging buffer
            __syncwarp();
            const CUtensorMap* map; int x, y;
            if (turned) stage_turned(L.epi(ew), lane, w[u]);
            else if (P::kHalfChunks && mine < EPI_COLS) stage_packed_half(L.epi(ew), lane, w[u]);
            else stage_packed(L.epi(ew), lane, w[u]);
            if (lane == 0) {
              P::out_target(prm, ck.row0, col0, &map, &x, &y);
              if constexpr (P::kHalfChunks) {
                if (mine < EPI_COLS) P::out_target_half(prm, ck.row0, col0, &map, &x, &y);
              }
              if (map != nullptr) ptx::tma_store_2d(map, L.epi(ew), x, y);
              ptx::tma_commit_group();
            }
          }
        }
      } else if (P::kVarCols && (colhalf * 128 >= cols || ck.col0 >= cp.N)) {
        acc_done();
      } else {
        // the warp's two 64-column chunks (32 gate + 32 up each) make one 64-column output chunk
        if (lane == 0) ptx::tma_wait_group_read<0>();     // the previous tile's store has read the staging buffer
        __syncwarp();
        const uint32_t rowbase = L.epi(ew) + lane * 128;
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
          float f[64];                     // 32 gate pre-activations, then the 32 matching up-projections
          load_acc_chunk(tacc + hc * EPI_COLS, f);
          if (hc == 1) acc_done();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float g0 = f[j * 8 + 2 * q], g1 = f[j * 8 + 2 * q + 1];
              float u0 = f[32 + j * 8 + 2 * q], u1 = f[32 + j * 8 + 2 * q + 1];
              float h0 = g0 / (1.f + __expf(-g0)) * u0, h1 = g1 / (1.f + __expf(-g1)) * u1;
              w[q] = pack_bf16(h0, h1);
            }
            uint32_t dst = rowbase + (((hc * 4 + j) ^ (lane & 7)) << 4);
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
          }
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const CUtensorMap* map; int x, y;
          P::out_target(prm, ck.row0, ck.col0 / 2, &map, &x, &y);     // output column = half the accumulator column
          if (map != nullptr) ptx::tma_store_2d(map, L.epi(ew), x, y);
          ptx::tma_commit_group();
        }
      }
      P::tile_end(prm, L, st, ck, ew, lane);
    }
    if (lane == 0) ptx::tma_wait_group<0>();
    __syncwarp();
    if (ok) P::epilogue_drain(prm, L, st, ew, lane, g);
  }

  // ------------------------------ tail + teardown ---------------------------------------
  ptx::tc_fence_before();
  __syncthreads();
  if constexpr (P::kSplit) {
    cluster_sync_all();                               // every part of the tile is parked
    int m_blk, n_blk;
    P::tile_coords(prm, pair, &m_blk, &n_blk);
    if (!*L.abort_flag()) {
      if (S == 2) split_reduce<P, 2>(prm, L, crank, m_blk, n_blk);
      else split_reduce<P, 4>(prm, L, crank, m_blk, n_blk);
    }
  }
  if (!*L.abort_flag()) P::tail(prm, L, g);
  __syncthreads();
  if (*L.abort_flag()) {
    // let copies and MMAs that are still in flight land before smem/TMEM go away
    unsigned long long t0 = ptx::globaltimer();
    while (ptx::globaltimer() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  // neither CTA may leave (its shared memory and TMEM are read by the pair's MMAs and written by the
  // other CTA's arrivals) before both are done
  cluster_sync_all();
  if (warp == 1) {
    ptx::tc_fence_after();
    tmem_dealloc2(tmem_base, TMEM_COLS);
  }
}

}  // namespace gemm2
}  // namespace bshmem
