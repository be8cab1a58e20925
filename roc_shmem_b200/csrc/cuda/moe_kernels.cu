// moe_kernels.cu — expert-parallel MoE layer pieces for sm_100a: router + top-k, a
// deterministic dispatch plan, token dispatch and combine over NVLink with
// putmem + signal semantics, SwiGLU forward/backward and the transposes the
// weight-gradient GEMMs need.  The grouped expert GEMM itself is in moe_gemm.cu.
//
// Data flow (E experts over P PEs, E/P experts per PE, top-k routing):
//   router_topk   logits = x · Wr^T, softmax, top-k, renormalised weights
//   plan          per expert: position of every (token, k) entry in token order → `pos`, counts
//   (all-gather of the counts through the runtime's fcollect)
//   offsets       where this PE's entries start inside every destination expert's buffer
//                 (entries are laid out by source PE, then token order → reproducible bits)
//   dispatch      one warp per entry: putmem of the token row into the destination expert's
//                 receive buffer slot (peer stores), entry id into the meta array; one
//                 release-add per (CTA, destination) on the destination's arrival word
//   [grouped GEMM gate/up → SwiGLU → grouped GEMM down; waits on the arrival words]
//   combine_send  expert PE returns each output row to the source PE's per-entry buffer + signal
//   combine_reduce  out[token] = sum_k w[token,k] * y[entry]
// Backward runs the same flow with gradients (dispatch of w·d_out, combine of dX rows).
//
// Arrival words are double-buffered by call parity and zeroed one call ahead, every wait
// is bounded.  The reference has no MoE layer; the put + signal idiom is its
// put / fence / flag pattern (library/src/gpu_ib/context_ib_tmpl_device.hpp:184-236).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>
#include <string>
#include <utility>

#include "../include/bshmem_device.cuh"
#include "moe_common.h"
#include "ptx.cuh"

using namespace bshmem;
using dev::State;

namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------------------
// router; E <= 64 experts, top-k <= 8
// ---------------------------------------------------------------------------------------
// The logits are a skinny product, T x H by H x E: a block takes 16 tokens, its eight warps share the reduction in steps of
// 32 columns, and the tensor cores multiply (mma.sync: 64 columns at most are no work for a tcgen05 tile, whose launch and
// epilogue cost more than these kernels take).  The products of bf16 numbers are exact in fp32, but the unit truncates where it
// adds, which shows in a chain over the whole reduction: rel. error of the probabilities against fp64 3.5e-7 (16384 x 4096, 8
// experts) and 2.5e-7 (4096 x 2048, 64) where fp32 FMAs give 1.1e-7 and 1.6e-7.  So every product of 16 columns starts from
// zero and the sums are fp32 additions, the warps' in a tree: 0.9e-7 and 1.1e-7, 31 and 14 us (29 and 14 with the chain).
// Fragments come straight from global memory, 16 bytes per lane: the reduction may run over the columns in any order
// as long as both operands agree, so a lane's eight consecutive columns stand for two k-steps' worth of its elements.
// With a warp of FMAs per four tokens, Wr was read from L2 for every four and the FMAs took over for many experts: 16384 x
// 4096, 8 experts 92 us; 12000 x 2048, 64 experts 245 us (44 now).
constexpr int kRouterTok = 16;
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// Softmax over the experts, top-k, weights renormalised over the chosen ones; one warp per token, `lg` in shared memory.
__device__ __forceinline__ void router_select(float* lg, int E, int topk, int lane, int* __restrict__ idx, float* __restrict__ w,
                                              float* __restrict__ probs) {
  float mx = -INFINITY;
  for (int e = lane; e < E; e += 32) mx = fmaxf(mx, lg[e]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float p[2], den = 0.f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    p[h] = lane + 32 * h < E ? __expf(lg[lane + 32 * h] - mx) : 0.f;
    den += p[h];
  }
  den = warp_sum(den);
  // probabilities are not negative: their bit patterns order like the numbers (+1: 0 stands for taken); ties go to the lower
  // expert index
  unsigned key[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int e = lane + 32 * h;
    p[h] /= den;
    if (e < E && probs) probs[e] = p[h];
    key[h] = e < E ? __float_as_uint(p[h]) + 1u : 0u;
  }
  float wsum = 0.f, mine = 0.f;
  int best_e = 0;
  for (int k = 0; k < topk; ++k) {
    const unsigned best = __reduce_max_sync(0xffffffffu, max(key[0], key[1]));
    const unsigned low = __ballot_sync(0xffffffffu, key[0] == best), high = __ballot_sync(0xffffffffu, key[1] == best);
    const int e = min(low ? __ffs(low) - 1 : 31 + __ffs(high), E - 1);
    if (e == lane) key[0] = 0;
    if (e == lane + 32) key[1] = 0;
    const float pe = __uint_as_float(best - 1u);
    wsum += pe;
    if (lane == k) { mine = pe; best_e = e; }
  }
  if (lane < topk) { idx[lane] = best_e; w[lane] = mine / wsum; }
}

// kTiles: tiles of eight experts.  kWarps: eight, or sixteen with half the steps each while there are few blocks.
template <int kTiles, int kWarps>
__global__ void __launch_bounds__(32 * kWarps) k_router_topk(const bf16* __restrict__ x, const bf16* __restrict__ wr, int T, int H, int E,
                                                                   int topk, int* __restrict__ topk_idx, float* __restrict__ topk_w,
                                                                   float* __restrict__ probs) {
  constexpr int kPitch = kTiles * 8 + 2;
  __shared__ float part[8][kRouterTok * kPitch];
  __shared__ float lg[kWarps][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int t0 = blockIdx.x * kRouterTok;
  constexpr int kUnroll = kTiles >= 8 ? 2 : 4;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  ptx::grid_dependency_wait();
  const bf16* xa = x + (size_t)min(t0 + g, T - 1) * H;
  const bf16* xb = x + (size_t)min(t0 + g + 8, T - 1) * H;
  float acc[kTiles][4];
#pragma unroll
  for (int j = 0; j < kTiles; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
  const int steps = (H + 31) / 32;
  for (int s0 = warp; s0 < steps; s0 += kUnroll * kWarps) {
    uint4 a[kUnroll], b[kUnroll], w[kUnroll][kTiles];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int col = (s0 + u * kWarps) * 32 + c * 8;
      const bool in = col < H;
      a[u] = in ? __ldcg(reinterpret_cast<const uint4*>(xa + col)) : zero;
      b[u] = in ? __ldcg(reinterpret_cast<const uint4*>(xb + col)) : zero;
#pragma unroll
      for (int j = 0; j < kTiles; ++j)
        w[u][j] = in && j * 8 + g < E ? __ldg(reinterpret_cast<const uint4*>(wr + (size_t)(j * 8 + g) * H + col)) : zero;
    }
    // Every product starts from zero.  Eight products per addition to the accumulator, four or two where registers are short
    // (eight with 64 experts: 140 registers, 12000 x 2048 takes 59 us instead of 44).
    constexpr int kStep = kTiles == 1 ? kUnroll : kTiles == 2 ? 2 : 1;
#pragma unroll
    for (int u0 = 0; u0 < kUnroll; u0 += kStep)
#pragma unroll
      for (int j = 0; j < kTiles; ++j) {
        float c[2 * kStep][4];
#pragma unroll
        for (int v = 0; v < kStep; ++v) {
          const int u = u0 + v;
          mma_bf16(c[2 * v], a[u].x, b[u].x, a[u].y, b[u].y, w[u][j].x, w[u][j].y);
          mma_bf16(c[2 * v + 1], a[u].z, b[u].z, a[u].w, b[u].w, w[u][j].z, w[u][j].w);
        }
#pragma unroll
        for (int n = kStep; n > 0; n /= 2)
#pragma unroll
          for (int v = 0; v < n; ++v)
#pragma unroll
            for (int i = 0; i < 4; ++i) c[v][i] += c[v + n][i];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] += c[0][i];
      }
  }
  auto park = [&](bool add) {
    float* p0 = part[warp & 7] + g * kPitch + c * 2;
    float* p1 = p0 + 8 * kPitch;
#pragma unroll
    for (int j = 0; j < kTiles; ++j) {
      float2 lo = make_float2(acc[j][0], acc[j][1]), hi = make_float2(acc[j][2], acc[j][3]);
      float2* d0 = reinterpret_cast<float2*>(p0 + j * 8);
      float2* d1 = reinterpret_cast<float2*>(p1 + j * 8);
      if (add) { lo.x += d0->x; lo.y += d0->y; hi.x += d1->x; hi.y += d1->y; }
      *d0 = lo;
      *d1 = hi;
    }
  };
  if (kWarps > 8) {
    if (warp >= 8) park(false);
    __syncthreads();
  }
  if (warp < 8) park(kWarps > 8);
  __syncthreads();
  for (int r = warp; r < kRouterTok; r += kWarps) {
    const int t = t0 + r;
    if (t >= T) break;
    __syncwarp();
    for (int e = lane; e < E; e += 32) {
      float sum[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) sum[q] = part[q][r * kPitch + e];
#pragma unroll
      for (int step = 4; step > 0; step /= 2)
#pragma unroll
        for (int q = 0; q < step; ++q) sum[q] += sum[q + step];
      lg[warp][e] = sum[0];
    }
    __syncwarp();
    router_select(lg[warp], E, topk, lane, topk_idx + (size_t)t * topk, topk_w + (size_t)t * topk, probs ? probs + (size_t)t * E : nullptr);
  }
}

// ---------------------------------------------------------------------------------------
// plan: CTA e assigns positions to the entries routed to expert e, in entry order
// ---------------------------------------------------------------------------------------
// Every warp owns a contiguous run of entries, read 128 at a time: count, one scan over the warps, assign (a block-wide
// scan per 1024 entries took 54 us for 32768 entries).  Returns the expert's count to every thread.
__device__ __forceinline__ int plan_expert(const int* topk_idx, int n_entries, int e, int* __restrict__ pos) {
  __shared__ int warp_tot[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int per = ((n_entries + nw - 1) / nw + 127) / 128 * 128;
  const int b = min(wid * per, n_entries), end = min(b + per, n_entries);
  auto load = [&](int i) -> int4 {                   // entries i .. i+3; -1 past the end
    if (i + 4 <= end) return __ldcg(reinterpret_cast<const int4*>(topk_idx + i));
    int4 v = make_int4(-1, -1, -1, -1);
    if (i < end) v.x = __ldcg(topk_idx + i);
    if (i + 1 < end) v.y = __ldcg(topk_idx + i + 1);
    if (i + 2 < end) v.z = __ldcg(topk_idx + i + 2);
    return v;
  };
  int mine = 0;
#pragma unroll 4
  for (int i = b + lane * 4; i < end; i += 128) {
    const int4 v = load(i);
    mine += (v.x == e) + (v.y == e) + (v.z == e) + (v.w == e);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if (lane == 0) warp_tot[wid] = mine;
  __syncthreads();
  int before = 0, total = 0;
  for (int w = 0; w < nw; ++w) {
    if (w < wid) before += warp_tot[w];
    total += warp_tot[w];
  }
#pragma unroll 2
  for (int i0 = b; i0 < end; i0 += 128) {
    const int i = i0 + lane * 4;
    const int4 v = load(i);
    const int hits = (v.x == e) + (v.y == e) + (v.z == e) + (v.w == e);
    int incl = hits;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    int p = before + incl - hits;
    if (v.x == e) pos[i] = p++;
    if (v.y == e) pos[i + 1] = p++;
    if (v.z == e) pos[i + 2] = p++;
    if (v.w == e) pos[i + 3] = p++;
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
  return total;
}
__global__ void __launch_bounds__(1024) k_plan(const int* __restrict__ topk_idx, int n_entries, int* __restrict__ pos,
                                               int* __restrict__ counts) {
  ptx::grid_dependency_wait();
  const int total = plan_expert(topk_idx, n_entries, blockIdx.x, pos);
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

// ---------------------------------------------------------------------------------------
// offsets: from the gathered counts [P][E] derive everything the data movement needs
// ---------------------------------------------------------------------------------------
// count(s, e): entries of source s for expert e
template <class Count>
__device__ __forceinline__ void offsets_block(const MoePlanDev& pl, Count count, int parity) {
  const int P = pl.P, E = pl.E, Epr = E / P, me = pl.me, cap = pl.cap;
  const int tid = threadIdx.x;
  // start of my entries inside every expert's buffer
  for (int e = tid; e < E; e += blockDim.x) {
    int b = 0;
    for (int s = 0; s < me; ++s) b += count(s, e);
    pl.base_me[e] = b;
  }
  // local experts: rows that will arrive (clamped to the capacity), and each source's share
  for (int el = tid; el < Epr; el += blockDim.x) {
    int e = me * Epr + el, run = 0;
    for (int s = 0; s < P; ++s) {
      pl.src_start[el * (P + 1) + s] = run;
      run += count(s, e);
    }
    pl.src_start[el * (P + 1) + P] = run;
    pl.recv_count[el] = run < cap ? run : cap;
    if (run > cap) atomicAdd(pl.dropped, run - cap);
  }
  __syncthreads();
  // a warp per source, its lanes over the experts (one thread walking 64 experts of the only PE took 12 us)
  const int lane = tid & 31;
  for (int s = tid >> 5; s < P; s += blockDim.x >> 5) {
    // entries of source s that fit into my experts' buffers (what will arrive from s), and my entries that fit into PE s's
    // experts (what comes back from s in the combine)
    int exp_in = 0, out = 0;
    for (int el = lane; el < Epr; el += 32) {
      int a = pl.src_start[el * (P + 1) + s], b = pl.src_start[el * (P + 1) + s + 1];
      exp_in += min(b, cap) - min(a, cap);
      const int e = s * Epr + el;
      a = 0;
      for (int q = 0; q < me; ++q) a += count(q, e);
      b = a + count(me, e);
      out += min(b, cap) - min(a, cap);
    }
    exp_in = __reduce_add_sync(0xffffffffu, exp_in);
    out = __reduce_add_sync(0xffffffffu, out);
    if (lane == 0) {
      pl.expect_from[s] = exp_in;
      pl.send_to[s] = out;
    }
    // recycle the other parity's arrival words for the next call
    if (lane < 4) pl.arrive_sig[(parity ^ 1) * 4 * P + lane * P + s] = 0;
  }
}
__global__ void k_offsets(MoePlanDev pl, const int* __restrict__ counts_all, int parity) {
  ptx::grid_dependency_wait();
  offsets_block(pl, [&](int s, int e) { return __ldcg(counts_all + s * pl.E + e); }, parity);
}
// One PE: its own counts are all there is, so plan and offsets are one launch; the last block to finish (ticket, back
// to zero afterwards) derives the offsets.
__global__ void __launch_bounds__(1024) k_plan_local(MoePlanDev pl, const int* __restrict__ topk_idx, int n_entries, int* __restrict__ pos,
                                                     int* counts, int* counts_all, unsigned int* ticket, int parity) {
  __shared__ bool last;
  ptx::grid_dependency_wait();
  const int total = plan_expert(topk_idx, n_entries, blockIdx.x, pos);
  if (threadIdx.x == 0) {
    counts[blockIdx.x] = total;
    counts_all[blockIdx.x] = total;
    __threadfence();
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (last) offsets_block(pl, [&](int s, int e) { return __ldcg(counts_all + s * pl.E + e); }, parity);
}
// Up to kPlanFew entries: one block, a warp per expert (and 32 further on), everything in shared memory; no ticket and no
// round trips between blocks (8 entries, 16 experts: 4.8 us with a block per expert, 2.9 so; equal at about 512).
constexpr int kPlanFew = 256;
__global__ void __launch_bounds__(1024) k_plan_local_few(MoePlanDev pl, const int* __restrict__ topk_idx, int n_entries, int* __restrict__ pos,
                                                         int* counts, int* counts_all, int parity) {
  __shared__ int ent[kPlanFew];
  __shared__ int cnt[64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ptx::grid_dependency_wait();
  for (int i = threadIdx.x; i < n_entries; i += 1024) ent[i] = __ldcg(topk_idx + i);
  __syncthreads();
  for (int e = warp; e < pl.E; e += 32) {
    int before = 0;
#pragma unroll 4
    for (int i0 = 0; i0 < n_entries; i0 += 32) {
      const int i = i0 + lane;
      const unsigned hits = __ballot_sync(0xffffffffu, i < n_entries && ent[i < n_entries ? i : 0] == e);
      if (hits >> lane & 1) pos[i] = before + __popc(hits & ((1u << lane) - 1));
      before += __popc(hits);
    }
    if (lane == 0) {
      cnt[e] = before;
      counts[e] = before;
      counts_all[e] = before;
    }
  }
  __syncthreads();
  offsets_block(pl, [&](int, int e) { return cnt[e]; }, parity);
}

// ---------------------------------------------------------------------------------------
// dispatch: entry i = token * topk + k  →  row of the destination expert's receive buffer
// ---------------------------------------------------------------------------------------
template <bool kScale>
__global__ void __launch_bounds__(256) k_dispatch(State st, MoePlanDev pl, const bf16* __restrict__ rows, const float* __restrict__ scale,
                                                  const int* __restrict__ topk_idx, const int* __restrict__ pos, int n_entries, int topk,
                                                  int H, char* recv_sym, int* meta_sym, int parity, int which_sig) {
  __shared__ int sent[BSHMEM_MAX_PES];
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  const int Epr = pl.E / pl.P;
  if (threadIdx.x < BSHMEM_MAX_PES) sent[threadIdx.x] = 0;
  __syncthreads();
  const size_t row_bytes = (size_t)H * 2;
  for (int i = blockIdx.x * warps_per_block + (threadIdx.x >> 5); i < n_entries; i += gridDim.x * warps_per_block) {
    int e = topk_idx[i];
    int slot = pl.base_me[e] + pos[i];
    if (slot >= pl.cap) continue;                       // over capacity: dropped (counted in k_offsets)
    int r = e / Epr, el = e - r * Epr;
    const char* src = reinterpret_cast<const char*>(rows) + (size_t)(i / topk) * row_bytes;
    char* dst = dev::ptr(st, recv_sym, r) + ((size_t)el * pl.cap + slot) * row_bytes;
    if (!kScale) {
      dev::copy_bytes<dev::WARP>(dst, src, row_bytes);
    } else {
      const float w = scale[i];
      const uint4* s4 = reinterpret_cast<const uint4*>(src);
      uint4* d4 = reinterpret_cast<uint4*>(dst);
      for (int v = lane; v < H / 8; v += 32) {
        uint4 xv = s4[v];
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&xv);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float2 f = __bfloat1622float2(h[q]);
          h[q] = __floats2bfloat162_rn(f.x * w, f.y * w);
        }
        d4[v] = xv;
      }
    }
    if (lane == 0) {
      if (meta_sym) dev::ptr(st, meta_sym, r)[el * pl.cap + slot] = (pl.me << 26) | i;
      atomicAdd(&sent[r], 1);
    }
  }
  // publish: every warp's stores, then one release-add per destination from this CTA
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x < pl.P && sent[threadIdx.x] > 0) {
    int r = threadIdx.x;
    unsigned long long* sig = dev::ptr(st, pl.arrive_sig, r) + (size_t)parity * 4 * pl.P + (size_t)which_sig * pl.P + pl.me;
    ptx::fence_acq_rel_sys();
    ptx::red_release_sys_add_u64(reinterpret_cast<uint64_t*>(sig), (uint64_t)sent[r]);
  }
}

// Bounded wait until everything this PE expects has arrived (word s counts rows from PE s).
__global__ void k_wait_arrivals(MoePlanDev pl, int parity, int which_sig, const int* __restrict__ expected, unsigned long long timeout_ns,
                                int* err) {
  int s = threadIdx.x;
  if (s >= pl.P) return;
  const unsigned long long* sig = pl.arrive_sig + (size_t)parity * 4 * pl.P + (size_t)which_sig * pl.P + s;
  unsigned long long want = (unsigned long long)expected[s];
  unsigned long long t0 = ptx::globaltimer();
  while (ptx::ld_acquire_sys_u64(reinterpret_cast<const uint64_t*>(sig)) < want) {
    if (ptx::globaltimer() - t0 > timeout_ns) { atomicCAS(err, 0, 201 + which_sig); return; }
    __nanosleep(200);
  }
}

// combine_send: expert PE returns row (el, slot) to the entry buffer of the PE that sent it
__global__ void __launch_bounds__(256) k_combine_send(State st, MoePlanDev pl, const bf16* __restrict__ y, const int* __restrict__ meta,
                                                      int H, char* ybuf_sym, int parity, int which_sig) {
  __shared__ int sent[BSHMEM_MAX_PES];
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  const int Epr = pl.E / pl.P;
  if (threadIdx.x < BSHMEM_MAX_PES) sent[threadIdx.x] = 0;
  __syncthreads();
  const size_t row_bytes = (size_t)H * 2;
  const int total_rows = Epr * pl.cap;
  for (int rix = blockIdx.x * warps_per_block + (threadIdx.x >> 5); rix < total_rows; rix += gridDim.x * warps_per_block) {
    int el = rix / pl.cap, slot = rix - el * pl.cap;
    if (slot >= pl.recv_count[el]) continue;
    int m = meta[rix];
    int src_pe = m >> 26, entry = m & ((1 << 26) - 1);
    char* dst = dev::ptr(st, ybuf_sym, src_pe) + (size_t)entry * row_bytes;
    dev::copy_bytes<dev::WARP>(dst, reinterpret_cast<const char*>(y) + (size_t)rix * row_bytes, row_bytes);
    if (lane == 0) atomicAdd(&sent[src_pe], 1);
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x < pl.P && sent[threadIdx.x] > 0) {
    int r = threadIdx.x;
    unsigned long long* sig = dev::ptr(st, pl.arrive_sig, r) + (size_t)parity * 4 * pl.P + (size_t)which_sig * pl.P + pl.me;
    ptx::fence_acq_rel_sys();
    ptx::red_release_sys_add_u64(reinterpret_cast<uint64_t*>(sig), (uint64_t)sent[r]);
  }
}

// out[token] = sum_k w[entry] * ybuf[entry]   (entries over capacity contribute nothing)
// With `dlog` (backward pass only): out[token] += sum_k dlog[entry] * wr[expert of entry] — the gradient that reaches
// the layer input through the router logits, added here so that d_x is written once.
template <bool kWeighted>
__global__ void k_combine_reduce(MoePlanDev pl, const bf16* __restrict__ ybuf, const float* __restrict__ w, const int* __restrict__ topk_idx,
                                 const int* __restrict__ pos, int T, int topk, int H, bf16* __restrict__ out,
                                 const float* __restrict__ dlog = nullptr, const bf16* __restrict__ wr = nullptr) {
  const int token = blockIdx.x;
  if (token >= T) return;
  for (int v = threadIdx.x; v < H / 8; v += blockDim.x) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int k = 0; k < topk; ++k) {
      int i = token * topk + k;
      int e = topk_idx[i];
      if (pl.base_me[e] + pos[i] >= pl.cap) continue;
      float wk = kWeighted ? w[i] : 1.f;
      uint4 yv = ptx::ld_relaxed_v4(reinterpret_cast<const uint4*>(ybuf + (size_t)i * H) + v);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&yv);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 f = __bfloat1622float2(h[q]);
        acc[2 * q] += wk * f.x;
        acc[2 * q + 1] += wk * f.y;
      }
    }
    if (dlog != nullptr) {
      for (int k = 0; k < topk; ++k) {
        const int i = token * topk + k;
        const float g = dlog[i];
        uint4 wv = __ldg(reinterpret_cast<const uint4*>(wr + (size_t)topk_idx[i] * H) + v);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float2 f = __bfloat1622float2(h[q]);
          acc[2 * q] += g * f.x;
          acc[2 * q + 1] += g * f.y;
        }
      }
    }
    uint4 o;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int q = 0; q < 4; ++q) oh[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
    reinterpret_cast<uint4*>(out + (size_t)token * H)[v] = o;
  }
}

// ---- one PE: every expert is local ---------------------------------------------------------------------------------
// The rows need not leave the GPU: dispatch gathers without signals, and the way back reads the experts' output rows where
// they are (no per-entry return buffer, no arrival words).  One block per token; a row of x or d_out is read once and
// written top-k times.  All vectors of a row that a thread handles are in flight together.  The launches overlap the tail
// of their predecessor (programmatic serialization), so what that may have written is read past the first-level cache.
constexpr int kRowThreads = 128;

// kTop: top-k rounded up to a power of two, so that the loads of a token's rows are issued together.
template <int kTop, bool kGrad>
__global__ void __launch_bounds__(kRowThreads) k_dispatch_local(MoePlanDev pl, const bf16* __restrict__ rows, const int* __restrict__ topk_idx,
                                                                const int* __restrict__ pos, const float* __restrict__ w, int topk, int H,
                                                                bf16* __restrict__ recv, const bf16* __restrict__ y, float* __restrict__ dw,
                                                                float* __restrict__ dlog) {
  // kGrad (backward): the rows go out scaled by their routing weight, and with the experts' outputs y the block also has
  // everything for the routing gradient: dw_k = <y_k, row>, dlog_k = w_k (dw_k - sum_j w_j dw_j)
  __shared__ float part[kTop][kRowThreads / 32];
  const int t = blockIdx.x;
  ptx::grid_dependency_wait();
  size_t slot[kTop];
  float wk[kTop], acc[kTop];
  unsigned live = 0;
#pragma unroll
  for (int k = 0; k < kTop; ++k) {
    acc[k] = 0.f;
    wk[k] = 0.f;
    slot[k] = 0;
    if (k < topk) {
      const int e = __ldcg(topk_idx + t * topk + k), p = __ldcg(pos + t * topk + k);
      if (p < pl.cap) {                              // over capacity: dropped (counted with the offsets)
        live |= 1u << k;
        slot[k] = ((size_t)e * pl.cap + p) * (H / 8);
      }
      if (kGrad) wk[k] = __ldcg(w + t * topk + k);
    }
  }
  const uint4* src = reinterpret_cast<const uint4*>(rows + (size_t)t * H);
  for (int v = threadIdx.x; v < H / 8; v += kRowThreads) {
    uint4 yv[kTop];
    if (kGrad) {                                     // a dead entry reads row 0 and does not count
#pragma unroll
      for (int k = 0; k < kTop; ++k) yv[k] = __ldcg(reinterpret_cast<const uint4*>(y) + slot[k] + v);
    }
    const uint4 xv = __ldcg(src + v);
    const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&xv);
#pragma unroll
    for (int k = 0; k < kTop; ++k) {
      if (!(live >> k & 1)) continue;
      uint4 o = xv;
      if (kGrad) {
        const __nv_bfloat162* yh = reinterpret_cast<const __nv_bfloat162*>(&yv[k]);
        __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 f = __bfloat1622float2(xh[q]), g = __bfloat1622float2(yh[q]);
          oh[q] = __floats2bfloat162_rn(f.x * wk[k], f.y * wk[k]);
          acc[k] += f.x * g.x + f.y * g.y;
        }
      }
      reinterpret_cast<uint4*>(recv)[slot[k] + v] = o;
    }
  }
  if (kGrad) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < kTop; ++k) {
      if (k >= topk) break;
      const float s = warp_sum(acc[k]);
      if (lane == 0) part[k][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      float d[kTop], sum = 0.f;
#pragma unroll
      for (int k = 0; k < kTop; ++k) {
        if (k >= topk) break;
        d[k] = part[k][0] + part[k][1] + part[k][2] + part[k][3];
        dw[t * topk + k] = d[k];
        sum += wk[k] * d[k];
      }
#pragma unroll
      for (int k = 0; k < kTop; ++k) {
        if (k >= topk) break;
        dlog[t * topk + k] = wk[k] * (d[k] - sum);
      }
    }
  }
}

// out[token] = sum_k w_k * y[row of entry k], in k order; backward (kRouter): unweighted, plus sum_k dlog_k * wr[expert k].
// A warp takes a token's 256 columns (16 bytes per lane) at a time, `per` tokens one after the other, with all rows of a
// token in flight together; the lanes hold the token's entries, and the next token's are on their way.  The block's slice of
// wr waits in shared memory: read per token it was as many bytes as y itself.
constexpr int kCombineCols = 256, kCombineWarps = 8;
template <int kTop, bool kRouter>
__global__ void __launch_bounds__(32 * kCombineWarps) k_combine_local(MoePlanDev pl, const bf16* __restrict__ y, const float* __restrict__ w,
                                                                      const int* __restrict__ topk_idx, const int* __restrict__ pos, int T,
                                                                      int topk, int H, int per, bf16* __restrict__ out,
                                                                      const bf16* __restrict__ wr) {
  extern __shared__ __align__(16) char wr_s[];       // kRouter: [E][256 columns]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.y * kCombineCols, nv = min(kCombineCols, H - c0) / 8;
  ptx::grid_dependency_wait();
  if (kRouter) {
    for (int i = threadIdx.x; i < pl.E * 32; i += 32 * kCombineWarps)
      if ((i & 31) < nv) ptx::cp_async_16(ptx::smem_u32(wr_s) + i * 16, wr + (size_t)(i >> 5) * H + c0 + (i & 31) * 8);
    ptx::cp_async_commit();
    ptx::cp_async_wait<0>();
    __syncthreads();
  }
  const int t_first = (blockIdx.x * kCombineWarps + warp) * per, t_end = min(t_first + per, T);
  int e_next = 0, p_next = 0;
  float w_next = 0.f;
  auto fetch = [&](int t) {                          // lane k: entry k of token t (w: routing weight, or dlog)
    if (lane < topk && t < t_end) {
      e_next = __ldcg(topk_idx + (size_t)t * topk + lane);
      p_next = __ldcg(pos + (size_t)t * topk + lane);
      w_next = __ldcg(w + (size_t)t * topk + lane);
    }
  };
  fetch(t_first);
  const uint4* yl = reinterpret_cast<const uint4*>(y + c0) + min(lane, nv - 1);
  for (int t = t_first; t < t_end; ++t) {
    const int e = e_next;
    const float wl = w_next;
    const bool fits = p_next < pl.cap;               // over capacity: contributes nothing
    const unsigned live = __ballot_sync(0xffffffffu, fits && lane < topk);
    const unsigned row = fits ? (unsigned)e * (unsigned)pl.cap + (unsigned)p_next : 0u;
    fetch(t + 1);
    uint4 yv[kTop];
#pragma unroll
    for (int k = 0; k < kTop; ++k) yv[k] = __ldcg(yl + (size_t)__shfl_sync(0xffffffffu, row, k) * (H / 8));
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    auto add = [&](const uint4& v, float f) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 u = __bfloat1622float2(h[q]);
        acc[2 * q] += f * u.x;
        acc[2 * q + 1] += f * u.y;
      }
    };
#pragma unroll
    for (int k = 0; k < kTop; ++k) {
      const float wk = __shfl_sync(0xffffffffu, wl, k);
      if (live >> k & 1) add(yv[k], kRouter ? 1.f : wk);
    }
    if (kRouter) {
#pragma unroll
      for (int k = 0; k < kTop; ++k) {
        const float wk = __shfl_sync(0xffffffffu, wl, k);
        const int ek = __shfl_sync(0xffffffffu, e, k);
        if (k < topk) add(*reinterpret_cast<const uint4*>(wr_s + (ek * 32 + lane) * 16), wk);
      }
    }
    uint4 o;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int q = 0; q < 4; ++q) oh[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
    if (lane < nv) reinterpret_cast<uint4*>(out + (size_t)t * H + c0)[lane] = o;
  }
}

// d_w[entry] = <ybuf[entry], d_out[token]>   (gradient of the routing weight)
__global__ void k_router_weight_grad(MoePlanDev pl, const bf16* __restrict__ ybuf, const bf16* __restrict__ dout, const int* __restrict__ topk_idx,
                                     const int* __restrict__ pos, int n_entries, int topk, int H, float* __restrict__ dw) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n_entries) return;
  float acc = 0.f;
  if (pl.base_me[topk_idx[i]] + pos[i] < pl.cap) {
    const uint4* a = reinterpret_cast<const uint4*>(ybuf + (size_t)i * H);
    const uint4* b = reinterpret_cast<const uint4*>(dout + (size_t)(i / topk) * H);
    for (int v = lane; v < H / 8; v += 32) {
      uint4 av = ptx::ld_relaxed_v4(a + v), bv = b[v];
      const __nv_bfloat162* ah = reinterpret_cast<const __nv_bfloat162*>(&av);
      const __nv_bfloat162* bh = reinterpret_cast<const __nv_bfloat162*>(&bv);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 x = __bfloat1622float2(ah[q]), y = __bfloat1622float2(bh[q]);
        acc += x.x * y.x + x.y * y.y;
      }
    }
  }
  acc = warp_sum(acc);
  if (lane == 0) dw[i] = acc;
}

// Router backward.  The routing weights are a softmax over the chosen experts' logits (softmax over all experts,
// renormalised over the top-k), so only the chosen logits receive a gradient:
//   d_logit[entry k] = w_k * (d_w_k - sum_j w_j * d_w_j)
__global__ void k_router_dlogits(const float* __restrict__ w, const float* __restrict__ dw, int T, int topk, float* __restrict__ dlog) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  float s = 0.f;
  for (int k = 0; k < topk; ++k) s += w[t * topk + k] * dw[t * topk + k];
  for (int k = 0; k < topk; ++k) dlog[t * topk + k] = w[t * topk + k] * (dw[t * topk + k] - s);
}

// d_Wr[e, :] += sum over the CTA's tokens routed to e of d_logit * x[token, :]   (fp32 accumulation, atomics across CTAs).
// A CTA stages `tok` rows x 256 columns of x in shared memory and sorts its (token, k) entries by expert meanwhile; its
// warps then take equal shares of the sorted entries, with eight columns to a lane, and add a sum to global memory whenever
// the expert changes.  So x is read once, all of a CTA's loads are in flight together, and neither the number of experts
// nor an uneven routing leaves warps idle (with all warps walking the experts one after the other, every expert cost a
// round trip: 300 tokens, 64 experts, top-8: 191 us; 16384 tokens of 4096, 8 experts, top-2: 146 us).
constexpr int kDwrTok = 128, kDwrCols = 256, kDwrPitch = kDwrCols * 2 + 16;       // bytes per staged row
constexpr uint32_t kDwrSmem = kDwrTok * kDwrPitch;
__global__ void __launch_bounds__(256) k_router_dwr(const bf16* __restrict__ x, const int* __restrict__ topk_idx, const float* __restrict__ dlog,
                                                   int T, int H, int E, int topk, int tok, float* __restrict__ dwr) {
  extern __shared__ __align__(16) char rows[];
  __shared__ int cnt[64], fill[64];
  __shared__ unsigned short ent[kDwrTok * 8];            // sorted entries: token << 6 | expert
  __shared__ float grad[kDwrTok * 8];
  const int t0 = blockIdx.x * tok, nt = min(tok, T - t0), n_ent = nt * topk;
  const int c0 = blockIdx.y * kDwrCols, nv = min(kDwrCols, H - c0) / 8;      // 16-byte pieces per staged row
  const uint32_t rows_a = ptx::smem_u32(rows);
  if (threadIdx.x < 64) cnt[threadIdx.x] = 0;
  ptx::grid_dependency_wait();
  for (int i = threadIdx.x; i < nt * 32; i += 256) {
    const int r = i >> 5, v = i & 31;
    if (v < nv) ptx::cp_async_16(rows_a + r * kDwrPitch + v * 16, x + (size_t)(t0 + r) * H + c0 + v * 8);
  }
  ptx::cp_async_commit();
  __syncthreads();
  for (int i = threadIdx.x; i < n_ent; i += 256) atomicAdd(&cnt[topk_idx[(size_t)t0 * topk + i]], 1);
  __syncthreads();
  if (threadIdx.x < 32) {                                // exclusive scan over 64 counts
    const int c_lo = cnt[2 * threadIdx.x], c_hi = cnt[2 * threadIdx.x + 1];
    int incl = c_lo + c_hi;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)threadIdx.x >= o) incl += up;
    }
    fill[2 * threadIdx.x] = incl - c_lo - c_hi;
    fill[2 * threadIdx.x + 1] = incl - c_hi;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n_ent; i += 256) {
    const int e = topk_idx[(size_t)t0 * topk + i], at = atomicAdd(&fill[e], 1);
    ent[at] = (unsigned short)(i / topk << 6 | e);
    grad[at] = dlog[(size_t)t0 * topk + i];
  }
  ptx::cp_async_wait<0>();
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane >= nv) return;
  const int i0 = n_ent * warp / 8, i1 = n_ent * (warp + 1) / 8;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  auto flush = [&](int e) {
    float4* dst = reinterpret_cast<float4*>(dwr + (size_t)e * H + c0 + lane * 8);
    atomicAdd(dst, make_float4(acc[0], acc[1], acc[2], acc[3]));
    atomicAdd(dst + 1, make_float4(acc[4], acc[5], acc[6], acc[7]));
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  };
  int e_now = i0 < i1 ? ent[i0] & 63 : 0;
#pragma unroll 4
  for (int i = i0; i < i1; ++i) {
    const int v = ent[i];
    const float g = grad[i];
    const uint4 raw = *reinterpret_cast<const uint4*>(rows + (v >> 6) * kDwrPitch + lane * 16);
    if ((v & 63) != e_now) { flush(e_now); e_now = v & 63; }
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 f = __bfloat1622float2(h[q]);
      acc[2 * q] += g * f.x;
      acc[2 * q + 1] += g * f.y;
    }
  }
  if (i0 < i1) flush(e_now);
}

__global__ void k_f32_to_bf16(const float* __restrict__ in, bf16* __restrict__ out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) out[i] = __float2bfloat16_rn(in[i]);
}

// ---------------------------------------------------------------------------------------
// SwiGLU on the interleaved gate/up layout: every 64 columns = 32 gate followed by 32 up
// ---------------------------------------------------------------------------------------
__global__ void k_swiglu_fwd(const bf16* __restrict__ gu, const int* __restrict__ counts, int cap, int F, bf16* __restrict__ h) {
  const int row = blockIdx.x;
  const int el = row / cap;
  if (row - el * cap >= counts[el]) return;
  const bf16* g = gu + (size_t)row * 2 * F;
  bf16* o = h + (size_t)row * F;
  for (int c = threadIdx.x; c < F / 8; c += blockDim.x) {     // 8 outputs per thread
    int blk = (c * 8) / 32, in = (c * 8) % 32;
    uint4 gv = *reinterpret_cast<const uint4*>(g + blk * 64 + in);
    uint4 uv = *reinterpret_cast<const uint4*>(g + blk * 64 + 32 + in);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv);
    const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&uv);
    uint4 ov;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float2 gf = __bfloat1622float2(gh[q]), uf = __bfloat1622float2(uh[q]);
      oh[q] = __floats2bfloat162_rn(gf.x / (1.f + __expf(-gf.x)) * uf.x, gf.y / (1.f + __expf(-gf.y)) * uf.y);
    }
    *reinterpret_cast<uint4*>(o + c * 8) = ov;
  }
}

// d_gu (interleaved) from d_h and the saved pre-activations
__global__ void k_swiglu_bwd(const bf16* __restrict__ gu, const bf16* __restrict__ dh, const int* __restrict__ counts, int cap, int F,
                             bf16* __restrict__ dgu) {
  const int row = blockIdx.x;
  const int el = row / cap;
  if (row - el * cap >= counts[el]) return;
  const bf16* g = gu + (size_t)row * 2 * F;
  const bf16* d = dh + (size_t)row * F;
  bf16* o = dgu + (size_t)row * 2 * F;
  for (int c = threadIdx.x; c < F / 8; c += blockDim.x) {
    int blk = (c * 8) / 32, in = (c * 8) % 32;
    uint4 gv = *reinterpret_cast<const uint4*>(g + blk * 64 + in);
    uint4 uv = *reinterpret_cast<const uint4*>(g + blk * 64 + 32 + in);
    uint4 dv = *reinterpret_cast<const uint4*>(d + c * 8);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv);
    const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&uv);
    const __nv_bfloat162* dhh = reinterpret_cast<const __nv_bfloat162*>(&dv);
    uint4 og, ou;
    __nv_bfloat162* ogh = reinterpret_cast<__nv_bfloat162*>(&og);
    __nv_bfloat162* ouh = reinterpret_cast<__nv_bfloat162*>(&ou);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float2 gf = __bfloat1622float2(gh[q]), uf = __bfloat1622float2(uh[q]), df = __bfloat1622float2(dhh[q]);
      float sx = 1.f / (1.f + __expf(-gf.x)), sy = 1.f / (1.f + __expf(-gf.y));
      float silx = gf.x * sx, sily = gf.y * sy;
      // d silu(g)/dg = s * (1 + g * (1 - s))
      ogh[q] = __floats2bfloat162_rn(df.x * uf.x * sx * (1.f + gf.x * (1.f - sx)), df.y * uf.y * sy * (1.f + gf.y * (1.f - sy)));
      ouh[q] = __floats2bfloat162_rn(df.x * silx, df.y * sily);
    }
    *reinterpret_cast<uint4*>(o + blk * 64 + in) = og;
    *reinterpret_cast<uint4*>(o + blk * 64 + 32 + in) = ou;
  }
}

// out[c][r] = in[r][c] for r < rows_valid (per expert region), zero for rows_valid <= r < ld_out:
// the zero padding makes the ragged K extent of the weight-gradient GEMMs harmless.
__global__ void k_transpose_pad(const bf16* __restrict__ in, const int* __restrict__ counts, int cap, int cols, bf16* __restrict__ out) {
  __shared__ bf16 tile[32][33];
  const int el = blockIdx.z;
  const int valid = counts[el];
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  const bf16* src = in + (size_t)el * cap * cols;
  bf16* dst = out + (size_t)el * cols * cap;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    int r = r0 + j, c = c0 + threadIdx.x;
    tile[j][threadIdx.x] = (r < valid && c < cols) ? src[(size_t)r * cols + c] : __float2bfloat16(0.f);
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    int c = c0 + j, r = r0 + threadIdx.x;
    if (c < cols && r < cap) dst[(size_t)c * cap + r] = tile[threadIdx.x][j];
  }
}

// Threads of a plan block: 128 entries per warp as long as that is less than a full block.
int plan_threads(int n_entries) {
  const int warps = (n_entries + 127) / 128;
  return 32 * (warps < 1 ? 1 : (warps > 32 ? 32 : warps));
}

// Launch that may overlap the tail of the stream's previous kernel; `k` calls ptx::grid_dependency_wait() first thing.
template <class... P, class... A>
cudaError_t launch_pdl_smem(void (*k)(P...), dim3 grid, dim3 block, uint32_t smem, void* stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.dynamicSmemBytes = smem;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, static_cast<P>(std::forward<A>(args))...);
}
template <class... P, class... A>
cudaError_t launch_pdl(void (*k)(P...), dim3 grid, dim3 block, void* stream, A&&... args) {
  return launch_pdl_smem(k, grid, block, 0, stream, std::forward<A>(args)...);
}

// The instance of a kernel for top-k rounded up to a power of two.
template <class K>
K by_top(int topk, K k1, K k2, K k4, K k8) { return topk <= 1 ? k1 : topk <= 2 ? k2 : topk <= 4 ? k4 : k8; }

thread_local std::string g_err;
#define RT_TRY(call) do { cudaError_t _e = (call); if (_e != cudaSuccess) { g_err = std::string(#call) + ": " + cudaGetErrorString(_e); return 7; } } while (0)

}  // namespace

extern "C" {

const char* bshmem_moe_last_error() { return g_err.c_str(); }

int bshmem_moe_router_topk(const void* x, const void* wr, int T, int H, int E, int topk, int* topk_idx, float* topk_w, float* probs,
                           void* stream) {
  if (E > 64 || topk > 8 || topk > E || H % 8) { g_err = "router: E <= 64, topk <= min(8, E), H % 8 == 0"; return 1; }
  if (T <= 0) return 0;
  const int blocks = (T + kRouterTok - 1) / kRouterTok;
  const bool few = blocks <= 148;
  auto k = E <= 8 ? (few ? k_router_topk<1, 16> : k_router_topk<1, 8>) : E <= 16 ? (few ? k_router_topk<2, 16> : k_router_topk<2, 8>)
           : E <= 32 ? (few ? k_router_topk<4, 16> : k_router_topk<4, 8>) : (few ? k_router_topk<8, 16> : k_router_topk<8, 8>);
  RT_TRY(launch_pdl(k, dim3(blocks), dim3(few ? 512 : 256), stream, (const bf16*)x, (const bf16*)wr, T, H, E, topk, topk_idx, topk_w, probs));
  return 0;
}

// topk_idx: 16-byte aligned
int bshmem_moe_plan(const int* topk_idx, int n_entries, int E, int* pos, int* counts, void* stream) {
  RT_TRY(launch_pdl(k_plan, dim3(E), dim3(plan_threads(n_entries)), stream, topk_idx, n_entries, pos, counts));
  return 0;
}

int bshmem_moe_offsets(const MoePlanDev* pl, const int* counts_all, int parity, void* stream) {
  RT_TRY(launch_pdl(k_offsets, dim3(1), dim3(128), stream, *pl, counts_all, parity));
  return 0;
}

// One PE: plan and offsets in one launch.  `ticket` is a zeroed word that the call leaves zero.
int bshmem_moe_plan_local(const MoePlanDev* pl, const int* topk_idx, int n_entries, int* pos, int* counts, int* counts_all,
                          unsigned int* ticket, int parity, void* stream) {
  if (pl->P != 1) { g_err = "plan_local: more than one PE"; return 1; }
  if (n_entries <= kPlanFew && pl->E <= 64) {
    RT_TRY(launch_pdl(k_plan_local_few, dim3(1), dim3(1024), stream, *pl, topk_idx, n_entries, pos, counts, counts_all, parity));
    return 0;
  }
  RT_TRY(launch_pdl(k_plan_local, dim3(pl->E), dim3(plan_threads(n_entries)), stream, *pl, topk_idx, n_entries, pos, counts, counts_all, ticket,
                    parity));
  return 0;
}

// One PE: rows of x to their experts' buffers.
int bshmem_moe_dispatch_local(const MoePlanDev* pl, const void* rows, const int* topk_idx, const int* pos, int T, int topk, int H, void* recv,
                              void* stream) {
  if (pl->P != 1 || H % 8 || topk > 8) { g_err = "dispatch_local: one PE, H % 8 == 0, at most top-8"; return 1; }
  RT_TRY(launch_pdl(by_top(topk, k_dispatch_local<1, false>, k_dispatch_local<2, false>, k_dispatch_local<4, false>, k_dispatch_local<8, false>),
                    dim3(T), dim3(kRowThreads), stream, *pl, (const bf16*)rows, topk_idx, pos, nullptr, topk, H, (bf16*)recv, nullptr, nullptr,
                    nullptr));
  return 0;
}
// One PE, backward: w * d_out to the experts' gradient buffers, and the gradients of the routing weights (dw) and of the
// chosen experts' logits (dlog) from the experts' outputs y of the forward pass.
int bshmem_moe_dispatch_grad_local(const MoePlanDev* pl, const void* dout, const int* topk_idx, const int* pos, const float* w, int T, int topk,
                                   int H, void* recv, const void* y, float* dw, float* dlog, void* stream) {
  if (pl->P != 1 || H % 8 || topk > 8) { g_err = "dispatch_local: one PE, H % 8 == 0, at most top-8"; return 1; }
  RT_TRY(launch_pdl(by_top(topk, k_dispatch_local<1, true>, k_dispatch_local<2, true>, k_dispatch_local<4, true>, k_dispatch_local<8, true>),
                    dim3(T), dim3(kRowThreads), stream, *pl, (const bf16*)dout, topk_idx, pos, w, topk, H, (bf16*)recv,
                    (const bf16*)y, dw, dlog));
  return 0;
}
// One PE: out = sum over k of w_k times the expert's output row; with `wr`, w holds the logit gradients instead and out
// gets the unweighted rows plus w_k times the expert's row of wr.
int bshmem_moe_combine_local(const MoePlanDev* pl, const void* y, const float* w, const int* topk_idx, const int* pos, int T, int topk, int H,
                             void* out, const void* wr, void* stream) {
  if (pl->P != 1 || H % 8 || topk > 8) { g_err = "combine_local: one PE, H % 8 == 0, at most top-8"; return 1; }
  auto k = wr ? by_top(topk, k_combine_local<1, true>, k_combine_local<2, true>, k_combine_local<4, true>, k_combine_local<8, true>)
              : by_top(topk, k_combine_local<1, false>, k_combine_local<2, false>, k_combine_local<4, false>, k_combine_local<8, false>);
  // four tokens per warp share the block's slice of wr and hide the entries' round trip; one while that fills the chip better
  const int col_blocks = (H + kCombineCols - 1) / kCombineCols;
  const int per = (long long)T * col_blocks >= 4ll * kCombineWarps * 4 * 148 ? 4 : 1;
  RT_TRY(launch_pdl_smem(k, dim3((T + kCombineWarps * per - 1) / (kCombineWarps * per), col_blocks), dim3(32 * kCombineWarps),
                         wr ? (uint32_t)pl->E * 512u : 0u, stream, *pl, (const bf16*)y, w, topk_idx, pos, T, topk, H, per, (bf16*)out,
                         (const bf16*)wr));
  return 0;
}

// rows: [T, H] bf16 token rows (x, or d_out in the backward pass with scale = routing weights)
int bshmem_moe_dispatch(const bshmem_dev_state_t* st, const MoePlanDev* pl, const void* rows, const float* scale, const int* topk_idx,
                        const int* pos, int n_entries, int topk, int H, void* recv_sym, int* meta_sym, int parity, int which_sig, int ctas,
                        void* stream) {
  if (H % 8) { g_err = "dispatch: H % 8 != 0"; return 1; }
  if (ctas < 1) ctas = 1;
  if (scale)
    k_dispatch<true><<<ctas, 256, 0, (cudaStream_t)stream>>>(*st, *pl, (const bf16*)rows, scale, topk_idx, pos, n_entries, topk, H,
                                                             (char*)recv_sym, meta_sym, parity, which_sig);
  else
    k_dispatch<false><<<ctas, 256, 0, (cudaStream_t)stream>>>(*st, *pl, (const bf16*)rows, nullptr, topk_idx, pos, n_entries, topk, H,
                                                              (char*)recv_sym, meta_sym, parity, which_sig);
  RT_TRY(cudaGetLastError());
  return 0;
}

int bshmem_moe_wait_arrivals(const MoePlanDev* pl, int parity, int which_sig, const int* expected, int timeout_ms, int* err, void* stream) {
  k_wait_arrivals<<<1, 32, 0, (cudaStream_t)stream>>>(*pl, parity, which_sig, expected, (unsigned long long)timeout_ms * 1000000ull, err);
  RT_TRY(cudaGetLastError());
  return 0;
}

int bshmem_moe_combine_send(const bshmem_dev_state_t* st, const MoePlanDev* pl, const void* y, const int* meta, int H, void* ybuf_sym,
                            int parity, int which_sig, int ctas, void* stream) {
  if (ctas < 1) ctas = 1;
  k_combine_send<<<ctas, 256, 0, (cudaStream_t)stream>>>(*st, *pl, (const bf16*)y, meta, H, (char*)ybuf_sym, parity, which_sig);
  RT_TRY(cudaGetLastError());
  return 0;
}

int bshmem_moe_combine_reduce(const MoePlanDev* pl, const void* ybuf, const float* w, const int* topk_idx, const int* pos, int T, int topk,
                              int H, void* out, void* stream) {
  if (w) k_combine_reduce<true><<<T, 256, 0, (cudaStream_t)stream>>>(*pl, (const bf16*)ybuf, w, topk_idx, pos, T, topk, H, (bf16*)out);
  else k_combine_reduce<false><<<T, 256, 0, (cudaStream_t)stream>>>(*pl, (const bf16*)ybuf, nullptr, topk_idx, pos, T, topk, H, (bf16*)out);
  RT_TRY(cudaGetLastError());
  return 0;
}

// The same reduction for the backward pass's closing step, plus the router term (see k_combine_reduce).
int bshmem_moe_combine_reduce_router(const MoePlanDev* pl, const void* ybuf, const int* topk_idx, const int* pos, int T, int topk, int H,
                                     void* out, const float* dlog, const void* wr, void* stream) {
  k_combine_reduce<false><<<T, 256, 0, (cudaStream_t)stream>>>(*pl, (const bf16*)ybuf, nullptr, topk_idx, pos, T, topk, H, (bf16*)out, dlog,
                                                                (const bf16*)wr);
  RT_TRY(cudaGetLastError());
  return 0;
}

// Router backward: d_logits of the chosen experts [T * topk] from the routing weights and their gradient, then
// d_Wr [E, H] = d_logits^T · x (accumulated in the fp32 scratch `dwr_f32`, which this call clears first) as bf16.
int bshmem_moe_router_backward(const void* x, const int* topk_idx, const float* topk_w, const float* dtopk_w, int T, int H, int E, int topk,
                               float* dlog, float* dwr_f32, void* dwr, void* stream) {
  if (E > 64 || topk > 8 || H % 8) { g_err = "router backward: at most 64 experts, top-8, H % 8 == 0"; return 1; }
  cudaStream_t st = (cudaStream_t)stream;
  if (topk_w) {                        // null: dlog is already there (bshmem_moe_dispatch_grad_local)
    k_router_dlogits<<<(T + 255) / 256, 256, 0, st>>>(topk_w, dtopk_w, T, topk, dlog);
    RT_TRY(cudaGetLastError());
  }
  RT_TRY(cudaMemsetAsync(dwr_f32, 0, sizeof(float) * (size_t)E * H, st));
  // fewer tokens to a CTA while that leaves multiprocessors idle (each CTA adds up to E x 256 sums at its end)
  const int col_blocks = (H + kDwrCols - 1) / kDwrCols;
  int tok = kDwrTok;
  while (tok > 16 && (long long)((T + tok - 1) / tok) * col_blocks < 148) tok /= 2;
  static std::once_flag once[64];
  int dev = 0;
  RT_TRY(cudaGetDevice(&dev));
  std::call_once(once[dev & 63], [] { cudaFuncSetAttribute(k_router_dwr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDwrSmem); });
  RT_TRY(launch_pdl_smem(k_router_dwr, dim3((T + tok - 1) / tok, col_blocks), dim3(256), (uint32_t)(tok * kDwrPitch), stream, (const bf16*)x, topk_idx, (const float*)dlog, T, H, E, topk,
                    tok, dwr_f32));
  k_f32_to_bf16<<<64, 256, 0, st>>>(dwr_f32, (bf16*)dwr, (size_t)E * H);
  RT_TRY(cudaGetLastError());
  return 0;
}

int bshmem_moe_router_weight_grad(const MoePlanDev* pl, const void* ybuf, const void* dout, const int* topk_idx, const int* pos, int n_entries,
                                  int topk, int H, float* dw, void* stream) {
  int threads = 256, blocks = (n_entries * 32 + threads - 1) / threads;
  k_router_weight_grad<<<blocks, threads, 0, (cudaStream_t)stream>>>(*pl, (const bf16*)ybuf, (const bf16*)dout, topk_idx, pos, n_entries, topk, H, dw);
  RT_TRY(cudaGetLastError());
  return 0;
}

int bshmem_moe_swiglu_fwd(const void* gu, const int* counts, int groups, int cap, int F, void* h, void* stream) {
  if (F % 32) { g_err = "swiglu: F % 32 != 0"; return 1; }
  k_swiglu_fwd<<<groups * cap, 256, 0, (cudaStream_t)stream>>>((const bf16*)gu, counts, cap, F, (bf16*)h);
  RT_TRY(cudaGetLastError());
  return 0;
}

int bshmem_moe_swiglu_bwd(const void* gu, const void* dh, const int* counts, int groups, int cap, int F, void* dgu, void* stream) {
  if (F % 32) { g_err = "swiglu: F % 32 != 0"; return 1; }
  k_swiglu_bwd<<<groups * cap, 256, 0, (cudaStream_t)stream>>>((const bf16*)gu, (const bf16*)dh, counts, cap, F, (bf16*)dgu);
  RT_TRY(cudaGetLastError());
  return 0;
}

// in: [groups][cap][cols] → out: [groups][cols][cap], rows beyond counts[g] become zero columns
int bshmem_moe_transpose_pad(const void* in, const int* counts, int groups, int cap, int cols, void* out, void* stream) {
  dim3 grid((cols + 31) / 32, (cap + 31) / 32, groups), block(32, 8);
  k_transpose_pad<<<grid, block, 0, (cudaStream_t)stream>>>((const bf16*)in, counts, cap, cols, (bf16*)out);
  RT_TRY(cudaGetLastError());
  return 0;
}

}  // extern "C"
