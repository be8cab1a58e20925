// coll_kernels_impl.cuh — body of one collective-kernel translation unit.  The including .cu defines
//   COLL_UNIT        name of the unit (move, f32, ...)
//   COLL_TYPES(X)    X(dtype code, C type) for every element type the unit reduces (empty for `move`)
// and gets a per-PE kernel, the kernels of a local group and their launchers (see coll_kernels.h).
#include "../include/bshmem_coll.cuh"
#include "../include/bshmem_gpu.h"
#include "coll_kernels.h"

namespace bshmem {
namespace collk {
namespace {

#ifdef COLL_UNIT_MOVE
constexpr int kThreads = kMoveThreads;
#else
constexpr int kThreads = kReduceThreads;
#endif

#define COLL_CAT2(a, b) a##b
#define COLL_CAT(a, b) COLL_CAT2(a, b)

// dynamic shared memory: the staging rings of coll::reduce_bulk and of the bulk moves.  A move gets its ring only where it
// is used and all blocks are resident with it (one to a multiprocessor).
#ifndef COLL_UNIT_MOVE
constexpr uint32_t kDynSmem = coll::kBulkSmemBytes;
// without it where no block reduces enough for the ring (its share of the vector, or of a PE's part of it)
uint32_t dyn_smem(const CollArgs& a, int ctas, int) { return a.n * bshmem_dtype_size(a.dtype) / ctas + 16 >= coll::kBulkMinBytes ? kDynSmem : 0; }
#else
constexpr uint32_t kDynSmem = coll::kMoveSmemBytes;
uint32_t dyn_smem(const CollArgs& a, int ctas, int blocks) {
  int dev = 0, sms = 0;
  if (!wants_move_ring(a, ctas, coll::kMoveMinBytes) || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || blocks > sms)
    return 0;
  return kDynSmem;
}
#endif
__device__ __forceinline__ char* ring_smem() {
  extern __shared__ __align__(128) char coll_dyn_smem[];
  uint32_t bytes;
  asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(bytes));
  return bytes >= kDynSmem ? coll_dyn_smem : nullptr;
}

template <typename T>
__device__ int reduce_typed(const State& s, const DTeam& t, const CollArgs& a, int cta, int ncta) {
  char* bulk = ring_smem();
  T* d = reinterpret_cast<T*>(s.heap_base[s.my_pe] + a.dst_off);
  const T* src = reinterpret_cast<const T*>(s.heap_base[s.my_pe] + a.src_off);
  if (a.kind == BSHMEM_COLL_REDUCE_ROOT) return coll::team_reduce_root<T>(s, t, a.op, d, src, a.n, a.root, cta, ncta, bulk);
  if (a.kind == BSHMEM_COLL_REDUCE_SCATTER) {
    if constexpr (std::is_same<T, float>::value || std::is_same<T, __nv_bfloat16>::value) {
      // large sums on the whole world: the switch reduces (see the allreduce below)
      if (a.use_nvls && s.mc_base && t.size == s.n_pes && a.op == BSHMEM_SUM && ((a.dst_off | a.src_off) & 15) == 0 &&
          (a.n * sizeof(T)) % 16 == 0 && !a.stage_seq)
        return coll::team_reduce_scatter_nvls<T>(s, t, d, src, a.n, cta, ncta);
    }
    if (a.stage_seq) return coll::team_reduce_scatter_staged<T>(s, t, a.op, d, src, a.n, a.stage_seq, cta, ncta, bulk);
    return coll::team_reduce_scatter<T>(s, t, a.op, d, src, a.n, cta, ncta, bulk);
  }
  if constexpr (std::is_same<T, float>::value || std::is_same<T, __nv_bfloat16>::value) {
    // the multicast mapping spans every PE, so the in-switch reduction only fits a team that is the whole world
    // (small vectors stay on the one-exchange slots: a switch round trip per vector only pays off in bandwidth)
    if (a.use_nvls && s.mc_base && t.size == s.n_pes && a.op == BSHMEM_SUM && ((a.dst_off | a.src_off) & 15) == 0 &&
        (a.n * sizeof(T)) % 16 == 0 && a.ll_epoch == 0 && a.n * sizeof(T) > BSHMEM_LLB_PAYLOAD_BYTES)
      return coll::team_reduce_nvls<T>(s, t, d, src, a.n, cta, ncta);
  }
  if (a.stage_seq && a.stage_oneshot) return coll::team_reduce_staged_oneshot<T>(s, t, a.op, d, src, a.n, a.stage_seq, cta, ncta, bulk);
  if (a.stage_seq) return coll::team_reduce_staged<T>(s, t, a.op, d, src, a.n, a.stage_seq, cta, ncta, bulk);
  return coll::team_reduce<T>(s, t, a.op, d, src, a.n, cta, ncta, a.ll_epoch, bulk);
}

__device__ __noinline__ int run_coll(const State& s, DTeam t, const CollArgs& a, int cta, int ncta) {
  char* base = s.heap_base[s.my_pe];
  if (t.slot < 0) t.psync = reinterpret_cast<long*>(base + a.psync_off);
  switch (a.kind) {
#ifdef COLL_UNIT_MOVE
    case BSHMEM_COLL_SYNC: return coll::team_sync(s, t, cta);
    case BSHMEM_COLL_BARRIER: return coll::team_barrier(s, t, cta);
    case BSHMEM_COLL_BROADCAST: return coll::team_broadcast(s, t, base + a.dst_off, base + a.src_off, a.n, a.root, cta, ncta);
    case BSHMEM_COLL_FCOLLECT:
      if (a.stage_seq) return coll::team_fcollect_staged(s, t, base + a.dst_off, base + a.src_off, a.n, a.stage_seq, a.use_nvls, cta, ncta);
      return coll::team_fcollect(s, t, base + a.dst_off, base + a.src_off, a.n, cta, ncta, ring_smem());
    case BSHMEM_COLL_ALLTOALL:
      if (a.stage_seq) return coll::team_alltoall_staged(s, t, base + a.dst_off, base + a.src_off, a.n, a.stage_seq, cta, ncta);
      return coll::team_alltoall(s, t, base + a.dst_off, base + a.src_off, a.n, cta, ncta, ring_smem());
    case BSHMEM_COLL_EXCHANGE: {
      // publish one u64 (held in a.n) in every member's exchange row, sync, leave the row for the host
      if (threadIdx.x < t.size) {
        uint64_t* row = reinterpret_cast<uint64_t*>(s.heap_base[dev::team_pe(t, threadIdx.x)] + BSHMEM_OFF_XCHG) +
                        (size_t)t.slot * BSHMEM_MAX_PES;
        row[t.my_idx] = a.n;
      }
      int rc = coll::team_barrier(s, t, cta);
      if (rc != BSHMEM_OK) return rc;
      return coll::team_sync(s, t, cta);   // nobody overwrites a row that is still being read... by the next exchange
    }
#endif
    case BSHMEM_COLL_REDUCE: case BSHMEM_COLL_REDUCE_SCATTER: case BSHMEM_COLL_REDUCE_ROOT:
      switch (a.dtype) {
#define COLL_CASE(code, T) case code: return reduce_typed<T>(s, t, a, cta, ncta);
        COLL_TYPES(COLL_CASE)
#undef COLL_CASE
      }
      return BSHMEM_ERR_UNSUPPORTED;
  }
  return BSHMEM_ERR_INVALID;
}

__global__ void __launch_bounds__(kThreads) COLL_CAT(k_coll_, COLL_UNIT)(State s, DTeam t, CollArgs a, int* status) {
  int rc = run_coll(s, t, a, blockIdx.x, gridDim.x);
  if (rc != BSHMEM_OK && threadIdx.x == 0) atomicCAS(status, 0, rc);
}

// The status is in host memory: a block that failed has it there before it is counted, so that the word that says that all are
// done needs no fence of system scope (results are in this GPU's memory).
__device__ __forceinline__ void group_failed(int* status, int rc) {
  atomicCAS_system(status, 0, rc);
  __threadfence_system();
}

// All PEs of a local group in ONE cooperative launch: blockIdx.y is the PE.  Runs the multi-PE algorithms, flag exchanges
// included, on a single GPU (kernels that wait on one another must not be separate launches on one device): syncs, and what is
// no pass (below).
// The block works on a copy of its PE's state in shared memory (a private copy is 220 bytes of local memory per thread).
__global__ void __launch_bounds__(kThreads) COLL_CAT(k_coll_group_, COLL_UNIT)(const State* states, const DTeam* teams,
                                                                                CollArgs a, int* status, GroupDone done) {
  static_assert(sizeof(State) % 4 == 0, "copied in words");
  __shared__ State s;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(states + blockIdx.y);
  for (unsigned i = threadIdx.x; i < sizeof(State) / 4; i += kThreads) reinterpret_cast<uint32_t*>(&s)[i] = src[i];
  const DTeam t = teams[blockIdx.y];
  __syncthreads();
  if (t.my_idx >= 0) {
    const int rc = run_coll(s, t, a, blockIdx.x, gridDim.x);
    if (rc != BSHMEM_OK && threadIdx.x == 0) group_failed(status, rc);
  }
  if (done.word == nullptr) return;
  // the last block to get here tells the host; the count is back at zero then
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();                       // a system fence per block took 4 us; the blocks of a group share the GPU
    const unsigned n = gridDim.x * gridDim.y;
    if (atomicInc(done.count, n - 1) == n - 1) {
      __threadfence();
      asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(done.word), "l"(done.token) : "memory");
    }
  }
}

// ---- the group as one pass (GroupPass) ----
// Bound by the launch and one round trip to memory where little is moved, by HBM beyond.  Before: up to eight blocks as a cluster with
// two barriers, more of them cooperatively with two flag exchanges, large reductions staged through shared memory.  Whole calls, before
// and now, us: allreduce 16 KiB fp32, 4 PEs 14.9 -> 9.6; 1 MiB bf16, 8 PEs 23.4 -> 12.6; 32 MiB fp32, 8 PEs 117 -> 103; reduce-scatter
// 32 MiB bf16, 8 PEs 83.7 -> 59.8 (302 MB, 46 at the copy rate), 32 MiB fp32, 4 PEs 50.0 -> 39.8; fcollect 16 MiB, 8 PEs 44.4 -> 38.4;
// alltoall 32 MiB, 8 PEs 110 -> 98, 2 MiB, 4 PEs 20.1 -> 12.3.
// 512 threads; a reduction has up to 16 loads of 16 bytes on their way per thread, and so 128 KB per block, a move eight; a block to a
// multiprocessor, as many as the caller asked for.  24 MB per PE in 128 blocks, us, staged as before / one vector at a time for numbers of members
// other than 2, 4 and 8 and for the rarer types and operators / so:  fp32 sum, 3 / 6 / 7 PEs 48.5 / 49.5 / 37.9, 76 / 88 / 68, 90 / 95 / 78; int16
// maximum, 2 PEs 36.4 / 53 / 23.5; fp32 product, 8 PEs 135 / 102 / 83; reduce-scatter of int8 sums, 5 PEs 67 / 63 / 40.  One vector
// at a time is still the better way for the rarer operators on eight bytes: AND of 7 PEs 141 / 73, two at a time 78.
constexpr int kPassThreads = 512;

__device__ __forceinline__ State pass_state(const GroupPass& g) {      // what the counters and the trace take of a state
  State s;
  s.stats = g.stats[blockIdx.y];
  s.my_pe = g.pe[blockIdx.y];
  return s;
}
// The launch's blocks are counted, and the last one tells the host; a few blocks each tell it themselves, which spares the way to the
// counter and back.  A system fence per block took 4 us; the group shares the GPU.
__device__ __forceinline__ void pass_end(const GroupPass& g, unsigned long long cap, unsigned long long traced_bytes) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const State s = pass_state(g);
    dev::stat(s, BSHMEM_DSTAT_COLL);
    dev::trace_with(s, cap, BSHMEM_TRACE_COLL, s.my_pe, traced_bytes);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned n = gridDim.x * gridDim.y;
    uint64_t* word = g.done.word;
    if (g.done.count == nullptr) {
      word += blockIdx.y * gridDim.x + blockIdx.x;
    } else {
      if (atomicInc(g.done.count, n - 1) != n - 1) return;
      __threadfence();
    }
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(word), "l"(g.done.token) : "memory");
  }
}
__device__ __forceinline__ unsigned long long pass_trace_capacity(const GroupPass& g) {
  return blockIdx.x == 0 && threadIdx.x == 0 ? dev::trace_capacity(pass_state(g)) : 0ull;
}

#ifndef COLL_UNIT_MOVE
// nv vectors of every member from byte src_at of its heap on, reduced in team order, to byte dst_at of the heaps of members
// [d0, d0 + nd).  NS sources (more than `size`: those beyond it are left out), U vectors of each on their way per thread.
template <typename T, int OP, int NS, int U>
__device__ __forceinline__ void pass_vectors(const GroupPass& g, int size, uint64_t src_at, uint64_t dst_at, int d0, int nd, size_t nv) {
  using A = typename coll::Acc<T>::type;
  constexpr int VE = 16 / sizeof(T);
  for (size_t v0 = threadIdx.x; v0 < nv; v0 += (size_t)U * blockDim.x) {
    coll::Vec16<T> in[U][NS];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t v = v0 + (size_t)u * blockDim.x;
      if (v < nv) {
#pragma unroll
        for (int k = 0; k < NS; ++k)
          if (k < size) in[u][k].raw = *reinterpret_cast<const uint4*>(g.base[k] + src_at + v * 16);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t v = v0 + (size_t)u * blockDim.x;
      if (v < nv) {
        A acc[VE];
#pragma unroll
        for (int e = 0; e < VE; ++e) acc[e] = coll::to_acc<T>(in[u][0].e[e]);
#pragma unroll
        for (int k = 1; k < NS; ++k) {
          if (k < size) {
#pragma unroll
            for (int e = 0; e < VE; ++e) acc[e] = coll::apply<A>(OP, acc[e], coll::to_acc<T>(in[u][k].e[e]));
          }
        }
        coll::Vec16<T> out;
#pragma unroll
        for (int e = 0; e < VE; ++e) out.e[e] = coll::from_acc<T>(acc[e]);
        for (int d = d0; d < d0 + nd; ++d) *reinterpret_cast<uint4*>(g.base[d] + dst_at + v * 16) = out.raw;
      }
    }
  }
}
template <typename T, int OP>
__device__ __forceinline__ void pass_reduce_op(const GroupPass& g, uint64_t src_at, uint64_t dst_at, int d0, int nd, size_t n) {
  using A = typename coll::Acc<T>::type;
  constexpr int VE = 16 / sizeof(T);
  const size_t nv = ((src_at | dst_at) & 15) == 0 ? n / VE : 0;
  // sixteen loads on their way per thread, or what the number of members leaves of the next form's; for the types and operators of bulk
  // reductions also without a question per load whether there is such a member (1 % of 32 MiB)
  constexpr bool kHot = (OP == BSHMEM_SUM || OP == BSHMEM_MAX || OP == BSHMEM_MIN) &&
                        (std::is_same<T, float>::value || std::is_same<T, double>::value || std::is_same<T, __half>::value ||
                         std::is_same<T, __nv_bfloat16>::value || std::is_same<T, int32_t>::value || std::is_same<T, long long>::value);
  if (kHot && g.size == 8) pass_vectors<T, OP, 8, 2>(g, 8, src_at, dst_at, d0, nd, nv);
  else if (kHot && g.size == 4) pass_vectors<T, OP, 4, 4>(g, 4, src_at, dst_at, d0, nd, nv);
  else if (kHot && g.size == 2) pass_vectors<T, OP, 2, 8>(g, 2, src_at, dst_at, d0, nd, nv);
  else if (g.size <= 2) pass_vectors<T, OP, 2, 8>(g, g.size, src_at, dst_at, d0, nd, nv);
  else if (g.size <= 4) pass_vectors<T, OP, 4, 4>(g, g.size, src_at, dst_at, d0, nd, nv);
  else if (g.size <= 8 && (kHot || sizeof(T) < 8)) pass_vectors<T, OP, 8, 2>(g, g.size, src_at, dst_at, d0, nd, nv);
  else pass_vectors<T, OP, BSHMEM_MAX_PES, 1>(g, g.size, src_at, dst_at, d0, nd, nv);
  // what is left behind the last whole vector, or all of it where the two sides are not on 16-byte boundaries
  for (size_t i = nv * VE + threadIdx.x; i < n; i += blockDim.x) {
    A acc = coll::to_acc<T>(reinterpret_cast<const T*>(g.base[0] + src_at)[i]);
    for (int k = 1; k < g.size; ++k) acc = coll::apply<A>(OP, acc, coll::to_acc<T>(reinterpret_cast<const T*>(g.base[k] + src_at)[i]));
    for (int d = d0; d < d0 + nd; ++d) reinterpret_cast<T*>(g.base[d] + dst_at)[i] = coll::from_acc<T>(acc);
  }
}

// A block's share: of an allreduce and a rooted reduction a part of the vector, of a reduce-scatter a part of member blockIdx.y's
// block.  An element is read and written by one thread, so the results may take the place of the sources.
template <typename T>
__global__ void __launch_bounds__(kPassThreads) COLL_CAT(k_coll_pass_, COLL_UNIT)(const __grid_constant__ GroupPass g) {
  const CollArgs& a = g.a;
  const unsigned long long cap = pass_trace_capacity(g);
  asm volatile("griddepcontrol.wait;" ::: "memory");         // launched before its predecessor's end
  const int me = blockIdx.y;
  const bool scatter = a.kind == BSHMEM_COLL_REDUCE_SCATTER;
  size_t b, e;
  if (scatter) coll::split_range(a.n, gridDim.x, blockIdx.x, 16 / sizeof(T), &b, &e);
  else coll::split_range(a.n, gridDim.x * gridDim.y, blockIdx.y * gridDim.x + blockIdx.x, 16 / sizeof(T), &b, &e);
  const uint64_t dst_at = a.dst_off + b * sizeof(T), src_at = a.src_off + (b + (scatter ? (size_t)me * a.n : 0)) * sizeof(T);
  const int d0 = a.kind == BSHMEM_COLL_REDUCE ? 0 : scatter ? me : a.root, nd = a.kind == BSHMEM_COLL_REDUCE ? g.size : 1;
  switch (a.op) {
    case BSHMEM_SUM: pass_reduce_op<T, BSHMEM_SUM>(g, src_at, dst_at, d0, nd, e - b); break;
    case BSHMEM_MIN: pass_reduce_op<T, BSHMEM_MIN>(g, src_at, dst_at, d0, nd, e - b); break;
    case BSHMEM_MAX: pass_reduce_op<T, BSHMEM_MAX>(g, src_at, dst_at, d0, nd, e - b); break;
    case BSHMEM_PROD: pass_reduce_op<T, BSHMEM_PROD>(g, src_at, dst_at, d0, nd, e - b); break;
    default:
      if constexpr (!std::is_floating_point<typename coll::Acc<T>::type>::value) {
        if (a.op == BSHMEM_AND) pass_reduce_op<T, BSHMEM_AND>(g, src_at, dst_at, d0, nd, e - b);
        else if (a.op == BSHMEM_OR) pass_reduce_op<T, BSHMEM_OR>(g, src_at, dst_at, d0, nd, e - b);
        else pass_reduce_op<T, BSHMEM_XOR>(g, src_at, dst_at, d0, nd, e - b);
      }
  }
  pass_end(g, cap, a.kind == BSHMEM_COLL_REDUCE_ROOT ? a.n * sizeof(T) : 0);
}
#else
// Member me's part of an alltoall from byte b of its blocks on, nv vectors of each, as one range: eight vectors on their way per thread
// whatever block they belong to.  Block by block, each with an end of its own, 8 PEs: 256 KiB per block 12.3 us in the kernel, 8.2 so;
// 2.8 MB 65.6 and 61.4 (359 MB: 55 at the copy rate); four on their way 71.6, sixteen 67.4.
__device__ __forceinline__ void pass_exchange(const GroupPass& g, int me, size_t b, size_t nv) {
  const CollArgs& a = g.a;
  constexpr int U = 8;
  if (nv == 0) return;
  int k = 0;                                     // the block of the next vector, counted from the own one on
  size_t v = threadIdx.x;
  auto wrap = [&] {
    while (k < g.size && v >= nv) { v -= nv; ++k; }
  };
  wrap();
  while (k < g.size) {
    uint4 x[U];
    uint4* d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      d[u] = nullptr;
      if (k < g.size) {
        const int j = me + k < g.size ? me + k : me + k - g.size;
        x[u] = reinterpret_cast<const uint4*>(g.base[me] + a.src_off + (uint64_t)j * a.n + b)[v];
        d[u] = reinterpret_cast<uint4*>(g.base[j] + a.dst_off + (uint64_t)me * a.n + b) + v;
        v += kPassThreads;
        wrap();
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (d[u]) *d[u] = x[u];
  }
}
// fcollect: member blockIdx.y's block to everybody, read once.  alltoall: member blockIdx.y's blocks to their owners.  broadcast: the
// root's vector to member blockIdx.y, the root's own dest left as it is.
__global__ void __launch_bounds__(kPassThreads) k_coll_pass_move(const __grid_constant__ GroupPass g) {
  const CollArgs& a = g.a;
  const unsigned long long cap = pass_trace_capacity(g);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int me = blockIdx.y;
  size_t b, e;
  coll::split_range(a.n, gridDim.x, blockIdx.x, 16, &b, &e);
  const size_t n = e - b;
  if (a.kind == BSHMEM_COLL_BROADCAST) {
    if (me != a.root) dev::copy_bytes<dev::BLOCK>(g.base[me] + a.dst_off + b, g.base[a.root] + a.src_off + b, n);
  } else if (a.kind == BSHMEM_COLL_ALLTOALL) {
    if (((a.src_off | a.dst_off | a.n) & 15) == 0) {
      pass_exchange(g, me, b, n >> 4);
    } else {
      for (int k = 0; k < g.size; ++k) {
        const int j = (me + k) % g.size;
        dev::copy_bytes<dev::BLOCK>(g.base[j] + a.dst_off + (uint64_t)me * a.n + b, g.base[me] + a.src_off + (uint64_t)j * a.n + b, n);
      }
    }
  } else {
    const uint64_t src_at = a.src_off + b, dst_at = a.dst_off + (uint64_t)me * a.n + b;
    size_t done = 0;
    if (((src_at | dst_at) & 15) == 0) {
      constexpr int U = 8;
      const size_t nv = n >> 4;
      const uint4* src = reinterpret_cast<const uint4*>(g.base[me] + src_at);
      for (size_t v0 = threadIdx.x; v0 < nv; v0 += (size_t)U * blockDim.x) {
        uint4 x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v0 + (size_t)u * blockDim.x < nv) x[u] = src[v0 + (size_t)u * blockDim.x];
        for (int d = 0; d < g.size; ++d) {
          uint4* dst = reinterpret_cast<uint4*>(g.base[d] + dst_at);
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (v0 + (size_t)u * blockDim.x < nv) dst[v0 + (size_t)u * blockDim.x] = x[u];
        }
      }
      done = nv << 4;
    }
    for (int d = 0; d < g.size; ++d) dev::copy_bytes<dev::BLOCK>(g.base[d] + dst_at + done, g.base[me] + src_at + done, n - done);
  }
  pass_end(g, cap, 0);
}
#endif

template <class Kernel>
cudaError_t launch_pass_kernel(Kernel* kernel, const GroupPass& g, int ctas, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas, (unsigned)g.size);
  cfg.blockDim = dim3(kPassThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, g);
}

}  // namespace

cudaError_t COLL_CAT(launch_, COLL_UNIT)(const State& s, const DTeam& t, const CollArgs& a, int ctas, int* status, cudaStream_t stream) {
  COLL_CAT(k_coll_, COLL_UNIT)<<<ctas, kThreads, dyn_smem(a, ctas, ctas), stream>>>(s, t, a, status);
  return cudaGetLastError();
}

cudaError_t COLL_CAT(launch_group_, COLL_UNIT)(const State* states, const DTeam* teams, const CollArgs& a, int ctas, int n,
                                               int* status, cudaStream_t stream, const GroupDone& done) {
  CollArgs args_copy = a;
  GroupDone done_copy = done;
  void* args[] = {&states, &teams, &args_copy, &status, &done_copy};
  return cudaLaunchCooperativeKernel((void*)COLL_CAT(k_coll_group_, COLL_UNIT), dim3(ctas, n), dim3(kThreads), args,
                                     dyn_smem(a, ctas, ctas * n), stream);
}

cudaError_t COLL_CAT(launch_pass_, COLL_UNIT)(const GroupPass& g, int ctas, cudaStream_t stream) {
#ifdef COLL_UNIT_MOVE
  return launch_pass_kernel(k_coll_pass_move, g, ctas, stream);
#else
  switch (g.a.dtype) {
#define COLL_CASE(code, T) case code: return launch_pass_kernel(COLL_CAT(k_coll_pass_, COLL_UNIT)<T>, g, ctas, stream);
    COLL_TYPES(COLL_CASE)
#undef COLL_CASE
  }
  return cudaErrorInvalidValue;
#endif
}

void COLL_CAT(preload_, COLL_UNIT)() {
  cudaFuncAttributes fa;
#ifdef COLL_UNIT_MOVE
  cudaFuncGetAttributes(&fa, k_coll_pass_move);
#else
#define COLL_CASE(code, T) cudaFuncGetAttributes(&fa, COLL_CAT(k_coll_pass_, COLL_UNIT)<T>);
  COLL_TYPES(COLL_CASE)
#undef COLL_CASE
#endif
  cudaFuncGetAttributes(&fa, COLL_CAT(k_coll_, COLL_UNIT));
  cudaFuncGetAttributes(&fa, COLL_CAT(k_coll_group_, COLL_UNIT));
  if (kDynSmem) {      // per device: the caller has made the PE's device current
    cudaFuncSetAttribute(COLL_CAT(k_coll_, COLL_UNIT), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynSmem);
    cudaFuncSetAttribute(COLL_CAT(k_coll_group_, COLL_UNIT), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynSmem);
  }
}

}  // namespace collk
}  // namespace bshmem
