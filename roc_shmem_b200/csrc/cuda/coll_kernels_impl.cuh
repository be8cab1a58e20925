// coll_kernels_impl.cuh — body of one collective-kernel translation unit.  The including .cu defines
//   COLL_UNIT        name of the unit (move, f32, ...)
//   COLL_TYPES(X)    X(dtype code, C type) for every element type the unit reduces (empty for `move`)
// and gets a per-PE kernel, a local-group kernel and their launchers (see coll_kernels.h).
#include <cstring>

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

// All PEs of a local group in ONE cooperative launch: blockIdx.y is the PE.  Used to exercise the multi-PE
// algorithms on a single GPU (kernels that wait on one another must not be separate launches on one device).
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

// The group as one cluster.  Bound by the launch and two round trips to memory: allreduce of 16 KiB of fp32 over 4 PEs, whole call,
// 14.9 us, cooperatively launched with flags in memory 19.5.
struct ClusterGroup {
  State states[kClusterBlocks];
  DTeam teams[kClusterBlocks];
};
__global__ void __launch_bounds__(kThreads) COLL_CAT(k_coll_cluster_, COLL_UNIT)(const __grid_constant__ ClusterGroup g, CollArgs a, int* status,
                                                                                  GroupDone done) {
  __shared__ State s;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(&g.states[blockIdx.y]);
  for (unsigned i = threadIdx.x; i < sizeof(State) / 4; i += kThreads) reinterpret_cast<uint32_t*>(&s)[i] = src[i];
  const DTeam t = g.teams[blockIdx.y];
  __syncthreads();
  if (threadIdx.x == 0) s.one_gpu = BSHMEM_ONE_CLUSTER;
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");         // launched before its predecessor's end
  const int rc = run_coll(s, t, a, blockIdx.x, gridDim.x);
  if (rc != BSHMEM_OK && threadIdx.x == 0) group_failed(status, rc);
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) {
    __threadfence();
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(done.word), "l"(done.token) : "memory");
  }
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

cudaError_t COLL_CAT(launch_cluster_, COLL_UNIT)(const State* states, const DTeam* teams, const CollArgs& a, int ctas, int n, int* status,
                                                 cudaStream_t stream, const GroupDone& done) {
  ClusterGroup g;
  memset(&g, 0, sizeof(g));
  memcpy(g.states, states, sizeof(State) * n);
  memcpy(g.teams, teams, sizeof(DTeam) * n);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas, (unsigned)n);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = dyn_smem(a, ctas, ctas * n);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)ctas; attr[1].val.clusterDim.y = (unsigned)n; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, COLL_CAT(k_coll_cluster_, COLL_UNIT), g, a, status, done);
}

void COLL_CAT(preload_, COLL_UNIT)() {
  cudaFuncAttributes fa;
  cudaFuncGetAttributes(&fa, COLL_CAT(k_coll_cluster_, COLL_UNIT));
  cudaFuncGetAttributes(&fa, COLL_CAT(k_coll_, COLL_UNIT));
  cudaFuncGetAttributes(&fa, COLL_CAT(k_coll_group_, COLL_UNIT));
  if (kDynSmem) {      // per device: the caller has made the PE's device current
    cudaFuncSetAttribute(COLL_CAT(k_coll_, COLL_UNIT), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynSmem);
    cudaFuncSetAttribute(COLL_CAT(k_coll_group_, COLL_UNIT), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynSmem);
    cudaFuncSetAttribute(COLL_CAT(k_coll_cluster_, COLL_UNIT), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynSmem);
  }
}

}  // namespace collk
}  // namespace bshmem
