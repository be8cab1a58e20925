// gpu_backend.cu — the NVLink transport behind the host API, and the kernels the
// host launches on behalf of a PE.
//
// Host-initiated RMA is a copy on the peer mapping; host atomics, waits and
// signals are one-thread kernels using the device API; host collectives launch
// the device collectives striped over several CTAs.  Everything is ordered on one
// CUDA stream per PE (settable, so a PyTorch caller can pass its current stream);
// in blocking mode each call also synchronises the stream and reports device-side
// timeouts, in stream mode calls only enqueue work.
//
// Parity: this replaces the reference's host path over MPI windows
// (library/src/host/host.cpp:160-235, host_templates.hpp) and the GPU-IB backend
// wiring (gpu_ib/backend_ib.cpp:70-111); there is no NIC, so no queue pairs,
// segments or doorbells exist here.
#include <vector>
#include <cuda_runtime.h>

#include <chrono>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <utility>

#include "../host/backend.h"
#include "../host/runtime.h"
#include "../include/bshmem_coll.cuh"
#include "../include/bshmem_gpu.h"
#include "coll_kernels.h"
#include "call_service.h"
#include "gpu_heap.h"
#include "launch_choice.h"
#include "message_ring.h"

using namespace bshmem;
using dev::State;
using DTeam = bshmem::dev::Team;
using collk::CollArgs;

namespace {

// ---------------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------------
template <typename W>
__device__ uint64_t amo_exec(W* p, int dtype, int op, uint64_t value, uint64_t cond) {
  W v = (W)value, c = (W)cond, old = 0;
  switch (op) {
    case BSHMEM_AMO_FETCH_ADD: case BSHMEM_AMO_ADD: case BSHMEM_AMO_FETCH_INC: case BSHMEM_AMO_INC: {
      bool inc = (op == BSHMEM_AMO_FETCH_INC || op == BSHMEM_AMO_INC);
      if (dtype == BSHMEM_FLOAT) {
        float f = inc ? 1.0f : __uint_as_float((unsigned)v);
        old = (W)__float_as_uint(atomicAdd_system(reinterpret_cast<float*>(p), f));
      } else if (dtype == BSHMEM_DOUBLE) {
        double d = inc ? 1.0 : __longlong_as_double((long long)v);
        old = (W)__double_as_longlong(atomicAdd_system(reinterpret_cast<double*>(p), d));
      } else {
        old = atomicAdd_system(p, inc ? (W)1 : v);
      }
      break;
    }
    case BSHMEM_AMO_FETCH: old = atomicOr_system(p, (W)0); break;
    case BSHMEM_AMO_FETCH_CSWAP: case BSHMEM_AMO_CSWAP: old = atomicCAS_system(p, c, v); break;
    case BSHMEM_AMO_SET: case BSHMEM_AMO_SWAP: old = atomicExch_system(p, v); break;
    case BSHMEM_AMO_FETCH_AND: case BSHMEM_AMO_AND: old = atomicAnd_system(p, v); break;
    case BSHMEM_AMO_FETCH_OR: case BSHMEM_AMO_OR: old = atomicOr_system(p, v); break;
    case BSHMEM_AMO_FETCH_XOR: case BSHMEM_AMO_XOR: old = atomicXor_system(p, v); break;
  }
  return (uint64_t)old;
}

// The kernels of messages are launched with programmatic serialization: such a launch costs the host 2.9 us instead of 3.7 (2.4
// on a faster host) and the kernel is on the device when its predecessor in the stream ends, for which it waits here before it touches anything.
__device__ __forceinline__ void after_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
cudaError_t launch_overlapping(void (*kernel)(P...), unsigned grid, unsigned block, unsigned smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}
template <class... P, class... A>
cudaError_t launch_small(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t st, A&&... args) {
  return launch_overlapping(kernel, grid, block, 0, st, std::forward<A>(args)...);
}

// How a one-block kernel tells the host that it is done.  The host polls pinned words instead of synchronising the stream,
// which costs 3.4 us more per call (launch + poll 8.7 us, launch + cudaStreamSynchronize 12.0 us); stream order makes the
// word of a later kernel imply the completion of everything before it.  word == null: nobody waits.
// A result travels in the words themselves, 32 bits of it next to 32 bits of the token in each, so that it needs no fence:
// one of system scope takes 3 to 4 us, as long as the rest of the kernel.
struct Done {
  uint64_t* word;                // two words
  uint64_t token;
};
__device__ __forceinline__ void signal_done(const Done& d) {
  if (d.word) asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(d.word), "l"(d.token) : "memory");
}
__device__ __forceinline__ void signal_result(const Done& d, uint64_t value) {
  if (!d.word) return;
  const uint64_t tag = d.token << 32;
  asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(d.word), "l"(tag | (uint32_t)value) : "memory");
  asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(d.word + 1), "l"(tag | (value >> 32)) : "memory");
}

__global__ void k_amo(State s, int pe, uint64_t off, int dtype, int op, uint64_t value, uint64_t cond, Done done) {
  after_predecessor();
  char* p = s.heap_base[pe] + off;
  uint64_t r = (bshmem_dtype_size(dtype) == 4) ? amo_exec<unsigned int>((unsigned int*)p, dtype, op, value, cond)
                                               : amo_exec<unsigned long long>((unsigned long long*)p, dtype, op, value, cond);
  signal_result(done, r);
}

template <typename T> __device__ T bits_as(uint64_t v) { T t; memcpy(&t, &v, sizeof(T)); return t; }

__device__ int wait_dispatch(const State& s, const char* p, int dtype, int cmp, uint64_t value) {
  switch (dtype) {
    case BSHMEM_INT8: return dev::wait_until<int8_t>(s, (const int8_t*)p, cmp, bits_as<int8_t>(value));
    case BSHMEM_UINT8: return dev::wait_until<uint8_t>(s, (const uint8_t*)p, cmp, bits_as<uint8_t>(value));
    case BSHMEM_INT16: return dev::wait_until<int16_t>(s, (const int16_t*)p, cmp, bits_as<int16_t>(value));
    case BSHMEM_UINT16: return dev::wait_until<uint16_t>(s, (const uint16_t*)p, cmp, bits_as<uint16_t>(value));
    case BSHMEM_INT32: return dev::wait_until<int32_t>(s, (const int32_t*)p, cmp, bits_as<int32_t>(value));
    case BSHMEM_UINT32: return dev::wait_until<uint32_t>(s, (const uint32_t*)p, cmp, bits_as<uint32_t>(value));
    case BSHMEM_INT64: return dev::wait_until<int64_t>(s, (const int64_t*)p, cmp, bits_as<int64_t>(value));
    case BSHMEM_UINT64: return dev::wait_until<uint64_t>(s, (const uint64_t*)p, cmp, value);
    case BSHMEM_FLOAT: return dev::wait_until<float>(s, (const float*)p, cmp, bits_as<float>(value));
    case BSHMEM_DOUBLE: return dev::wait_until<double>(s, (const double*)p, cmp, bits_as<double>(value));
    default: return BSHMEM_ERR_UNSUPPORTED;
  }
}

// What a wait would see at its first look.
__device__ int test_dispatch(const State& s, const char* p, int dtype, int cmp, uint64_t value) {
  int h = 0;
  switch (dtype) {
    case BSHMEM_INT8: h = dev::test<int8_t>(s, (const int8_t*)p, cmp, bits_as<int8_t>(value)); break;
    case BSHMEM_UINT8: h = dev::test<uint8_t>(s, (const uint8_t*)p, cmp, bits_as<uint8_t>(value)); break;
    case BSHMEM_INT16: h = dev::test<int16_t>(s, (const int16_t*)p, cmp, bits_as<int16_t>(value)); break;
    case BSHMEM_UINT16: h = dev::test<uint16_t>(s, (const uint16_t*)p, cmp, bits_as<uint16_t>(value)); break;
    case BSHMEM_INT32: h = dev::test<int32_t>(s, (const int32_t*)p, cmp, bits_as<int32_t>(value)); break;
    case BSHMEM_UINT32: h = dev::test<uint32_t>(s, (const uint32_t*)p, cmp, bits_as<uint32_t>(value)); break;
    case BSHMEM_INT64: h = dev::test<int64_t>(s, (const int64_t*)p, cmp, bits_as<int64_t>(value)); break;
    case BSHMEM_UINT64: h = dev::test<uint64_t>(s, (const uint64_t*)p, cmp, bits_as<uint64_t>(value)); break;
    case BSHMEM_FLOAT: h = dev::test<float>(s, (const float*)p, cmp, bits_as<float>(value)); break;
    case BSHMEM_DOUBLE: h = dev::test<double>(s, (const double*)p, cmp, bits_as<double>(value)); break;
  }
  return h ? BSHMEM_OK : BSHMEM_ERR_TIMEOUT;
}

__global__ void k_wait_until(State s, uint64_t off, int dtype, int cmp, uint64_t value, Done done) {
  after_predecessor();
  signal_result(done, (uint32_t)wait_dispatch(s, s.heap_base[s.my_pe] + off, dtype, cmp, value));
}

// One element of `size` bytes (any alignment) between a heap and a word.
__device__ uint64_t read_bits(const char* src, int size) {
  uint64_t v = 0;
  if ((reinterpret_cast<uintptr_t>(src) & (size - 1)) == 0) {
    switch (size) {
      case 8: v = *reinterpret_cast<const volatile uint64_t*>(src); break;
      case 4: v = *reinterpret_cast<const volatile uint32_t*>(src); break;
      case 2: v = *reinterpret_cast<const volatile uint16_t*>(src); break;
      default: v = *reinterpret_cast<const volatile uint8_t*>(src);
    }
  } else {
    for (int i = 0; i < size; ++i) v |= (uint64_t)(*reinterpret_cast<const volatile uint8_t*>(src + i)) << (8 * i);
  }
  return v;
}
__global__ void k_read_word(const char* src, int size, Done done) {
  after_predecessor();
  signal_result(done, read_bits(src, size));
}
__global__ void k_write_word(char* dst, uint64_t v, int size) {
  after_predecessor();
  if ((reinterpret_cast<uintptr_t>(dst) & (size - 1)) == 0) {
    switch (size) {
      case 8: *reinterpret_cast<uint64_t*>(dst) = v; return;
      case 4: *reinterpret_cast<uint32_t*>(dst) = (uint32_t)v; return;
      case 2: *reinterpret_cast<uint16_t*>(dst) = (uint16_t)v; return;
      default: *reinterpret_cast<uint8_t*>(dst) = (uint8_t)v; return;
    }
  }
  for (int i = 0; i < size; ++i) reinterpret_cast<uint8_t*>(dst)[i] = (uint8_t)(v >> (8 * i));
}

// Small device-to-device messages.  A copy-engine request costs the host 3.4 us, a kernel launch 2.4 us (measured
// back to back on one host), and that is the message rate; the copy itself is shorter than either.  A block moves kSmallPiece
// bytes: one 16-byte access per thread, so a message of up to kSmallCopyMax takes one round trip to memory.
// The line: 64 puts of 256 KiB to 1 MiB take 157 to 162 us through the kernel and 245 to 259 us through the copy engine.
// At 2 MiB (230 and 262 us) the kernel's own time shows, and that size stays with the copy engine, which takes no SM.
// Where the two sides are misaligned against each other the kernel moves words or bytes and falls behind beyond 128 KiB
// (64 puts of 256 KiB - 1, one byte apart: 248 us against 227; of 1 MiB - 1: 656 against 400).
constexpr uint64_t kSmallPiece = 4096, kSmallCopyMax = 1u << 20, kSmallCopyMaxSkewed = 128u << 10;
__global__ void __launch_bounds__(256) k_copy_small(char* dst, const char* src, uint64_t n) {
  after_predecessor();
  const uint64_t b = blockIdx.x * kSmallPiece, e = b + kSmallPiece < n ? b + kSmallPiece : n;
  dev::copy_bytes<dev::BLOCK>(dst + b, src + b, e - b);
}
// Non-blocking messages of a context between device buffers need no launch each: the host writes them into a ring in pinned memory
// and one block on the context's stream takes them from there (16 KiB and less; longer ones: k_ring_wide).  The block is launched by the
// first message, stays while messages follow one another closely (kRingIdleNs) and at most kRingLifeNs.  While it stays it has
// its multiprocessor's place, beside kernels that take a whole one per block too: 8192 x 8192 x 3584 products with 64 messages
// before each take 358 to 360 us (356 to 361 with one launch per message); 1024 rows 50 (173 to 181), with four messages 49
// (43).  Ending after 2 us without a message instead of 5 gains nothing there and costs a window 8 of 48 us.  The host path
// bounds a window of messages: 64 puts of 64 bytes and a quiet took 177 us by one launch each (2.4 us apart and more), 25 so.  A
// block with sixteen warps moves a message per warp, 16 KiB in four round trips to memory.
// message_ring.h has the protocol.
constexpr unsigned kRingThreads = 512, kRingBatch = kRingThreads / 32;
constexpr unsigned long long kRingIdleNs = 5000, kRingLifeNs = 100000;
__device__ __forceinline__ void st_host(uint64_t* p, uint64_t v) { asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory"); }

struct RingMessages {
  struct { char* dst; const char* src; uint32_t n; } msg[kRingBatch];
  int found, over;                     // messages of the batch; whether the block is to end (1) or has nothing left (2)
};
// One look at the ring, by one warp.  The last load acquires: what the host had seen done before it wrote a message is behind it (a
// window of 64 puts of 64 bytes takes 25 us so, 29 with relaxed loads and a fence of system scope, 59 if all three acquire).
__device__ __forceinline__ void ring_look(Ring* ring, uint32_t next, uint32_t generation, int lane, bool closing, unsigned long long begun,
                                          unsigned long long& last, RingMessages& b) {
  const uint32_t index = next + lane;
  const uint64_t* w = ring->slot[index % kRingSlots].w;
  uint64_t v0 = 0, v1 = 0, v2 = 0, stop = 0;
  if (lane == 31) asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(stop) : "l"(&ring->stop) : "memory");
  if (lane < kRingBatch) {
    asm volatile("ld.relaxed.sys.global.v2.u64 {%0, %1}, [%2];" : "=l"(v0), "=l"(v1) : "l"(w) : "memory");
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v2) : "l"(w + 2) : "memory");       // last: what follows it waits for it
  }
  stop = __shfl_sync(0xffffffffu, stop, 31);
  const uint64_t low48 = (1ull << 48) - 1;
  const bool here = lane < kRingBatch && ring_arrived(v0, v1, v2, index, generation);
  const uint32_t size = (uint32_t)v2;
  const unsigned got = __ballot_sync(0xffffffffu, here), starts = __ballot_sync(0xffffffffu, here && (size & kRingOrdered)) & ~1u;
  int count = __ffs(~got) - 1;
  if (starts && __ffs(starts) - 1 < count) count = __ffs(starts) - 1;      // an ordered message begins a batch
  if (lane < count) {
    b.msg[lane].dst = reinterpret_cast<char*>(v0 & low48);
    b.msg[lane].src = reinterpret_cast<const char*>(v1 & low48);
    b.msg[lane].n = size & kRingSizeMask;
  }
  if (lane == 0) {
    const unsigned long long now = dev::timer();
    if (count) last = now;
    b.found = count;
    b.over = closing ? (count ? 0 : 2) : ring_stopped(stop, generation) || now - begun > kRingLifeNs || now - last > kRingIdleNs ? 1 : 0;
  }
  __syncwarp();
}

// The last warp says how far the messages are done, while the first one looks for more.  System scope, also on one GPU: a quiet that
// sees the count ends like a stream synchronisation, for readers on the host too.
constexpr unsigned kRingPublisher = kRingThreads - 32;
__device__ __forceinline__ void ring_publish(Ring* ring, uint32_t next) {
  if (threadIdx.x == kRingPublisher) {
    asm volatile("fence.acq_rel.sys;" ::: "memory");
    st_host(&ring->consumed, next);
  }
}

__global__ void __launch_bounds__(kRingThreads) k_ring(Ring* ring, uint32_t next, uint32_t generation) {
  after_predecessor();
  __shared__ RingMessages b;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned long long begun = dev::timer();
  unsigned long long last = begun;
  bool closing = false;
  while (true) {
    if (warp == 0) ring_look(ring, next, generation, lane, closing, begun, last, b);
    __syncthreads();
    const int count = b.found, end = b.over;
    if (count) {
      if (warp < count) dev::copy_bytes<dev::WARP>(b.msg[warp].dst, b.msg[warp].src, b.msg[warp].n);
      __syncthreads();
      next += count;
      ring_publish(ring, next);
    }
    if (end == 2) break;
    if (end == 1) {
      closing = true;
      if (threadIdx.x == 0) {
        st_host(&ring->closed, generation);
        asm volatile("fence.sc.sys;" ::: "memory");            // ... before the last look
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == kRingPublisher) asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(&ring->final), "l"((uint64_t)generation << 32 | next) : "memory");
}

// The same by several blocks, for messages that one block is too slow for.  The first block to run looks at the ring; those that have
// come by the time it finds messages take their part of them, pieces of 4 KiB, one round trip to memory of a warp, in turn.  None of them is
// needed: beside a kernel that leaves a single place, of what a launch per message took, the first block does all, and the rest pass
// through behind it.  (As a cluster of eight blocks of 512 threads, all of which had to find their places at once, this had no progress there.)
// us by a launch each (2.3 to 2.7 apart, the host's) / as a cluster / so.  Windows of 64 puts of 17 KB 175 / 56 / 35, 64 KiB 175 / 69 / 38, 256 KiB
// 175 / 95 / 63, 512 KiB 175 / 140 / 93; eight puts of 64 KiB and a quiet 26 / 20 / 15, two 13 / 22 / 12.  A product of 1024 rows behind one message of
// 64 KiB 42.7 / 46.3 / 42.6, behind four 49 / 52 / 49, behind 64 160 / 70 / 56 (41.5 without any).  Up to 16 KiB one block is as fast and holds
// one multiprocessor.  All of it in this GPU's own memory; a peer's is behind a link, where a block moves less.
// A batch of up to four rounds of the first block's warps is not handed out: that takes 2 us.
constexpr unsigned kWideThreads = 256, kWideBlocks = 16, kWideWarps = kWideThreads / 32, kWidePublisher = kWideThreads - 32, kRingPiece = 4096;
constexpr unsigned long long kWideComeNs = 3000;               // from the first block's begin on
constexpr unsigned long long kWideLimitNs = 2000000000;        // of the waits for one another, each of which ends by itself
struct RingShare {                     // device memory, zero between launches
  unsigned long long batch;            // by the first block: the batch's number | how many blocks it is for; number ~0: no more
  unsigned int came, done, left;       // blocks: begun, finished with their parts (of all batches), ended
  RingMessages b;
};
__device__ __forceinline__ void copy_pieces(const RingMessages& b, int count, unsigned piece, unsigned step) {
  unsigned first = 0;
  for (int m = 0; m < count; ++m) {
    const uint32_t n = b.msg[m].n, pieces = (n + kRingPiece - 1) / kRingPiece;
    for (; piece - first < pieces; piece += step) {
      const uint32_t at = (piece - first) * kRingPiece;
      dev::copy_bytes<dev::WARP>(b.msg[m].dst + at, b.msg[m].src + at, min(kRingPiece, n - at));
    }
    first += pieces;
  }
}
__device__ __forceinline__ void ring_share_out(Ring* ring, RingShare* share, RingMessages& b, uint32_t next, uint32_t generation) {
  __shared__ unsigned blocks;          // that the batch is for
  __shared__ int failed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned long long begun = dev::timer();
  unsigned long long last = begun;
  unsigned batch = 0, parts = 0;       // of the publisher: the others' parts handed out so far
  bool closing = false;
  if (threadIdx.x == 0) failed = 0;
  while (true) {
    if (warp == 0) {
      do ring_look(ring, next, generation, lane, closing, begun, last, b);
      while (b.found == 0 && b.over == 0);
    }
    __syncthreads();                   // the others' parts of the last batch are done, too
    const int count = b.found, end = b.over;
    if (failed) break;
    if (count) {
      if (warp == 0) {
        unsigned pieces = lane < count ? (b.msg[lane].n + kRingPiece - 1) / kRingPiece : 0;
        pieces = __reduce_add_sync(0xffffffffu, pieces);
        unsigned here = 1;
        if (pieces > 4 * kWideWarps) {
          for (unsigned i = lane; i < sizeof(RingMessages) / 4; i += 32) reinterpret_cast<uint32_t*>(&share->b)[i] = reinterpret_cast<const uint32_t*>(&b)[i];
          // launched together, they come together; a moment for those that are behind, once
          if (lane == 0)
            do asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(here) : "l"(&share->came) : "memory");
            while (here != gridDim.x && dev::timer() - begun < kWideComeNs);
          here = __shfl_sync(0xffffffffu, here, 0);
          __syncwarp();
        }
        if (lane == 0) {
          blocks = here;
          if (here > 1) asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(&share->batch), "l"((unsigned long long)(batch + 1) << 32 | here) : "memory");
        }
      }
      __syncthreads();
      const unsigned here = blocks;
      batch += here > 1;
      copy_pieces(b, count, warp, here * kWideWarps);
      last = dev::timer();             // idle from here on
      __syncthreads();
      next += count;
      // one thread waits for the others' parts and says how far the messages are done, while the first warp looks for more
      if (threadIdx.x == kWidePublisher) {
        parts += here - 1;
        bool ok = here == 1;
        for (const unsigned long long t0 = dev::timer(); !ok && dev::timer() - t0 < kWideLimitNs;) {
          unsigned done;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(done) : "l"(&share->done) : "memory");
          ok = done == parts;
        }
        if (ok) {
          asm volatile("fence.acq_rel.sys;" ::: "memory");
          st_host(&ring->consumed, next);
        } else {
          failed = 1;
          st_host(&ring->failed, generation);
        }
      }
    }
    if (end == 2) break;
    if (end == 1) {
      if (threadIdx.x == 0) {
        st_host(&ring->closed, generation);
        asm volatile("fence.sc.sys;" ::: "memory");
      }
      closing = true;
    }
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(&share->batch), "l"(~0ull) : "memory");
  if (threadIdx.x == kWidePublisher) asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(&ring->final), "l"((uint64_t)generation << 32 | next) : "memory");
}
__device__ __forceinline__ void ring_take_part(RingShare* share, RingMessages& b, unsigned me) {
  __shared__ unsigned blocks;          // that the batch is for; 0: no more
  unsigned seen = 0;                   // thread 0's
  while (true) {
    if (threadIdx.x == 0) {
      unsigned long long v = 0;
      const unsigned long long t0 = dev::timer();
      do {
        if (dev::timer() - t0 > 2 * kWideLimitNs) v = ~0ull;   // beyond what the first block lives and waits
        else asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&share->batch) : "memory");
        if (v != ~0ull && me >= (unsigned)v) seen = (unsigned)(v >> 32);    // not for this block
      } while ((unsigned)(v >> 32) == seen);
      seen = (unsigned)(v >> 32);
      blocks = v == ~0ull ? 0 : (unsigned)v;
    }
    __syncthreads();
    const unsigned here = blocks;
    if (!here) return;
    for (unsigned i = threadIdx.x; i < sizeof(RingMessages) / 4; i += kWideThreads)
      reinterpret_cast<uint32_t*>(&b)[i] = __ldcg(reinterpret_cast<const uint32_t*>(&share->b) + i);
    __syncthreads();
    copy_pieces(b, b.found, me * kWideWarps + (threadIdx.x >> 5), here * kWideWarps);
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&share->done) : "memory");
  }
}
__global__ void __launch_bounds__(kWideThreads) k_ring_wide(Ring* ring, RingShare* share, uint32_t next, uint32_t generation) {
  after_predecessor();
  __shared__ RingMessages b;
  __shared__ unsigned order;
  static_assert(sizeof(RingMessages) % 4 == 0, "passed on in words");
  if (threadIdx.x == 0) order = atomicAdd(&share->came, 1u);
  __syncthreads();
  if (order == 0) ring_share_out(ring, share, b, next, generation);
  else ring_take_part(share, b, order);
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&share->left, 1u) == gridDim.x - 1) {      // nobody looks at it any more
    share->batch = 0;
    share->came = share->done = share->left = 0;
  }
}

// Payload and signal of a small message in one block: the block barrier orders every thread's stores before the
// release of the signal word.  Up to kSmallSignalMax bytes one block (8 KiB per round) is done before a second launch
// would have reached the device.
constexpr uint64_t kSmallSignalMax = 32u << 10;
__global__ void __launch_bounds__(512) k_put_signal(State s, char* dst, const char* src, uint64_t n, uint64_t* sig, uint64_t value, int sig_op, Done done) {
  after_predecessor();
  if (n) dev::copy_bytes<dev::BLOCK>(dst, src, n);
  __syncthreads();
  if (threadIdx.x == 0) {
    dev::fence_peers(s);
    dev::signal_update(sig, value, sig_op);
    signal_done(done);
  }
}

// Blocking calls of the default context that follow one another closely need no launch each.  While one block on a stream of the
// runtime's own looks at a slot in pinned memory, a call is a store by the host, the operation, and the answer in the call's own words:
// 2.3 us where a launch and its answer take 6.6.  The calls belong behind what the caller's stream holds, so the host asks first
// whether that stream is idle (1.4 us); if it is not, the call is a launch in that stream as ever.  Of a blocking stream that is not asked:
// its launches wait for the legacy default stream, and its answer leaves out what is there; the legacy stream's own counts all that
// its launches wait for.  No order is lost the other way: a
// call has been answered before the caller enqueues anything else.  A block that has waited kCallIdleNs for a request, or lived for kCallLifeNs,
// ends: until then a device-wide synchronisation waits for it, and a kernel that wants every multiprocessor for one of them (with 5 us the gaps of
// a loop of calls end it).  So blocks are launched, in the shadow of a call's own launch, where the program has had a use for them
// (CallSeries), and asked when they say that they are there.  us, by launches / so: fetch-add, put with signal of 4 KiB, wait and read, over and
// over 33.9 / 25.5; with a device-wide synchronisation behind each of these passes 40.0 / 40.7 (45.3 while every series had its block); a
// kernel, then a call 13.9 / 14.0 (14.5 while every series asked); a kernel, then two 21.8 / 22.1 (23.0); single passes the same.  The
// look at the slot is an acquire, so that the block sees what kernels wrote before the host asked.  The block's stream is ordered against the
// caller's by answers alone, so an answer comes when what the call did has been done at its place: an atomic's carries what was there, and a
// fence stands between a signal and its answer.  call_service.h has the protocol.
constexpr unsigned kCallThreads = 512;
constexpr unsigned long long kCallIdleNs = 8000, kCallLifeNs = 500000;
// Puts with signal: what the block copies as fast as two launches begin.  The four calls above with 32 / 64 / 128 / 256 / 400 / 512 KiB by launches
// 33.9 / 34.4 / 34.4 / 34.4 / 34.3 / 34.6 us, so 25.8 / 26.2 / 26.9 / 30.0 / 33.0 / 40.0.  (Off each other's alignment kSmallSignalMax.)
// All of it in this GPU's own memory: over a link one block moves some 50 GB/s.
constexpr uint64_t kServedSignalMax = 256u << 10;
__global__ void __launch_bounds__(kCallThreads) k_calls(State s, CallSlot* slot, uint32_t seq, uint32_t generation) {
  __shared__ uint32_t req[kCallWords];
  __shared__ int over;
  if (threadIdx.x == 0) st_host(&slot->begun, generation);
  const int lane = threadIdx.x & 31;
  const unsigned long long begun = dev::timer();
  while (true) {
    if (threadIdx.x < 32) {
      const unsigned long long since = dev::timer();
      while (true) {
        uint64_t v = 0;
        if (lane < (int)kCallWords) asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(&slot->w[lane]) : "memory");
        const unsigned long long now = dev::timer();
        const bool end = __shfl_sync(0xffffffffu, (int)(now - since > kCallIdleNs || now - begun > kCallLifeNs), 0);
        if (end || __all_sync(0xffffffffu, lane >= (int)kCallWords || (uint32_t)(v >> 32) == seq)) {
          if (lane < (int)kCallWords) req[lane] = (uint32_t)v;
          if (lane == 0) over = end;
          break;
        }
      }
    }
    __syncthreads();
    if (over) break;
    auto pair = [&](CallWord at) { return (uint64_t)req[at + 1] << 32 | req[at]; };
    const uint32_t head = req[CALL_HEAD];
    const int dtype = head >> 8 & 0xFF, op = head >> 16 & 0xFF, size = head >> 24;
    char* addr = reinterpret_cast<char*>(pair(CALL_ADDR));
    const uint64_t value = pair(CALL_VALUE), other = pair(CALL_OTHER);
    const Done done{reinterpret_cast<uint64_t*>(pair(CALL_DONE)), pair(CALL_TOKEN)};
    switch (head & 0xFF) {
      case CALL_AMO:
        if (threadIdx.x == 0)
          signal_result(done, size == 4 ? amo_exec<unsigned int>((unsigned int*)addr, dtype, op, value, other)
                                        : amo_exec<unsigned long long>((unsigned long long*)addr, dtype, op, value, other));
        break;
      case CALL_READ:
        if (threadIdx.x == 0) signal_result(done, read_bits(addr, size));
        break;
      case CALL_TEST:
        if (threadIdx.x == 0) signal_result(done, (uint32_t)test_dispatch(s, addr, dtype, op, value));
        break;
      case CALL_PUT_SIGNAL:
        if (req[CALL_BYTES]) dev::copy_bytes<dev::BLOCK>(addr, reinterpret_cast<const char*>(other), req[CALL_BYTES]);
        __syncthreads();
        if (threadIdx.x == 0) {
          dev::fence_peers(s);
          dev::signal_update(reinterpret_cast<uint64_t*>(pair(CALL_SIG)), value, op);
          dev::fence_peers(s);         // no stream orders what follows the answer behind the signal
          signal_done(done);
        }
        break;
    }
    __syncthreads();
    ++seq;
  }
  if (threadIdx.x == 0) asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(&slot->final), "l"((uint64_t)generation << 32 | (seq - 1)) : "memory");
}

// Runs after the payload copy on the same stream: publish, then update the signal word.
__global__ void k_signal(State s, int pe, uint64_t sig_off, uint64_t value, int sig_op, Done done) {
  after_predecessor();
  uint64_t* sig = reinterpret_cast<uint64_t*>(s.heap_base[pe] + sig_off);
  dev::fence_peers(s);
  dev::signal_update(sig, value, sig_op);
  signal_done(done);
}

// Large messages: each CTA moves its share with bulk async copies through a shared-memory ring (no payload in
// registers; see dev::bulk_copy_block).  `src` / `dst` are already translated to the peer mapping.  Bound by the launch up to
// some 8 MiB and by HBM beyond it: launched behind their predecessor's end, these kernels and k_rma took 4.1 us per
// message of 64 KiB to 1 MiB and 33.9 us per 96 MB; overlapping its launch they take 2.5 and 31.7 us.
constexpr int kBulkStages = 4, kBulkChunk = 32768;
__global__ void __launch_bounds__(128) k_rma_bulk(State s, char* dst, const char* src, uint64_t n, int* status) {
  after_predecessor();
  extern __shared__ __align__(128) char bulk_smem[];
  __shared__ __align__(8) uint64_t bars[kBulkStages];
  uint64_t per = ((n + gridDim.x - 1) / gridDim.x + 127) & ~127ull;
  uint64_t b = per * blockIdx.x, e = b + per < n ? b + per : n;
  if (b >= n) return;
  int rc = dev::bulk_copy_block<kBulkStages, kBulkChunk>(s, dst + b, src + b, e - b, bulk_smem, bars);
  if (rc != BSHMEM_OK && threadIdx.x == 0) atomicCAS(status, 0, rc);
}

// Device-initiated put / get of a large message striped over the grid.  The grid walks the message in 256 KiB pieces,
// piece i to CTA i mod grid: at any time the CTAs touch one window of grid x 256 KiB instead of one 2 MiB page each,
// which matters once the message is much larger than what the address-translation caches cover (132 CTAs on
// 256 MiB lost 8 % with one contiguous share per CTA).
constexpr uint64_t kRmaPiece = 256u << 10;
__global__ void __launch_bounds__(512) k_rma(State s, int pe, uint64_t sym_off, char* local, uint64_t n, int is_put, int scope) {
  after_predecessor();
  char* sym = s.heap_base[s.my_pe] + sym_off;
  // a message of up to grid x 256 KiB is still split evenly: every CTA gets one contiguous share
  uint64_t piece = ((n + gridDim.x - 1) / gridDim.x + 15) & ~15ull;
  if (piece > kRmaPiece) piece = kRmaPiece;
  for (uint64_t b = (uint64_t)blockIdx.x * piece; b < n; b += (uint64_t)gridDim.x * piece) {
    const uint64_t e = b + piece < n ? b + piece : n;
    if (scope == dev::BLOCK) {
      if (is_put) dev::putmem_nbi<dev::BLOCK>(s, sym + b, local + b, e - b, pe);
      else dev::getmem<dev::BLOCK>(s, local + b, sym + b, e - b, pe);
    } else if (scope == dev::WARP) {
      // each warp takes a contiguous share of the piece
      int nw = blockDim.x >> 5, w = threadIdx.x >> 5;
      uint64_t wper = (((e - b) + nw - 1) / nw + 15) & ~15ull;
      uint64_t wb = b + wper * w, we = wb + wper < e ? wb + wper : e;
      if (wb < e) {
        if (is_put) dev::putmem_nbi<dev::WARP>(s, sym + wb, local + wb, we - wb, pe);
        else dev::getmem<dev::WARP>(s, local + wb, sym + wb, we - wb, pe);
      }
    } else {
      int nt = blockDim.x, t = threadIdx.x;
      uint64_t tper = (((e - b) + nt - 1) / nt + 15) & ~15ull;
      uint64_t tb = b + tper * t, te = tb + tper < e ? tb + tper : e;
      if (tb < e) {
        if (is_put) dev::putmem_nbi<dev::THREAD>(s, sym + tb, local + tb, te - tb, pe);
        else dev::getmem<dev::THREAD>(s, local + tb, sym + tb, te - tb, pe);
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// Backend
// ---------------------------------------------------------------------------------
#define RT_TRY(call) do { cudaError_t _e = (call); if (_e != cudaSuccess) return cuda_fail(#call, _e); } while (0)

constexpr int kResultSlots = 64;
struct Pinned {
  bshmem_error_record_t err;       // lane 0's copy is the device-visible error record of the PE
  int status[kResultSlots];
  uint64_t done[kResultSlots][2];  // completion tokens and results (see Done)
  CallSlot calls;                  // lane 0's
  uint64_t pass[collk::kPassWords];    // lane 0's: a group's pass of a few blocks, one word per block
};

// What a host context owns on this backend: its ordering domain (a stream) and the pinned words its blocking calls
// read results from.  Lane 0 is the default context; its stream is the settable PE stream.
struct Lane {
  cudaStream_t stream = nullptr;
  Pinned* pinned = nullptr;
  int* dstatus = nullptr;          // device status word of collectives launched on this lane
  std::atomic<unsigned> next{0};
  std::atomic<bool> taken[kResultSlots] = {};      // slots whose call still waits for its answer
  bool open = false;
  RingWriter ring;                                 // of a context other than the default one, whose stream the caller owns (see k_ring)
  RingShare* share = nullptr;                      // of the ring's blocks
};

// A waiting call's own result slot of its lane, from before the launch until the answer has been read: threads that share the
// lane do not meet on one, however many calls the others make meanwhile.  A call that nobody waits for has none (its kernel
// signals nothing, also when it is replayed from a graph later on).
class Ticket {
 public:
  explicit Ticket(Lane* lane) : lane_(lane) {
    if (!lane) return;
    for (;; std::this_thread::yield()) {             // beyond kResultSlots waiting calls: until one of them has returned
      const unsigned k = lane->next.fetch_add(1, std::memory_order_relaxed);
      slot = k % kResultSlots;
      if (lane->taken[slot].exchange(true, std::memory_order_acquire)) continue;
      done = {lane->pinned->done[slot], (uint64_t)k + 1};
      return;
    }
  }
  ~Ticket() { if (lane_) lane_->taken[slot].store(false, std::memory_order_release); }
  Ticket(const Ticket&) = delete;
  Ticket& operator=(const Ticket&) = delete;
  unsigned slot = 0;
  Done done{};

 private:
  Lane* lane_;
};

// Selection of the calling thread (see Backend::ctx_select) and an optional binding of the thread to one lane for
// everything it issues, collectives included (the reverse-offload service thread runs on a lane of its own).
thread_local int tl_selected_ctx = 0;
thread_local const void* tl_bound_backend = nullptr;
thread_local int tl_bound_ctx = -1;
thread_local bool tl_local_is_device = false;   // the caller vouches that the local buffer is memory of this PE's GPU
thread_local std::string tl_err;

// While it exists, the calling thread may synchronise streams that are not captured although another one is.
class RelaxedCapture {
 public:
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  RelaxedCapture(const RelaxedCapture&) = delete;
  RelaxedCapture& operator=(const RelaxedCapture&) = delete;

 private:
  cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

class GpuBackend final : public Backend {
 public:
  GpuBackend(gpu::Heap* heap, bool own_heap) : heap_(heap), own_heap_(own_heap) {}

  int setup(const bshmem_config_t& cfg, int coll_ctas) {
    RT_TRY(cudaSetDevice(heap_->device));
    RT_TRY(cudaStreamCreateWithFlags(&own_stream_, cudaStreamNonBlocking));
    stream_ = own_stream_;
    RT_TRY(cudaHostAlloc(&pinned_, sizeof(Pinned), cudaHostAllocMapped));
    memset(pinned_, 0, sizeof(Pinned));
    lanes_[0].pinned = pinned_;
    calls_.slot = &pinned_->calls;
    RT_TRY(cudaStreamCreateWithFlags(&calls_stream_, cudaStreamNonBlocking));
    lanes_[0].open = true;
    // counters followed by the (initially disabled) event ring
    RT_TRY(cudaMalloc(&dstats_, sizeof(unsigned long long) * (BSHMEM_DSTAT_COUNT + BSHMEM_TRACE_WORDS)));
    RT_TRY(cudaMemset(dstats_, 0, sizeof(unsigned long long) * (BSHMEM_DSTAT_COUNT + BSHMEM_TRACE_WORDS)));
    RT_TRY(cudaMalloc(&dstatus_, sizeof(int)));
    RT_TRY(cudaMemset(dstatus_, 0, sizeof(int)));
    lanes_[0].dstatus = dstatus_;
    memset(&state_, 0, sizeof(state_));
    state_.my_pe = heap_->my_pe;
    state_.n_pes = heap_->n_pes;
    state_.heap_bytes = heap_->heap_bytes;
    for (int p = 0; p < heap_->n_pes; ++p) state_.heap_base[p] = heap_->base[p];
    state_.mc_base = heap_->mc_base;
    state_.err = &pinned_->err;
    state_.timeout_ns = cfg.timeout_us * 1000ull;
    state_.stats = cfg.profile ? dstats_ : nullptr;
    state_.debug = cfg.debug;
    state_.one_gpu = heap_->n_pes == 1 || heap_->mode == gpu::HEAP_LOCAL_GROUP ? 1 : 0;
    coll_ctas_ = coll_ctas < 1 ? 1 : (coll_ctas > BSHMEM_MAX_COLL_CTAS ? BSHMEM_MAX_COLL_CTAS : coll_ctas);
    int sms = 0;
    RT_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, heap_->device));
    if (coll_ctas_ > sms) coll_ctas_ = sms;
    sms_ = sms;
    return BSHMEM_OK;
  }

  ~GpuBackend() override {
    cudaSetDevice(heap_->device);
    cudaDeviceSynchronize();
    for (int i = 1; i < BSHMEM_MAX_CTXS; ++i) ctx_close(i);
    if (own_stream_) cudaStreamDestroy(own_stream_);
    if (calls_stream_) cudaStreamDestroy(calls_stream_);
    if (group_dev_) cudaFree(group_dev_);
    if (dstats_) cudaFree(dstats_);
    if (dstatus_) cudaFree(dstatus_);
    if (pinned_) cudaFreeHost(pinned_);
    if (own_heap_) gpu::heap_destroy(heap_);
  }

  const char* name() const override { return "nvlink"; }
  int my_pe() const override { return heap_->my_pe; }
  int n_pes() const override { return heap_->n_pes; }
  uint64_t heap_bytes() const override { return heap_->heap_bytes; }
  uint64_t reserved_bytes() const override { return BSHMEM_INTERNAL_BYTES; }
  char* local_base() const override { return heap_->base[heap_->my_pe]; }
  char* peer_base(int pe) const override { return heap_->mapped[pe] ? heap_->base[pe] : nullptr; }
  bool host_dereferenceable() const override { return false; }
  void set_timeout_us(uint64_t t) override { state_.timeout_ns = t * 1000ull; }
  std::string last_error() const override { return tl_err; }

  // ---- host contexts -----------------------------------------------------------------
  int ctx_open(int idx, long) override {
    if (idx <= 0 || idx >= BSHMEM_MAX_CTXS) return BSHMEM_ERR_INVALID;
    Lane& L = lanes_[idx];
    if (L.open) return BSHMEM_OK;
    RT_TRY(cudaSetDevice(heap_->device));
    RT_TRY(cudaStreamCreateWithFlags(&L.stream, cudaStreamNonBlocking));
    RT_TRY(cudaHostAlloc(&L.pinned, sizeof(Pinned), cudaHostAllocMapped));
    memset(L.pinned, 0, sizeof(Pinned));
    RT_TRY(cudaMalloc(&L.dstatus, sizeof(int)));
    RT_TRY(cudaMemsetAsync(L.dstatus, 0, sizeof(int), L.stream));       // where they are used: that stream does not wait for the default one
    Ring* ring = nullptr;
    RT_TRY(cudaHostAlloc(&ring, sizeof(Ring), cudaHostAllocMapped));
    memset(ring, 0, sizeof(Ring));
    RT_TRY(cudaMalloc(&L.share, sizeof(RingShare)));
    RT_TRY(cudaMemsetAsync(L.share, 0, sizeof(RingShare), L.stream));
    L.ring.open(ring);
    L.open = true;
    return BSHMEM_OK;
  }
  void ctx_close(int idx) override {
    if (idx <= 0 || idx >= BSHMEM_MAX_CTXS || !lanes_[idx].open) return;
    Lane& L = lanes_[idx];
    L.open = false;
    enter(L);
    if (L.stream) { cudaStreamSynchronize(L.stream); cudaStreamDestroy(L.stream); L.stream = nullptr; }
    if (L.pinned) { cudaFreeHost(L.pinned); L.pinned = nullptr; }
    if (L.dstatus) { cudaFree(L.dstatus); L.dstatus = nullptr; }
    if (L.ring.ring) { cudaFreeHost(L.ring.ring); L.ring.ring = nullptr; }
    if (L.share) { cudaFree(L.share); L.share = nullptr; }
  }
  void ctx_select(int idx) override { tl_selected_ctx = idx; }
  // Everything the calling thread issues from now on (collectives too) runs on context idx's lane; -1 unbinds.
  int bind_thread(int idx) {
    if (idx >= 0 && (idx >= BSHMEM_MAX_CTXS || !lanes_[idx].open)) return BSHMEM_ERR_INVALID;
    tl_bound_backend = idx >= 0 ? this : nullptr;
    tl_bound_ctx = idx;
    return BSHMEM_OK;
  }
  bool thread_is_bound() const { return tl_bound_backend == this && tl_bound_ctx >= 0; }
  Lane& lane() {
    int i = thread_is_bound() ? tl_bound_ctx : tl_selected_ctx;
    if (i < 0 || i >= BSHMEM_MAX_CTXS || !lanes_[i].open) i = 0;
    return lanes_[i];
  }
  // Collectives belong to no context: they run on the PE stream unless the thread is bound to a lane.
  Lane& coll_lane() { return thread_is_bound() ? lanes_[tl_bound_ctx] : lanes_[0]; }
  cudaStream_t stream_of(const Lane& L) const { return &L == &lanes_[0] ? stream_ : L.stream; }

  // ---- the message ring of a context (see k_ring) ----------------------------------------
  // The lane's stream for anything but a ring message: it follows the messages written so far.  Messages of other threads wait until
  // the operation is enqueued: to be called then, before the operation is waited for.
  struct Entry {
    cudaStream_t st;
    std::unique_lock<std::mutex> held;               // of a lane with a ring
    void enqueued() { if (held) held.unlock(); }
  };
  Entry enter(Lane& L) {
    if (L.ring.ring) return {stream_of(L), L.ring.stop()};
    return {stream_of(L), {}};
  }
  bool ring_takes(const Lane& L, const void* a, const void* b, uint64_t n, bool nbi) const {
    const bool skewed = ((reinterpret_cast<uintptr_t>(a) ^ reinterpret_cast<uintptr_t>(b)) & 15) != 0;
    return nbi && tl_local_is_device && n > 0 && n <= (skewed ? kSmallCopyMaxSkewed : kRingMessageMax) && L.ring.ring &&
           !thread_is_bound() &&
           ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) >> 48) == 0;
  }
  int ring_message(Lane& L, char* dst, const char* src, uint32_t n) {
    const int rc = L.ring.message(
        reinterpret_cast<uintptr_t>(dst), reinterpret_cast<uintptr_t>(src), n,
        [&](uint32_t from, uint32_t generation) -> int {
          if (n > kRingNarrowMax) RT_TRY(launch_small(k_ring_wide, kWideBlocks, kWideThreads, L.stream, L.ring.ring, L.share, from, generation));
          else RT_TRY(launch_small(k_ring, 1, kRingThreads, L.stream, L.ring.ring, from, generation));
          return BSHMEM_OK;
        },
        [&](auto arrived) {
          // a message that nobody waits for may be sent while another stream is captured: its wait for room is no part of that
          const RelaxedCapture relaxed;
          return poll(arrived, L.stream);
        });
    if (rc == BSHMEM_ERR_STATE) tl_err = "the context's messages were not taken";
    return rc;
  }

  bshmem_error_record_t last_record(bool clear) override {
    bshmem_error_record_t r = pinned_->err;
    if (clear) memset(&pinned_->err, 0, sizeof(pinned_->err));
    return r;
  }

  // ---- knobs used by the C entry points below ---------------------------------
  // (cudaStream_t)-1 selects the runtime's own stream; any other handle (0 = the legacy default stream) is used as given.
  void set_stream(cudaStream_t s) {
    stream_ = (s == reinterpret_cast<cudaStream_t>(-1)) ? own_stream_ : s;
    stream_tells_ = -1;
  }
  cudaStream_t stream() const { return stream_; }
  void set_blocking(bool b) { blocking_ = b; }
  void set_coll_ctas(int n) { if (n >= 1 && n <= BSHMEM_MAX_COLL_CTAS) coll_ctas_ = n; }
  void set_nvls(bool on) { use_nvls_ = on && heap_->mc_base != nullptr; }
  const State& state() const { return state_; }
  gpu::Heap* heap() const { return heap_; }
  unsigned long long* dstats() const { return dstats_; }
  void refresh_mc() { state_.mc_base = heap_->mc_base; }

  // a thread bound to a lane (the reverse-offload service thread) always completes what it issues: the device
  // producer that waits for its answer cannot synchronise a host stream
  bool blocking_now() const { return blocking_ || thread_is_bound(); }
  int finish(const char* what, cudaStream_t st) {
    if (!blocking_now()) return BSHMEM_OK;
    RT_TRY(cudaStreamSynchronize(st));
    return check_device_error(what);
  }

  // Waits until the kernel that got this ticket has signalled.  Polls for about 50 us; what takes longer (a wait_until,
  // a busy stream) or went wrong is left to a stream synchronisation.
  template <class Arrived>
  int poll(Arrived arrived, cudaStream_t st) {
    for (int i = 0; i < 2000; ++i) {
      if (arrived()) return BSHMEM_OK;
#if defined(__x86_64__)
      __builtin_ia32_pause();
#endif
    }
    RT_TRY(cudaStreamSynchronize(st));
    return BSHMEM_OK;
  }
  int wait_done(const Ticket& t, cudaStream_t st) {
    const auto* w = reinterpret_cast<const std::atomic<uint64_t>*>(t.done.word);
    return poll([&] { return w->load(std::memory_order_acquire) == t.done.token; }, st);
  }
  static bool read_result(const Ticket& t, uint64_t* out) {
    const auto* w = reinterpret_cast<const std::atomic<uint64_t>*>(t.done.word);
    const uint32_t tag = (uint32_t)t.done.token;
    const uint64_t lo = w[0].load(std::memory_order_acquire), hi = w[1].load(std::memory_order_acquire);
    if ((uint32_t)(lo >> 32) != tag || (uint32_t)(hi >> 32) != tag) return false;
    *out = (uint32_t)lo | hi << 32;
    return true;
  }
  int wait_result(const Ticket& t, cudaStream_t st, uint64_t* out) {
    const int rc = poll([&] { return read_result(t, out); }, st);
    if (rc != BSHMEM_OK) return rc;
    if (!read_result(t, out)) { tl_err = "the call's kernel ended without an answer"; return BSHMEM_ERR_STATE; }
    return BSHMEM_OK;
  }

  // ---- blocking calls through a block that is there already (see k_calls) ----------------
  // Whether the call has been carried out and answered() is true.  Where it is not, nothing has happened: the caller launches.
  template <class Answered>
  bool served(const Lane& L, const Ticket& t, Call& call, Answered answered, AskAhead* ahead = nullptr) {
    if (&L != &lanes_[0] || thread_is_bound() || stream_tells_ == 0) return false;
    const std::unique_lock<std::mutex> lock(calls_mu_, std::try_to_lock);
    if (!lock) return false;
    const long long now = std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now().time_since_epoch()).count();
    if (!series_.long_enough(now) || (ahead && !ahead->now())) return false;
    const RelaxedCapture relaxed;                    // the questions are no part of another stream's capture
    if (stream_tells_ < 0) {                         // not where the stream is set: it may be capturing
      unsigned flags = cudaStreamNonBlocking;
      if (stream_ && stream_ != cudaStreamLegacy && cudaStreamGetFlags(stream_, &flags) != cudaSuccess) {
        cudaGetLastError();
        flags = 0;
      }
      stream_tells_ = (flags & cudaStreamNonBlocking) ? 1 : 0;
      if (!stream_tells_) return false;
    }
    // a launch of this lane's last call has answered, and may be about to end
    int asks = calls_served_ ? 1 : 4;
    calls_served_ = false;
    while (cudaStreamQuery(stream_) != cudaSuccess) {
      cudaGetLastError();                            // "not ready" is not for somebody's next launch
      if (--asks) continue;
      series_.refused();
      return false;
    }
    bool done = false;
    if (calls_.ready()) {
      call.set(CALL_DONE, reinterpret_cast<uintptr_t>(t.done.word)).set(CALL_TOKEN, t.done.token);
      done = calls_.run(call, [](uint32_t, uint32_t) -> int { return BSHMEM_ERR_STATE; }, answered, [&]() -> int {
        RT_TRY(cudaStreamSynchronize(calls_stream_));  // the block is there: to its end
        return BSHMEM_OK;
      });
    }
    if (calls_block_ && !calls_.serving()) {
      calls_block_ = false;
      series_.ended(calls_.taken());
    }
    calls_wanted_ = !done && !calls_block_ && series_.long_enough();
    calls_served_ = done;
    return done;
  }
  // Between a call's launch and its wait: the block for the calls to come, if the call would have liked one.
  void prepare_calls() {
    if (!calls_wanted_.load(std::memory_order_relaxed)) return;
    const std::unique_lock<std::mutex> lock(calls_mu_, std::try_to_lock);
    if (!lock || !calls_wanted_.exchange(false)) return;
    calls_block_ = calls_.prepare([&](uint32_t first, uint32_t generation) -> int {
      RT_TRY(launch_small(k_calls, 1, kCallThreads, calls_stream_, state_, calls_.slot, first, generation));
      return BSHMEM_OK;
    });
  }
  bool served(const Lane& L, const Ticket& t, Call& call, uint64_t* result, AskAhead* ahead = nullptr) {
    return served(L, t, call, [&] { return read_result(t, result); }, ahead);
  }

  int check_device_error(const char* what) {
    if (pinned_->err.code != 0) {
      int code = (int)pinned_->err.code;
      tl_err = std::string(what) + ": device-side " + bshmem_status_string(code) + " at site " +
             std::to_string(pinned_->err.where) + " waiting for pe " + std::to_string(pinned_->err.pe);
      return code;
    }
    return BSHMEM_OK;
  }

  // ---- RMA ------------------------------------------------------------------------
  // Small messages between device buffers go through a kernel (k_copy_small); everything else — host buffers, whose
  // lifetime and staging the copy engine handles, and messages it moves faster — through cudaMemcpyAsync.
  int move(char* dst, const char* src, uint64_t n, cudaStream_t st) {
    const bool skewed = ((reinterpret_cast<uintptr_t>(dst) ^ reinterpret_cast<uintptr_t>(src)) & 15) != 0;
    if (tl_local_is_device && n <= (skewed ? kSmallCopyMaxSkewed : kSmallCopyMax)) {
      RT_TRY(launch_small(k_copy_small, (unsigned)((n + kSmallPiece - 1) / kSmallPiece), n >= kSmallPiece ? 256 : 64, st, dst, src, n));
    } else {
      RT_TRY(cudaMemcpyAsync(dst, src, n, cudaMemcpyDefault, st));
    }
    return BSHMEM_OK;
  }
  int put(int pe, uint64_t dst_off, const void* local, uint64_t n, bool nbi) override {
    Lane& L = lane();
    if (ring_takes(L, heap_->base[pe] + dst_off, local, n, nbi)) return ring_message(L, heap_->base[pe] + dst_off, static_cast<const char*>(local), (uint32_t)n);
    Entry e = enter(L);
    const int rc = move(heap_->base[pe] + dst_off, static_cast<const char*>(local), n, e.st);
    e.enqueued();
    if (rc != BSHMEM_OK || nbi) return rc;
    return finish("put", e.st);
  }
  int get(int pe, void* local, uint64_t src_off, uint64_t n, bool nbi) override {
    Lane& L = lane();
    if (ring_takes(L, heap_->base[pe] + src_off, local, n, nbi)) return ring_message(L, static_cast<char*>(local), heap_->base[pe] + src_off, (uint32_t)n);
    Entry e = enter(L);
    const int rc = move(static_cast<char*>(local), heap_->base[pe] + src_off, n, e.st);
    e.enqueued();
    if (rc != BSHMEM_OK || nbi) return rc;
    return finish("get", e.st);
  }
  int put_signal(int pe, uint64_t dst_off, const void* local, uint64_t n, uint64_t sig_off, uint64_t sig_val, int sig_op,
                 bool nbi) override {
    Lane& L = lane();
    const bool wait = !nbi && blocking_now();
    const Ticket t(wait ? &L : nullptr);
    const bool skewed = (((reinterpret_cast<uintptr_t>(heap_->base[pe]) + dst_off) ^ reinterpret_cast<uintptr_t>(local)) & 15) != 0;
    if (wait && (n == 0 || (tl_local_is_device && n <= (skewed ? kSmallSignalMax : kServedSignalMax)))) {
      Call call(CALL_PUT_SIGNAL, 0, sig_op, 0);
      call.set(CALL_ADDR, reinterpret_cast<uintptr_t>(heap_->base[pe] + dst_off)).set(CALL_VALUE, sig_val);
      call.set(CALL_OTHER, reinterpret_cast<uintptr_t>(local)).set(CALL_SIG, reinterpret_cast<uintptr_t>(heap_->base[pe] + sig_off));
      call.w[CALL_BYTES] = (uint32_t)n;
      const auto* w = reinterpret_cast<const std::atomic<uint64_t>*>(t.done.word);
      if (served(L, t, call, [&] { return w->load(std::memory_order_acquire) == t.done.token; })) return check_device_error("put_signal");
    }
    Entry e = enter(L);
    const cudaStream_t st = e.st;
    if (n == 0 || (tl_local_is_device && n <= kSmallSignalMax)) {
      RT_TRY(launch_small(k_put_signal, 1, n > 4096 ? 512 : 128, st, state_, heap_->base[pe] + dst_off, static_cast<const char*>(local), n,
                                                       reinterpret_cast<uint64_t*>(heap_->base[pe] + sig_off), sig_val, sig_op, t.done));
    } else {
      const int rc = move(heap_->base[pe] + dst_off, static_cast<const char*>(local), n, st);
      if (rc != BSHMEM_OK) return rc;
      RT_TRY(launch_small(k_signal, 1, 1, st, state_, pe, sig_off, sig_val, sig_op, t.done));
    }
    e.enqueued();
    if (!wait) return BSHMEM_OK;
    prepare_calls();
    const int rc = wait_done(t, st);
    return rc != BSHMEM_OK ? rc : check_device_error("put_signal");
  }
  int read_word(int pe, uint64_t off, uint64_t size, uint64_t* out) override {
    Lane& L = lane();
    const Ticket t(&L);
    Call call(CALL_READ, 0, 0, (int)size);
    call.set(CALL_ADDR, reinterpret_cast<uintptr_t>(heap_->base[pe] + off));
    if (served(L, t, call, out)) return blocking_now() ? check_device_error("get") : BSHMEM_OK;
    Entry e = enter(L);
    RT_TRY(launch_small(k_read_word, 1, 1, e.st, heap_->base[pe] + off, (int)size, t.done));
    e.enqueued();
    prepare_calls();
    const int rc = wait_result(t, e.st, out);      // the value is the call's result: it is waited for in stream mode too
    if (rc != BSHMEM_OK) return rc;
    return blocking_now() ? check_device_error("get") : BSHMEM_OK;
  }
  int write_word(int pe, uint64_t off, uint64_t bits, uint64_t size) override {
    const Entry e = enter(lane());
    RT_TRY(launch_small(k_write_word, 1, 1, e.st, heap_->base[pe] + off, bits, (int)size));
    return BSHMEM_OK;
  }
  int amo(int pe, uint64_t off, int dtype, int op, uint64_t value, uint64_t cond, uint64_t* fetched) override {
    Lane& L = lane();
    const bool fetching = op <= BSHMEM_AMO_FETCH_CSWAP || op == BSHMEM_AMO_SWAP || (op >= BSHMEM_AMO_FETCH_AND && op <= BSHMEM_AMO_FETCH_XOR);
    const bool wait = fetching || blocking_now();
    const Ticket t(wait ? &L : nullptr);
    if (wait) {
      Call call(CALL_AMO, dtype, op, (int)bshmem_dtype_size(dtype));
      call.set(CALL_ADDR, reinterpret_cast<uintptr_t>(heap_->base[pe] + off)).set(CALL_VALUE, value).set(CALL_OTHER, cond);
      uint64_t old = 0;
      if (served(L, t, call, &old)) {
        if (fetched) *fetched = old;
        return BSHMEM_OK;
      }
    }
    Entry e = enter(L);
    RT_TRY(launch_small(k_amo, 1, 1, e.st, state_, pe, off, dtype, op, value, cond, t.done));
    e.enqueued();
    if (wait) {
      prepare_calls();
      uint64_t old = 0;
      const int rc = wait_result(t, e.st, &old);
      if (rc != BSHMEM_OK) return rc;
      if (fetched) *fetched = old;
    }
    return BSHMEM_OK;
  }
  // operations of one stream reach each PE in order; so do ring messages across this
  int fence() override {
    Lane& L = lane();
    if (L.ring.ring) L.ring.fence();
    return BSHMEM_OK;
  }
  int quiet() override {
    // Stream mode: operations of the PE's stream complete in order, and whatever the caller
    // enqueues next on that stream runs after them, so there is nothing to wait for on the
    // host; bshmem_gpu_synchronize() is the explicit host-side wait.
    if (!blocking_now()) return BSHMEM_OK;
    Lane& L = lane();                                     // this context's operations only
    uint32_t head;
    if (L.ring.ring && L.ring.serving(&head)) {
      for (int i = 0; i < 2000; ++i) {
        if (L.ring.done(head)) return check_device_error("quiet");
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
      }
    }
    const cudaStream_t st = enter(L).st;
    RT_TRY(cudaStreamSynchronize(st));
    if (L.ring.ring && L.ring.failed()) {
      tl_err = "the context's messages were not taken";
      return BSHMEM_ERR_STATE;
    }
    return check_device_error("quiet");
  }
  int wait_until(uint64_t off, int dtype, int cmp, uint64_t value, uint64_t timeout_us) override {
    State s = state_;
    s.timeout_ns = timeout_us * 1000ull;
    Lane& L = lane();
    const bool wait = blocking_now();
    if (wait) {                                      // what holds already needs no kernel that waits for it
      const Ticket asked(&L);
      Call call(CALL_TEST, dtype, cmp, 0);
      call.set(CALL_ADDR, reinterpret_cast<uintptr_t>(local_base() + off)).set(CALL_VALUE, value);
      uint64_t answer = 0;
      if (served(L, asked, call, &answer, &waits_)) {
        const bool holds = (uint32_t)answer == BSHMEM_OK;
        const std::lock_guard<std::mutex> lock(calls_mu_);
        waits_.told(holds);
        if (holds) return BSHMEM_OK;
      }
    }
    const Ticket t(wait ? &L : nullptr);
    Entry e = enter(L);
    RT_TRY(launch_small(k_wait_until, 1, 1, e.st, s, off, dtype, cmp, value, t.done));
    e.enqueued();
    if (!wait) return BSHMEM_OK;
    prepare_calls();
    uint64_t status = 0;
    int rc = wait_result(t, e.st, &status);
    if (rc != BSHMEM_OK) return rc;
    rc = (int)(uint32_t)status;
    if (rc != BSHMEM_OK) tl_err = "wait_until: device-side timeout";
    return rc;
  }
  int test(uint64_t off, int dtype, int cmp, uint64_t value, int* result) override {
    State s = state_;
    s.timeout_ns = 0;   // a wait that gives up at once is a test
    s.err = nullptr;
    s.stats = nullptr;
    Lane& L = lane();
    const Ticket t(&L);
    Entry e = enter(L);
    RT_TRY(launch_small(k_wait_until, 1, 1, e.st, s, off, dtype, cmp, value, t.done));
    e.enqueued();
    uint64_t status = 0;
    const int rc = wait_result(t, e.st, &status);
    if (rc != BSHMEM_OK) return rc;
    *result = (uint32_t)status == BSHMEM_OK ? 1 : 0;
    return BSHMEM_OK;
  }

  // ---- collectives ---------------------------------------------------------------------
  DTeam team_of(const CollGroup& g) const {
    DTeam t;
    t.pe_start = g.set.pe_start; t.stride = g.set.stride; t.size = g.set.size; t.my_idx = g.my_idx;
    t.slot = g.slot; t.reserved = 0; t.psync = nullptr;
    return t;
  }

  int launch(const CollGroup& g, CollArgs a, uint64_t bytes, const char* what) {
    if (heap_->mode == gpu::HEAP_LOCAL_GROUP) {
      // PEs of a local group share one GPU: a per-PE launch that waits for the others must not
      // exist.  Host syncs are no-ops (the caller owns ordering); data collectives go through
      // bshmem_gpu_group_collective, which runs all PEs in one launch.
      if (a.kind == BSHMEM_COLL_SYNC || a.kind == BSHMEM_COLL_BARRIER) return BSHMEM_OK;
      tl_err = std::string(what) + ": use the group collective entry for a local group";
      return BSHMEM_ERR_UNSUPPORTED;
    }
    a.psync_off = g.psync_off;
    // in-switch reductions pay off from four PEs on (with two, pulling the one peer's data is faster)
    a.use_nvls = (use_nvls_ && (heap_->n_pes > 2 || a.kind == BSHMEM_COLL_FCOLLECT)) ? 1 : 0;
    int ctas = 1;
    if (g.slot >= 0 && bytes > (32u << 10)) {   // one CTA per 32 KiB: remote latency, not bandwidth, bounds a CTA
      ctas = (int)((bytes + (32u << 10) - 1) / (32u << 10));
      if (ctas > coll_ctas_) ctas = coll_ctas_;
    }
    Lane& L = coll_lane();
    const bool main_lane = &L == &lanes_[0];   // the slot / staging fast paths count calls per PE, so only the PE stream takes them
    a.ll_epoch = 0;
    const uint64_t unit = bshmem_dtype_size(a.dtype) > 4 ? bshmem_dtype_size(a.dtype) : 4;
    if (main_lane && a.kind == BSHMEM_COLL_REDUCE && g.slot == 0 && g.set.size == heap_->n_pes &&
        bytes > BSHMEM_LL_PAYLOAD_BYTES && bytes <= BSHMEM_LLB_PAYLOAD_BYTES && bytes % unit == 0 &&
        ((a.dst_off | a.src_off) & (unit - 1)) == 0) {
      // mid-size allreduce on the world team: one exchange through the per-sender slots.  The conditions are exactly
      // those under which the kernel takes that path, and every PE makes the same sequence of such calls, so this
      // counter is the same everywhere and its parity alternates between consecutive uses of the slots.
      a.ll_epoch = ++ll_epoch_;
      ctas = (int)((bytes + (4u << 10) - 1) / (4u << 10));      // 4 KiB of payload per block: four words per thread, polled one after the other
      if (ctas > coll_ctas_) ctas = coll_ctas_;
    }
    // One exchange through the staging region instead of sync + work + barrier: world team, what a PE receives fits a
    // staging half, 16-byte granular.  Every PE evaluates the same conditions on the same arguments, so the call
    // number (and with it the staging half) is the same everywhere.
    a.stage_seq = 0;
    a.stage_oneshot = 0;
    if (main_lane && g.slot == 0 && g.set.size == heap_->n_pes && heap_->n_pes > 1 && a.ll_epoch == 0 && bytes >= 16 &&
        bytes + 4096 <= BSHMEM_STAGE_BYTES && ((a.dst_off | a.src_off) & 15) == 0) {
      const uint64_t es = bshmem_dtype_size(a.dtype);
      bool fits = false;
      switch (a.kind) {
        case BSHMEM_COLL_FCOLLECT: case BSHMEM_COLL_ALLTOALL: fits = a.n % 16 == 0; break;
        case BSHMEM_COLL_REDUCE_SCATTER: fits = (a.n * es) % 16 == 0; break;
        // the multicast reduction needs no staging; below the one-shot limit the pull form is a single pass
        case BSHMEM_COLL_REDUCE: fits = !(a.use_nvls && a.op == BSHMEM_SUM && (a.dtype == BSHMEM_FLOAT || a.dtype == BSHMEM_BF16)) &&
                                        bytes > BSHMEM_LLB_PAYLOAD_BYTES; break;
        default: break;
      }
      if (fits) {
        a.stage_seq = ++stage_seq_;
        if (a.kind == BSHMEM_COLL_REDUCE) {
          // one exchange moves (P-1) vectors per PE, two exchanges 2 (P-1)/P: the single exchange wins while the
          // extra (P-1)(P-2)/P vectors cost less than a flag exchange (about 8 us, i.e. about 5 MiB on the links)
          const uint64_t P = (uint64_t)heap_->n_pes;
          const uint64_t slot = (BSHMEM_STAGE_BYTES / P) & ~(uint64_t)15;
          if (bytes <= slot && bytes * (P - 1) * (P - 2) / P <= (5ull << 20)) a.stage_oneshot = 1;
        }
        // every channel runs its own flag exchange and the kernel ends with the slowest one, so a staged call wants
        // few, fat channels; a block pushes its share to P-1 peers at about 50 GB/s, so the share shrinks with P:
        // 64 KiB with two PEs, 32 KiB with four, 16 KiB with eight and more
        uint64_t gran = (128ull << 10) / (uint64_t)heap_->n_pes;
        if (gran < (16u << 10)) gran = 16u << 10;
        ctas = (int)((bytes + gran - 1) / gran);
        if (ctas > coll_ctas_) ctas = coll_ctas_;
        if (ctas < 1) ctas = 1;
      }
    }
    Entry e = enter(L);
    const cudaStream_t st = e.st;
    RT_TRY(collk::launch(state_, team_of(g), a, ctas, L.dstatus, st));
    e.enqueued();
    if (!blocking_now()) return BSHMEM_OK;
    int rc = 0;
    RT_TRY(cudaMemcpyAsync(&rc, L.dstatus, sizeof(int), cudaMemcpyDeviceToHost, st));
    RT_TRY(cudaStreamSynchronize(st));
    if (rc != 0) {
      cudaMemsetAsync(L.dstatus, 0, sizeof(int), st);
      check_device_error(what);
      if (tl_err.empty()) tl_err = std::string(what) + " failed on the device";
      return rc;
    }
    return BSHMEM_OK;
  }

  int sync(const CollGroup& g) override {
    CollArgs a{}; a.kind = BSHMEM_COLL_SYNC;
    return launch(g, a, 0, "sync");
  }
  int broadcast(const CollGroup& g, uint64_t d, uint64_t s, uint64_t nbytes, int root) override {
    CollArgs a{}; a.kind = BSHMEM_COLL_BROADCAST; a.dst_off = d; a.src_off = s; a.n = nbytes; a.root = root;
    return launch(g, a, nbytes, "broadcast");
  }
  int reduce(const CollGroup& g, int dtype, int op, uint64_t d, uint64_t s, uint64_t nelems) override {
    CollArgs a{}; a.kind = BSHMEM_COLL_REDUCE; a.dtype = dtype; a.op = op; a.dst_off = d; a.src_off = s; a.n = nelems;
    return launch(g, a, nelems * bshmem_dtype_size(dtype), "to_all");
  }
  int reduce_root(const CollGroup& g, int dtype, int op, uint64_t d, uint64_t s, uint64_t nelems, int root) override {
    CollArgs a{}; a.kind = BSHMEM_COLL_REDUCE_ROOT; a.dtype = dtype; a.op = op; a.dst_off = d; a.src_off = s; a.n = nelems; a.root = root;
    return launch(g, a, nelems * bshmem_dtype_size(dtype), "reduce");
  }
  int reduce_scatter(const CollGroup& g, int dtype, int op, uint64_t d, uint64_t s, uint64_t per_pe) override {
    CollArgs a{}; a.kind = BSHMEM_COLL_REDUCE_SCATTER; a.dtype = dtype; a.op = op; a.dst_off = d; a.src_off = s; a.n = per_pe;
    return launch(g, a, per_pe * bshmem_dtype_size(dtype) * g.size(), "reduce_scatter");
  }
  int fcollect(const CollGroup& g, uint64_t d, uint64_t s, uint64_t nbytes) override {
    CollArgs a{}; a.kind = BSHMEM_COLL_FCOLLECT; a.dst_off = d; a.src_off = s; a.n = nbytes;
    return launch(g, a, nbytes * g.size(), "fcollect");
  }
  int alltoall(const CollGroup& g, uint64_t d, uint64_t s, uint64_t nbytes) override {
    CollArgs a{}; a.kind = BSHMEM_COLL_ALLTOALL; a.dst_off = d; a.src_off = s; a.n = nbytes;
    return launch(g, a, nbytes * g.size(), "alltoall");
  }
  int exchange_u64(const CollGroup& g, uint64_t mine, uint64_t* all) override {
    if (g.slot < 0) return BSHMEM_ERR_UNSUPPORTED;
    CollArgs a{}; a.kind = BSHMEM_COLL_EXCHANGE; a.n = mine;
    bool was = blocking_;
    blocking_ = true;
    int rc = launch(g, a, 0, "exchange");
    blocking_ = was;
    if (rc != BSHMEM_OK) return rc;
    RT_TRY(cudaMemcpy(all, local_base() + BSHMEM_OFF_XCHG + (uint64_t)g.slot * BSHMEM_MAX_PES * 8, 8 * g.size(),
                      cudaMemcpyDeviceToHost));
    // a second sync keeps a fast member's next exchange from overwriting rows still being read
    CollArgs b{}; b.kind = BSHMEM_COLL_SYNC;
    blocking_ = true;
    rc = launch(g, b, 0, "exchange");
    blocking_ = was;
    return rc;
  }
  int global_exit(int) override { return BSHMEM_OK; }   // the Python layer raises the job-wide flag in the store
  int zero_local(uint64_t off, uint64_t n) override {
    RT_TRY(cudaMemsetAsync(local_base() + off, 0, n, stream_));
    RT_TRY(cudaStreamSynchronize(stream_));
    return BSHMEM_OK;
  }
  void reset_slot(int slot) override {
    if (slot <= 0 || slot >= BSHMEM_MAX_TEAMS) return;
    cudaStreamSynchronize(stream_);
    cudaMemset(local_base() + BSHMEM_OFF_FLAGS + (uint64_t)slot * BSHMEM_MAX_COLL_CTAS * BSHMEM_MAX_PES * 8, 0,
               (uint64_t)BSHMEM_MAX_COLL_CTAS * BSHMEM_MAX_PES * 8);
    cudaMemset(local_base() + BSHMEM_OFF_EPOCHS + (uint64_t)slot * BSHMEM_MAX_COLL_CTAS * 8, 0, BSHMEM_MAX_COLL_CTAS * 8);
    // the slot's low-latency allreduce block: epoch word and per-sender slots start from zero for the new team
    cudaMemset(local_base() + BSHMEM_OFF_LLT + (uint64_t)slot * BSHMEM_LLT_TEAM_BYTES, 0, BSHMEM_LLT_TEAM_BYTES);
  }

  int cuda_fail(const char* what, cudaError_t e) {
    tl_err = std::string(what) + ": " + cudaGetErrorString(e);
    return BSHMEM_ERR_CUDA;
  }

  int* dstatus() const { return dstatus_; }

  // A collective of the local group whose first PE this is: one pass over all members' memory where every member of the team is
  // here and the call's blocks fit the device one to a multiprocessor, else the multi-PE algorithms in a cooperative launch (which
  // turns away what does not fit).  The PE table of that one stays on the device and is rewritten only when it differs
  // from the last call's; completion and status come back through pinned words.  (With a table allocated,
  // copied and freed per call and a synchronous read of the status, the call cost 40 us around a 16 us kernel.)
  int group_launch(const State* hs, const DTeam* ht, int n, const CollArgs& a, int ctas) {
    std::lock_guard<std::mutex> lock(group_mu_);
    const Ticket t(&lanes_[0]);
    int* status = &pinned_->status[t.slot];
    *status = 0;
    collk::GroupDone done;
    done.word = t.done.word;
    done.token = t.done.token;
    if (!group_dev_) {
      // on the stream of the launch: it may be one that does not wait for the default stream
      char* mem = nullptr;
      RT_TRY(cudaMalloc(&mem, sizeof(GroupTable) + 16));
      const cudaError_t e = cudaMemsetAsync(mem, 0, sizeof(GroupTable) + 16, stream_);
      if (e != cudaSuccess) { cudaFree(mem); RT_TRY(e); }
      group_dev_ = mem;
      memset(&group_host_, 0, sizeof(group_host_));
    }
    done.count = reinterpret_cast<unsigned int*>(group_dev_ + sizeof(GroupTable));
    collk::GroupPass pass;
    int words = 0;
    auto one_pass = [&] {
      pass.a = a;
      pass.done = done;
      words = ctas * pass.size <= collk::kPassWords ? ctas * pass.size : 0;
      if (words) {
        pass.done.word = pinned_->pass;
        pass.done.count = nullptr;
      }
      const cudaError_t e = collk::launch_pass(pass, ctas, stream_);
      if (e == cudaSuccess) return (int)BSHMEM_OK;
      cudaGetLastError();                              // not for somebody's next launch
      words = 0;
      return (int)BSHMEM_ERR_CUDA;
    };
    auto cooperative = [&]() -> int {
      GroupTable img;
      memset(&img, 0, sizeof(img));
      memcpy(img.states, hs, sizeof(State) * n);
      memcpy(img.teams, ht, sizeof(DTeam) * n);
      if (memcmp(&img, &group_host_, sizeof(img)) != 0) {
        RT_TRY(cudaMemcpyAsync(group_dev_, &img, sizeof(img), cudaMemcpyHostToDevice, stream_));
        group_host_ = img;
      }
      GroupTable* dev = reinterpret_cast<GroupTable*>(group_dev_);
      const cudaError_t e = collk::launch_group(dev->states, dev->teams, a, ctas, n, status, stream_, done);
      if (e == cudaSuccess) return BSHMEM_OK;
      cudaGetLastError();        // reported here, not at somebody's next launch
      tl_err = std::string("cooperative launch: ") + cudaGetErrorString(e);
      return BSHMEM_ERR_CUDA;
    };
    int rc = launch_preferred(ctas * n <= sms_ && passes(hs, ht, n, a, &pass), (int)BSHMEM_OK, one_pass, cooperative);
    if (rc == BSHMEM_OK)
      rc = words ? poll([&] {
             while (words && reinterpret_cast<const std::atomic<uint64_t>&>(pinned_->pass[words - 1]).load(std::memory_order_acquire) == t.done.token) --words;
             return words == 0;
           }, stream_)
                 : wait_done(t, stream_);
    if (rc != BSHMEM_OK || *status == BSHMEM_OK) return rc;
    tl_err = std::string("device-side ") + bshmem_status_string(*status);
    return *status;
  }

 private:
  // Whether a group's collective can run as one pass (and over which members): every member of the team is here, they agree on where each
  // of them lives, and the call is one that the pass knows.  What does not fit keeps its own answer from the general form, errors included.
  static bool passes(const State* hs, const DTeam* ht, int n, const CollArgs& a, collk::GroupPass* pass) {
    if (!collk::pass_kind(a.kind)) return false;
    int size = 0, found = 0, slot = -1;
    bool seen[BSHMEM_MAX_PES] = {};
    for (int i = 0; i < n; ++i) {
      const int k = ht[i].my_idx;
      if (k < 0) continue;
      if (found++ == 0) { size = ht[i].size; slot = ht[i].slot; }
      if (size < 1 || size > BSHMEM_MAX_PES || k >= size || seen[k] || ht[i].size != size || ht[i].slot != slot || slot < 0) return false;
      seen[k] = true;
      pass->base[k] = hs[i].heap_base[hs[i].my_pe];
      pass->stats[k] = hs[i].stats;
      pass->pe[k] = hs[i].my_pe;
      if (!hs[i].one_gpu || reinterpret_cast<uintptr_t>(pass->base[k]) & 15) return false;
    }
    if (found == 0 || found != size) return false;
    const bool rooted = a.kind == BSHMEM_COLL_BROADCAST || a.kind == BSHMEM_COLL_REDUCE_ROOT;
    if (rooted && (a.root < 0 || a.root >= size)) return false;
    for (int i = 0; i < n; ++i)
      for (int k = 0; k < size && ht[i].my_idx >= 0; ++k) {
        const int pe = ht[i].pe_start + k * ht[i].stride;
        if (pe < 0 || pe >= hs[i].n_pes || hs[i].heap_base[pe] != pass->base[k]) return false;
      }
    pass->size = size;
    return true;
  }

  struct GroupTable {
    State states[BSHMEM_MAX_PES];
    DTeam teams[BSHMEM_MAX_PES];
  };
  std::mutex group_mu_;
  char* group_dev_ = nullptr;           // GroupTable, then the count of finished blocks
  GroupTable group_host_;               // what group_dev_ holds
  gpu::Heap* heap_;
  bool own_heap_;
  State state_{};
  cudaStream_t own_stream_ = nullptr, stream_ = nullptr;
  Pinned* pinned_ = nullptr;
  unsigned long long* dstats_ = nullptr;
  int* dstatus_ = nullptr;
  bool blocking_ = true;
  bool use_nvls_ = false;
  int coll_ctas_ = 32, sms_ = 0;
  std::atomic<int> stream_tells_{1};    // whether its being idle says that its launches would run at once (see k_calls); -1: not known yet
  std::mutex calls_mu_;                 // one request at a time
  std::atomic<bool> calls_wanted_{false};
  bool calls_block_ = false;            // launched, and not seen to have ended
  bool calls_served_ = false;           // the last call was carried out by a block
  CallSeries series_;
  AskAhead waits_;
  CallWriter calls_;
  cudaStream_t calls_stream_ = nullptr;
  Lane lanes_[BSHMEM_MAX_CTXS];
  unsigned long long ll_epoch_ = 0;     // epochs of host-launched low-latency allreduces
  unsigned long long stage_seq_ = 0;    // call numbers of staged one-exchange collectives
};

GpuBackend* gpu_of(bshmem_handle_t h) {
  if (!h || h->finalized || !h->backend) return nullptr;
  return dynamic_cast<GpuBackend*>(h->backend.get());
}

thread_local std::string g_err;

}  // namespace

// ---------------------------------------------------------------------------------
// C entry points (bshmem_gpu.h)
// ---------------------------------------------------------------------------------
extern "C" {

const char* bshmem_gpu_last_error(void) {
  if (!g_err.empty()) return g_err.c_str();
  return gpu::heap_error().c_str();
}

int bshmem_gpu_heap_create(int my_pe, int n_pes, uint64_t heap_bytes, int device, int mode, void** heap) {
  gpu::Heap* h = nullptr;
  g_err.clear();                 // what failed before on this thread is not this call's message
  int rc = gpu::heap_create(my_pe, n_pes, heap_bytes, device, mode, &h);
  if (rc == BSHMEM_OK) *heap = h;
  return rc;
}
int bshmem_gpu_heap_create_local_group(int n_pes, uint64_t heap_bytes, int device, void** heaps) {
  g_err.clear();
  return gpu::heap_create_local_group(n_pes, heap_bytes, device, reinterpret_cast<gpu::Heap**>(heaps));
}
int bshmem_gpu_heap_export_fd(void* heap, int* fd) { return gpu::heap_export_fd(static_cast<gpu::Heap*>(heap), fd); }
int bshmem_gpu_heap_import_fd(void* heap, int pe, int fd) { return gpu::heap_import_fd(static_cast<gpu::Heap*>(heap), pe, fd); }
int bshmem_gpu_heap_export_ipc(void* heap, void* handle64) { return gpu::heap_export_ipc(static_cast<gpu::Heap*>(heap), handle64); }
int bshmem_gpu_heap_import_ipc(void* heap, int pe, const void* handle64) { return gpu::heap_import_ipc(static_cast<gpu::Heap*>(heap), pe, handle64); }
int bshmem_gpu_multicast_supported(int device) { return gpu::heap_multicast_supported(device); }
int bshmem_gpu_multicast_create(void* heap, int* fd) { return gpu::heap_multicast_create(static_cast<gpu::Heap*>(heap), fd); }
int bshmem_gpu_multicast_import(void* heap, int fd) { return gpu::heap_multicast_import(static_cast<gpu::Heap*>(heap), fd); }
int bshmem_gpu_multicast_add_device(void* heap) { return gpu::heap_multicast_add_device(static_cast<gpu::Heap*>(heap)); }
int bshmem_gpu_multicast_bind(void* heap) { return gpu::heap_multicast_bind(static_cast<gpu::Heap*>(heap)); }
int bshmem_gpu_heap_destroy(void* heap) { return gpu::heap_destroy(static_cast<gpu::Heap*>(heap)); }
uint64_t bshmem_gpu_heap_bytes(void* heap) { return static_cast<gpu::Heap*>(heap)->heap_bytes; }

int bshmem_gpu_init(void* heap, const bshmem_config_t* cfg, int coll_ctas, int own_heap, bshmem_handle_t* out) {
  if (!heap || !out) return BSHMEM_ERR_INVALID;
  bshmem_config_t c;
  if (cfg) c = *cfg; else bshmem_config_default(&c);
  if (c.timeout_us == 0) c.timeout_us = 30ull * 1000 * 1000;
  auto* be = new GpuBackend(static_cast<gpu::Heap*>(heap), own_heap != 0);
  int rc = be->setup(c, coll_ctas);
  // Load every kernel of this library now.  With lazy module loading the first launch of a kernel
  // can need a device-wide quiet point; if that first launch came from the proxy thread, or a host thread that
  // answers, while a user kernel is spinning on the answer, neither would ever finish.
  {
    cudaFuncAttributes fa;
    cudaFuncGetAttributes(&fa, k_amo);
    cudaFuncGetAttributes(&fa, k_wait_until);
    cudaFuncGetAttributes(&fa, k_signal);
    cudaFuncGetAttributes(&fa, k_put_signal);
    cudaFuncGetAttributes(&fa, k_read_word);
    cudaFuncGetAttributes(&fa, k_write_word);
    cudaFuncGetAttributes(&fa, k_copy_small);
    cudaFuncGetAttributes(&fa, k_ring);
    cudaFuncGetAttributes(&fa, k_ring_wide);
    cudaFuncGetAttributes(&fa, k_calls);
    cudaFuncGetAttributes(&fa, k_rma);
    cudaFuncGetAttributes(&fa, k_rma_bulk);
    collk::preload();
  }
  if (rc != BSHMEM_OK) { g_err = be->last_error(); delete be; return rc; }
  *out = make_runtime(std::unique_ptr<Backend>(be), &c);
  return BSHMEM_OK;
}

int bshmem_gpu_set_stream(bshmem_handle_t h, void* stream) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  g->set_stream(static_cast<cudaStream_t>(stream));
  return BSHMEM_OK;
}
// Binds the calling thread to host context `ctx` of this PE: everything the thread issues from now on, collectives
// included, runs on that context's stream and completes before the call returns; ctx < 0 unbinds.  The
// reverse-offload service thread uses this so that its work never queues behind the kernel that waits for it.
int bshmem_gpu_bind_thread_ctx(bshmem_handle_t h, int ctx) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  return g->bind_thread(ctx);
}
int bshmem_gpu_get_device(bshmem_handle_t h, int* device) {
  GpuBackend* g = gpu_of(h);
  if (!g || !device) return BSHMEM_ERR_STATE;
  *device = g->heap()->device;
  return BSHMEM_OK;
}
int bshmem_gpu_get_stream(bshmem_handle_t h, void** stream) {
  GpuBackend* g = gpu_of(h);
  if (!g || !stream) return BSHMEM_ERR_STATE;
  *stream = g->stream();
  return BSHMEM_OK;
}
// Waits for everything enqueued on the PE's stream and reports device-side timeouts.
int bshmem_gpu_synchronize(bshmem_handle_t h) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  if (cudaStreamSynchronize(g->stream()) != cudaSuccess) return BSHMEM_ERR_CUDA;
  return g->check_device_error("synchronize");
}
int bshmem_gpu_set_blocking(bshmem_handle_t h, int blocking) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  g->set_blocking(blocking != 0);
  return BSHMEM_OK;
}
int bshmem_gpu_set_coll_ctas(bshmem_handle_t h, int n) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  g->set_coll_ctas(n);
  return BSHMEM_OK;
}
int bshmem_gpu_set_nvls(bshmem_handle_t h, int on) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  g->refresh_mc();
  g->set_nvls(on != 0);
  return BSHMEM_OK;
}
// Copies the device-side state (peer base table etc.) for a user kernel's argument list.
int bshmem_gpu_get_state(bshmem_handle_t h, bshmem_dev_state_t* out) {
  GpuBackend* g = gpu_of(h);
  if (!g || !out) return BSHMEM_ERR_STATE;
  *out = g->state();
  return BSHMEM_OK;
}
int bshmem_gpu_check_error(bshmem_handle_t h) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  return g->check_device_error("check");
}
int bshmem_gpu_get_device_stats(bshmem_handle_t h, uint64_t* out, int n) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  unsigned long long tmp[BSHMEM_DSTAT_COUNT];
  if (cudaMemcpy(tmp, g->dstats(), sizeof(tmp), cudaMemcpyDeviceToHost) != cudaSuccess) return BSHMEM_ERR_CUDA;
  for (int i = 0; i < n && i < BSHMEM_DSTAT_COUNT; ++i) out[i] = tmp[i];
  return BSHMEM_OK;
}
// Device timeline: keep the last `capacity` events (0 switches tracing off; at most BSHMEM_TRACE_MAX_EVENTS).
// Synchronises the runtime's stream, so call it between kernels.
int bshmem_gpu_trace_enable(bshmem_handle_t h, int capacity) {
  GpuBackend* g = gpu_of(h);
  if (!g || !g->dstats()) return BSHMEM_ERR_STATE;
  if (capacity < 0 || capacity > BSHMEM_TRACE_MAX_EVENTS) return BSHMEM_ERR_INVALID;
  if (cudaStreamSynchronize(g->stream()) != cudaSuccess) return BSHMEM_ERR_CUDA;
  unsigned long long head[2] = {(unsigned long long)capacity, 0ull};
  return cudaMemcpy(g->dstats() + BSHMEM_DSTAT_COUNT, head, sizeof(head), cudaMemcpyHostToDevice) == cudaSuccess ? BSHMEM_OK
                                                                                                                  : BSHMEM_ERR_CUDA;
}
// Copies the recorded events, oldest first, into out[4 * max_events] (time ns, op | pe << 8 | block << 32, bytes,
// sequence number); *n_out = events copied, *total = events recorded since tracing was enabled.
int bshmem_gpu_trace_read(bshmem_handle_t h, uint64_t* out, int max_events, int* n_out, uint64_t* total) {
  GpuBackend* g = gpu_of(h);
  if (!g || !g->dstats() || !out || !n_out) return BSHMEM_ERR_STATE;
  if (cudaStreamSynchronize(g->stream()) != cudaSuccess) return BSHMEM_ERR_CUDA;
  std::vector<unsigned long long> buf(BSHMEM_TRACE_WORDS);
  if (cudaMemcpy(buf.data(), g->dstats() + BSHMEM_DSTAT_COUNT, sizeof(unsigned long long) * BSHMEM_TRACE_WORDS,
                 cudaMemcpyDeviceToHost) != cudaSuccess)
    return BSHMEM_ERR_CUDA;
  const unsigned long long cap = buf[0], count = buf[1];
  if (total) *total = count;
  unsigned long long have = cap ? (count < cap ? count : cap) : 0;
  if (have > (unsigned long long)max_events) have = max_events;
  for (unsigned long long k = 0; k < have; ++k) {
    const unsigned long long seq = count - have + k;
    const unsigned long long* e = &buf[2 + 4 * (seq % cap)];
    for (int w = 0; w < 4; ++w) out[4 * k + w] = e[w];
  }
  *n_out = (int)have;
  return BSHMEM_OK;
}
int bshmem_gpu_reset_device_stats(bshmem_handle_t h) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  return cudaMemset(g->dstats(), 0, sizeof(unsigned long long) * BSHMEM_DSTAT_COUNT) == cudaSuccess ? BSHMEM_OK : BSHMEM_ERR_CUDA;
}

// Device-initiated put/get of `n` bytes between `local` (any device pointer) and the symmetric
// address `sym` on `pe`, striped over `ctas` CTAs of `threads` threads at the given scope
// (0 thread, 1 warp, 2 block).  This is the path the point-to-point bandwidth sweep times.
int bshmem_gpu_rma_kernel(bshmem_handle_t h, void* sym, void* local, uint64_t n, int pe, int is_put, int scope,
                          int ctas, int threads) {
  GpuBackend* g = gpu_of(h);
  if (!g) return BSHMEM_ERR_STATE;
  uint64_t off;
  if (!h->to_offset(sym, n, &off) || pe < 0 || pe >= g->n_pes()) return BSHMEM_ERR_RANGE;
  if (ctas < 1) ctas = 1;
  if (threads < 32) threads = 32;
  if (threads > 512) threads = 512;     // the kernel's launch bound: eight 16-byte accesses in flight per thread need the registers
  // scope 3 = bulk async copies through shared memory
  const bool aligned = ((reinterpret_cast<uintptr_t>(local) | off | n) & 15) == 0;
  if (scope == 3 && !aligned) return BSHMEM_ERR_INVALID;
  cudaError_t ce;
  if (scope == 3) {
    static bool attr_set[64] = {};
    const int d = g->heap()->device;
    if (d >= 0 && d < 64 && !attr_set[d]) {
      cudaFuncSetAttribute(k_rma_bulk, cudaFuncAttributeMaxDynamicSharedMemorySize, kBulkStages * kBulkChunk);
      attr_set[d] = true;
    }
    char* remote = g->heap()->base[pe] + off;
    char* loc = static_cast<char*>(local);
    ce = launch_overlapping(k_rma_bulk, ctas, 128, kBulkStages * kBulkChunk, g->stream(), g->state(), is_put ? remote : loc,
                            is_put ? loc : remote, n, g->dstatus());
  } else {
    ce = launch_overlapping(k_rma, ctas, threads, 0, g->stream(), g->state(), pe, off, static_cast<char*>(local), n, is_put, scope);
  }
  if (ce != cudaSuccess) {
    g_err = std::string("rma kernel launch: ") + cudaGetErrorString(ce);
    return BSHMEM_ERR_CUDA;
  }
  return BSHMEM_OK;
}

// Context RMA whose local buffer the caller knows to be memory of this PE's GPU (a CUDA tensor): small messages then
// need no copy-engine request.  Otherwise the same as bshmem_ctx_putmem / getmem(_nbi) and bshmem_ctx_putmem_signal(_nbi).
namespace {
struct LocalIsDevice {
  LocalIsDevice() { tl_local_is_device = true; }
  ~LocalIsDevice() { tl_local_is_device = false; }
};
}  // namespace
int bshmem_gpu_ctx_put_dev(bshmem_handle_t h, bshmem_ctx_t c, void* dest, const void* src, size_t n, int pe, int nbi) {
  LocalIsDevice hint;
  return nbi ? bshmem_ctx_putmem_nbi(h, c, dest, src, n, pe) : bshmem_ctx_putmem(h, c, dest, src, n, pe);
}
int bshmem_gpu_ctx_get_dev(bshmem_handle_t h, bshmem_ctx_t c, void* dest, const void* src, size_t n, int pe, int nbi) {
  LocalIsDevice hint;
  return nbi ? bshmem_ctx_getmem_nbi(h, c, dest, src, n, pe) : bshmem_ctx_getmem(h, c, dest, src, n, pe);
}
int bshmem_gpu_ctx_put_signal_dev(bshmem_handle_t h, bshmem_ctx_t c, void* dest, const void* src, size_t n, uint64_t* sig, uint64_t value,
                                  int sig_op, int pe, int nbi) {
  LocalIsDevice hint;
  return nbi ? bshmem_ctx_putmem_signal_nbi(h, c, dest, src, n, sig, value, sig_op, pe)
             : bshmem_ctx_putmem_signal(h, c, dest, src, n, sig, value, sig_op, pe);
}

// One collective for a whole local group in a single launch.
// handles[n]: the group's runtimes; team_slot: the team to run on (every member passes the same
// offsets, as with any symmetric call).
int bshmem_gpu_group_collective(bshmem_handle_t* handles, int n, int team_slot, int kind, int dtype, int op, int root,
                                uint64_t dst_off, uint64_t src_off, uint64_t count, int ctas) {
  if (!handles || n < 1 || n > BSHMEM_MAX_PES) return BSHMEM_ERR_INVALID;
  State hs[BSHMEM_MAX_PES];
  DTeam ht[BSHMEM_MAX_PES];
  GpuBackend* g0 = gpu_of(handles[0]);
  if (!g0) return BSHMEM_ERR_STATE;
  for (int i = 0; i < n; ++i) {
    GpuBackend* g = gpu_of(handles[i]);
    if (!g) return BSHMEM_ERR_STATE;
    hs[i] = g->state();
    CollGroup cg;
    if (handles[i]->group_of_team(team_slot, &cg) == BSHMEM_OK) ht[i] = g->team_of(cg);
    else { memset(&ht[i], 0, sizeof(DTeam)); ht[i].my_idx = -1; }
  }
  if (ctas > BSHMEM_MAX_COLL_CTAS) ctas = BSHMEM_MAX_COLL_CTAS;     // one flag row per channel exists, no more
  for (int i = 0; i < n; ++i) {
    if (ht[i].my_idx < 0) continue;
    uint64_t sb = 0, db = 0;
    collk::extent(kind, dtype, count, ht[i].size, &sb, &db);
    if (src_off > hs[i].heap_bytes || sb > hs[i].heap_bytes - src_off || dst_off > hs[i].heap_bytes || db > hs[i].heap_bytes - dst_off)
      return BSHMEM_ERR_RANGE;
  }
  CollArgs a{};
  a.kind = kind; a.dtype = dtype; a.op = op; a.root = root; a.dst_off = dst_off; a.src_off = src_off; a.n = count;
  if (ctas < 1) ctas = 1;
  const int rc = g0->group_launch(hs, ht, n, a, ctas);
  g_err = rc == BSHMEM_OK ? std::string() : g0->last_error();
  return rc;
}


// DTeam split for a local group, done for all PEs at once on the calling thread (the slot
// agreement of bshmem_team_split_strided needs a host exchange between PEs, which a
// single-threaded group cannot run).
int bshmem_gpu_group_team_split(bshmem_handle_t* handles, int n, int parent_slot, int start, int stride, int size,
                                int* out_slots) {
  if (!handles || !out_slots || n < 1 || n > BSHMEM_MAX_PES) return BSHMEM_ERR_INVALID;
  bshmem::Team plans[BSHMEM_MAX_PES];
  bool member[BSHMEM_MAX_PES];
  uint64_t mask = ~0ull;
  for (int i = 0; i < n; ++i) {
    out_slots[i] = -1;
    member[i] = false;
    if (!handles[i]->teams->get(parent_slot) || handles[i]->teams->get(parent_slot)->my_pe < 0) continue;
    int rc = handles[i]->teams->plan_split(parent_slot, start, stride, size, &plans[i], &member[i]);
    if (rc != BSHMEM_OK) return rc;
    if (member[i]) mask &= handles[i]->teams->free_mask();
  }
  int slot = TeamTracker::pick_slot(mask);
  if (slot < 0) return BSHMEM_ERR_LIMIT;
  for (int i = 0; i < n; ++i) {
    if (!member[i]) continue;
    int rc = handles[i]->teams->commit(plans[i], slot);
    if (rc != BSHMEM_OK) return rc;
    out_slots[i] = slot;
  }
  return BSHMEM_OK;
}

}  // extern "C"
