// call_service.h — the slot through which blocking calls of the default context reach the block that serves them while they follow one
// another closely (k_calls in gpu_backend.cu): its words, and the host's side.  Plain C++.
//
//  - There is one request at a time.  Each of its words carries 32 bits beside the request's number, so that it says by itself whether
//    it has arrived.
//  - A block serves request after request, from the one it was launched for on, and ends after a while without one or at the end of its
//    life.  Its last word, `final`, says up to which request it got: all of them have been answered, none behind them will be.
//  - The host waits for the answer or for that word.  A request that the block left is given to the next block.
#pragma once
#include <atomic>
#include <cstdint>
#include <initializer_list>

#include "../include/bshmem_types.h"

namespace bshmem {

enum CallKind : uint32_t { CALL_AMO = 1, CALL_READ, CALL_TEST, CALL_PUT_SIGNAL };
// what the words hold: kind | dtype << 8 | operator << 16 | size << 24, then pairs of halves
enum CallWord { CALL_HEAD = 0, CALL_ADDR = 1, CALL_VALUE = 3, CALL_OTHER = 5, CALL_BYTES = 7, CALL_SIG = 8, CALL_DONE = 10, CALL_TOKEN = 12 };
constexpr unsigned kCallWords = 14;

struct Call {
  uint32_t w[kCallWords] = {};
  Call(CallKind kind, int dtype, int op, int size) { w[CALL_HEAD] = kind | (uint32_t)dtype << 8 | (uint32_t)op << 16 | (uint32_t)size << 24; }
  Call& set(CallWord at, uint64_t v) {
    w[at] = (uint32_t)v;
    w[at + 1] = (uint32_t)(v >> 32);
    return *this;
  }
};
struct CallSlot {                      // pinned host memory
  alignas(128) uint64_t w[16];
  alignas(128) uint64_t final;         // by the block at its end: generation << 32 | the last request it answered
};

class CallWriter {
 public:
  CallSlot* slot = nullptr;

  // One request; the caller holds the lock that makes it the only one.  start(first, generation) launches a block that serves from request
  // `first` on, answered() looks at the caller's words, wait() returns when all blocks launched so far have ended; both return a
  // status.  True: answered.  False: no block has taken the request, and none will.
  template <class Start, class Answered, class Wait>
  bool run(const Call& call, Start start, Answered answered, Wait wait) {
    const uint32_t seq = ++seq_;
    for (unsigned i = 0; i < kCallWords; ++i)
      reinterpret_cast<std::atomic<uint64_t>&>(slot->w[i]).store((uint64_t)seq << 32 | call.w[i], std::memory_order_release);
    const auto& final = reinterpret_cast<const std::atomic<uint64_t>&>(slot->final);
    for (int attempt = 0; attempt < 2; ++attempt) {
      if (!serving_) {
        if (start(seq, generation_ + 1) != BSHMEM_OK) return false;
        ++generation_;
        serving_ = true;
      }
      for (unsigned it = 0;; ++it) {
        if (answered()) return true;
        const uint64_t f = final.load(std::memory_order_acquire);
        if ((uint32_t)(f >> 32) == generation_) {
          serving_ = false;
          if ((int32_t)((uint32_t)f - seq) >= 0) return answered();       // the answer precedes this word
          break;
        }
        if (it == 4000) {
          if (wait() != BSHMEM_OK) return false;
          it = 0;
        }
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
      }
    }
    return false;
  }

 private:
  uint32_t seq_ = 0, generation_ = 0;                // requests written, blocks launched
  bool serving_ = false;                             // the last block may be taking requests
};

}  // namespace bshmem
