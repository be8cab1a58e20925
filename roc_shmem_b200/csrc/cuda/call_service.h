// call_service.h — the slot through which blocking calls of the default context reach the block that serves them while they follow one
// another closely (k_calls in gpu_backend.cu): its words, and the host's side.  Plain C++.
//
//  - There is one request at a time.  Each of its words carries 32 bits beside the request's number, so that it says by itself whether
//    it has arrived.
//  - A block serves request after request, from the one it was launched for on, and ends after a while without one or at the end of its
//    life.  Its last word, `final`, says up to which request it got: all of them have been answered, none behind them will be.
//  - The host waits for the answer or for that word.  A request that the block left is given to the next block.
//  - A block may be launched ahead of its first request (prepare) and is asked once it says that it is there (ready), so that no
//    request waits for a place on the device: beside a kernel that leaves none, and that may itself wait for the call, the host launches
//    what needs less of one.
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
  alignas(128) uint64_t begun;         // by the block at its start: its generation
  alignas(128) uint64_t final;         // by the block at its end: generation << 32 | the last request it answered
};

// Which calls are worth the question whether their stream is idle, and a block: those that follow some others closely.  How many others is
// what the program's calls have been like: a refusal (the stream holds something) and a block that ended after a few requests make it
// more, a block that was worth its launch brings it back.  So a program that mostly enqueues work between its calls, or synchronises
// behind a few of them, asks once in a while and otherwise calls as if there were no blocks.
class CallSeries {
 public:
  static constexpr long long kCloseNs = 15000;       // from one call to the next (a launch and its answer take 8 of that)
  static constexpr unsigned kFew = 4, kMany = 64, kWorth = 16;
  bool long_enough(long long now_ns) {               // a call; whether it is to be asked for
    close_ = now_ns - last_ < kCloseNs ? close_ + 1 : 0;
    last_ = now_ns;
    return long_enough();
  }
  bool long_enough() const { return close_ >= needed_; }
  void refused() {
    needed_ = 2 * needed_ < kMany ? 2 * needed_ : kMany;
    close_ = 0;
  }
  void ended(unsigned taken) {                       // a block, after so many requests
    if (taken >= kWorth) needed_ = kFew;
    else refused();
  }

 private:
  long long last_ = -kCloseNs;
  unsigned close_ = 0, needed_ = kFew;
};
// The same for what a call asks ahead of its own launch: not again for a while after an answer that it had no use for.
class AskAhead {
 public:
  bool now() {
    if (skip_ == 0) return true;
    --skip_;
    return false;
  }
  void told(bool useful) {
    missed_ = useful ? 0 : 2 * missed_ + 1 < 63 ? 2 * missed_ + 1 : 63;
    skip_ = missed_;
  }

 private:
  unsigned skip_ = 0, missed_ = 0;
};

class CallWriter {
 public:
  CallSlot* slot = nullptr;

  // All of it under the lock that makes the caller the only one.
  // Launches a block for the requests to come, unless one may be taking them.
  template <class Start>
  bool prepare(Start start) {
    if (serving_) return true;
    if (start(seq_ + 1, generation_ + 1) != BSHMEM_OK) return false;
    launched();
    return true;
  }
  bool serving() const { return serving_; }
  // Whether the block is there and has not ended yet, as far as the host can see.
  bool ready() {
    if (serving_ && ended()) serving_ = false;
    return serving_ && word(slot->begun) == generation_;
  }
  unsigned taken() const { return taken_; }          // requests that the last block has answered

  // One request; the caller holds the lock that makes it the only one.  start(first, generation) launches a block that serves from request
  // `first` on, answered() looks at the caller's words, wait() returns when all blocks launched so far have ended; both return a
  // status.  True: answered.  False: no block has taken the request, and none will.
  template <class Start, class Answered, class Wait>
  bool run(const Call& call, Start start, Answered answered, Wait wait) {
    const uint32_t seq = ++seq_;
    for (unsigned i = 0; i < kCallWords; ++i)
      reinterpret_cast<std::atomic<uint64_t>&>(slot->w[i]).store((uint64_t)seq << 32 | call.w[i], std::memory_order_release);
    for (int attempt = 0; attempt < 2; ++attempt) {
      if (!serving_) {
        if (start(seq, generation_ + 1) != BSHMEM_OK) return false;
        launched();
      }
      for (unsigned it = 0;; ++it) {
        if (answered()) {
          ++taken_;
          return true;
        }
        if (ended()) {
          serving_ = false;
          if ((int32_t)((uint32_t)word(slot->final) - seq) < 0) break;
          ++taken_;
          return answered();                         // the answer precedes the last word
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
  static uint64_t word(const uint64_t& w) { return reinterpret_cast<const std::atomic<uint64_t>&>(w).load(std::memory_order_acquire); }
  bool ended() const { return (uint32_t)(word(slot->final) >> 32) == generation_; }
  void launched() {
    ++generation_;
    serving_ = true;
    taken_ = 0;
  }
  uint32_t seq_ = 0, generation_ = 0;                // requests written, blocks launched
  unsigned taken_ = 0;
  bool serving_ = false;                             // the last block may be taking requests
};

}  // namespace bshmem
