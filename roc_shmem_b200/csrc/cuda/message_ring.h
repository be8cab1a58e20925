// message_ring.h — the ring through which a context's non-blocking messages reach the block, or the blocks, that serve it
// (k_ring and k_ring_wide in gpu_backend.cu): its words, and the host's side.  Plain C++ but for the annotations, so that the two
// sides' protocol also runs as host threads (tests/test_cpu_message_ring.py, tests/test_cpu_message_ring_sizes.py).
//
//  - A message is three words, two addresses of 48 bits and a size, each beside a part of its number, so that each word says by
//    itself whether it has arrived (no order of the words is relied upon).
//  - The size also carries the generation of the block that is to take the message, and no other block does.  Operations of the
//    context that are no messages go through its stream: the host tells the block to end (stop) and enqueues them behind it, and
//    a message behind them is for the next block, which stands behind them in the stream.  The old block may still be looking
//    at the ring then, and must leave that message alone.
//  - Messages between two fences of the context are unordered, as the API has it, except that one which touches what an
//    earlier one touches waits for it, as does the first behind a fence (kRingOrdered).
//  - One block takes messages of up to kRingNarrowMax bytes, several all.  A longer message that finds the one block
//    tells it to end, as an operation would, and is for the blocks behind it, which take the short ones that follow as well.
//  - A block that ends says so first (closed), then looks for messages once more; the host looks at `closed` behind each message
//    that it has written.  One of the two sees the other, and `final` says how far the block got.  A message that it left is
//    given to the next block.
#pragma once
#include <atomic>
#include <cstdint>
#include <mutex>

#include "../include/bshmem_types.h"

#ifdef __CUDACC__
#define BSHMEM_RING_FN __host__ __device__ constexpr
#else
#define BSHMEM_RING_FN constexpr
#endif

namespace bshmem {

struct alignas(32) RingSlot { uint64_t w[4]; };
constexpr unsigned kRingSlots = 256, kRingNarrowMax = 16u << 10, kRingMessageMax = 512u << 10;
constexpr uint32_t kRingOrdered = 1u << 31, kRingSizeMask = kRingOrdered - 1;
struct Ring {                          // pinned host memory
  RingSlot slot[kRingSlots];
  alignas(64) uint64_t closed;         // by the block: its generation
  alignas(64) uint64_t final;          // by the block at its end: generation << 32 | messages taken since the ring exists
  alignas(64) uint64_t consumed;       // by the block: messages done since the ring exists (32 bits)
  alignas(64) uint64_t stop;           // by the host: this generation, and those before it, are to end
  alignas(64) uint64_t failed;         // by the block, should blocks wait for one another in vain: its generation.  (In front of `stop`: a window 1.5 us longer.)
};
// What stands beside the words of message `index`: 16 bits that differ from those of the message that the slot held before; and
// the generation beside the size (a block's successor starts at its end, so 15 bits do).
BSHMEM_RING_FN uint64_t ring_tag16(uint32_t index) { return (uint64_t)((index / kRingSlots + 1) & 0xFFFF) << 48; }
BSHMEM_RING_FN uint64_t ring_for(uint32_t generation) { return (uint64_t)(generation & 0x7FFF) << 32; }
static_assert(kRingMessageMax <= kRingSizeMask, "a size and the mark share half a word");
// Whether the words are those of message `index` and the block of this generation is to take it.
BSHMEM_RING_FN bool ring_arrived(uint64_t w0, uint64_t w1, uint64_t w2, uint32_t index, uint32_t generation) {
  const uint64_t high16 = ~((1ull << 48) - 1), tag = ring_tag16(index);
  return (w0 & high16) == tag && (w1 & high16) == tag && (w2 & ~(uint64_t)(kRingOrdered | kRingSizeMask)) == (tag | ring_for(generation));
}
BSHMEM_RING_FN bool ring_stopped(uint64_t stop, uint32_t generation) { return (int32_t)((uint32_t)stop - generation) >= 0; }

// The host's side: one per context.
class RingWriter {
 public:
  Ring* ring = nullptr;

  void open(Ring* r) {
    ring = r;
    head_ = generation_ = 0;
    serving_ = wide_ = order_next_ = false;
    n_recent_ = 0;
  }
  // Before anything but a message is enqueued in the context's stream, and held until it is there: a block that another thread's
  // message launched in between would stand before the operation, and what follows would take it to stand behind (serving()).
  // Every message written so far precedes the word that tells the block to end, so the block takes them all.
  std::unique_lock<std::mutex> stop() {
    std::unique_lock<std::mutex> lock(mu_);
    if (serving_) end_block();
    return lock;
  }
  void fence() {
    std::lock_guard<std::mutex> lock(mu_);
    order_next_ = true;
  }
  // Whether the context is done once done(head) is true: a block serves, and what was enqueued before it was done when it began.
  bool serving(uint32_t* head) {
    std::lock_guard<std::mutex> lock(mu_);
    *head = head_;
    return serving_;
  }
  bool done(uint32_t head) const { return (int32_t)(consumed() - head) >= 0; }
  bool failed() const { return word(ring->failed) != 0; }

  // One message.  start(from, generation) launches what serves the ring from message `from` on, several blocks for a message of more than
  // kRingNarrowMax bytes; wait(arrived) returns when arrived() or at the end of all blocks launched so far.  Both return a status;
  // BSHMEM_ERR_STATE: the blocks have ended without it.
  template <class Start, class Wait>
  int message(uint64_t dst, uint64_t src, uint32_t n, Start start, Wait wait) {
    std::lock_guard<std::mutex> lock(mu_);
    if (head_ - consumed() >= kRingSlots) {
      const int rc = wait([&] { return head_ - consumed() < kRingSlots; });      // the block takes all, then ends
      if (rc != BSHMEM_OK) return rc;
      if (head_ - consumed() >= kRingSlots) return BSHMEM_ERR_STATE;             // nothing undelivered is written over
    }
    const uint32_t index = head_;
    const uint32_t size = n | (ordered(dst, src, n) ? kRingOrdered : 0);
    auto* w = reinterpret_cast<std::atomic<uint64_t>*>(ring->slot[index % kRingSlots].w);
    const bool wide = n > kRingNarrowMax;
    if (serving_ && wide && !wide_) end_block();
    const bool beside = serving_;                    // else a block is launched for it
    w[0].store(ring_tag16(index) | dst, std::memory_order_relaxed);
    w[1].store(ring_tag16(index) | src, std::memory_order_relaxed);
    w[2].store(ring_tag16(index) | ring_for(beside ? generation_ : generation_ + 1) | size, std::memory_order_release);
    head_ = index + 1;
    if (beside) {
      std::atomic_thread_fence(std::memory_order_seq_cst);
      if (word(ring->closed) != generation_) return BSHMEM_OK;
      // the block has decided to end: it says how far it got in a moment
      const int rc = wait([&] { return (uint32_t)(word(ring->final) >> 32) == generation_; });
      if (rc != BSHMEM_OK) return rc;
      serving_ = false;
      const uint64_t final = word(ring->final);
      if ((uint32_t)(final >> 32) != generation_) return unserved(index, BSHMEM_ERR_STATE);
      if ((uint32_t)final == head_) return BSHMEM_OK;
      w[2].store(ring_tag16(index) | ring_for(generation_ + 1) | size, std::memory_order_release);
    }
    const int rc = start(index, generation_ + 1);
    if (rc != BSHMEM_OK) return unserved(index, rc);
    ++generation_;
    serving_ = true;
    wide_ = wide;
    return BSHMEM_OK;
  }

 private:
  void end_block() {
    reinterpret_cast<std::atomic<uint64_t>&>(ring->stop).store(generation_, std::memory_order_release);
    serving_ = false;
  }
  static uint64_t word(const uint64_t& w) { return reinterpret_cast<const std::atomic<uint64_t>&>(w).load(std::memory_order_acquire); }
  uint32_t consumed() const { return (uint32_t)word(ring->consumed); }
  int unserved(uint32_t index, int rc) {             // nobody takes message `index`
    head_ = index;
    order_next_ = true;
    return rc;
  }
  // Whether the message has to wait for the ones before it; keeps the list of those that it may run beside.
  bool ordered(uint64_t dst, uint64_t src, uint32_t n) {
    auto meet = [](uint64_t a, uint32_t na, uint64_t b, uint32_t nb) { return a < b + nb && b < a + na; };
    bool after = order_next_ || n_recent_ == (int)(sizeof(recent_) / sizeof(recent_[0]));
    for (int i = 0; i < n_recent_ && !after; ++i) {
      const Span& r = recent_[i];
      after = meet(dst, n, r.dst, r.n) || meet(dst, n, r.src, r.n) || meet(src, n, r.dst, r.n);
    }
    if (after) n_recent_ = 0;
    order_next_ = false;
    recent_[n_recent_++] = {dst, src, n};
    return after;
  }

  std::mutex mu_;
  uint32_t head_ = 0, generation_ = 0;               // messages written, blocks launched
  bool serving_ = false, wide_ = false;              // the last block, several of them if wide_, may be taking messages
  bool order_next_ = false;
  struct Span { uint64_t dst, src; uint32_t n; } recent_[16];      // messages since the last ordered one
  int n_recent_ = 0;
};

}  // namespace bshmem
