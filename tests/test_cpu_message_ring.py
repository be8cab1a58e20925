"""The protocol of a context's message ring (csrc/cuda/message_ring.h): the host's side as it is, the serving block (k_ring) as a host
thread that makes the same looks at the same words, the stream as a queue of work.  Every message is carried out once, behind
everything that was enqueued before it, and before a quiet returns."""
import shutil
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"

MODEL = r"""
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <thread>
#include <vector>
#include "message_ring.h"
using namespace bshmem;

static double us() { return std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now().time_since_epoch()).count(); }
static void spin(double t) { for (const double t0 = us(); us() - t0 < t;) std::this_thread::yield(); }

struct Stream {                          // work in order, on a thread of its own
  std::deque<std::function<void()>> q;
  std::mutex m;
  std::condition_variable cv;
  bool busy = false, stop = false;
  std::thread t{[this] {
    std::unique_lock<std::mutex> l(m);
    while (true) {
      cv.wait(l, [&] { return stop || !q.empty(); });
      if (q.empty()) return;
      auto f = std::move(q.front());
      q.pop_front();
      busy = true;
      l.unlock();
      f();
      l.lock();
      busy = false;
      cv.notify_all();
    }
  }};
  void enqueue(std::function<void()> f) { std::lock_guard<std::mutex> l(m); q.push_back(std::move(f)); cv.notify_all(); }
  void sync() { std::unique_lock<std::mutex> l(m); cv.wait(l, [&] { return q.empty() && !busy; }); }
  ~Stream() { { std::lock_guard<std::mutex> l(m); stop = true; cv.notify_all(); } t.join(); }
};

static auto& word(uint64_t& w) { return reinterpret_cast<std::atomic<uint64_t>&>(w); }
constexpr uint32_t kMessages = 1u << 20;
struct Done { std::atomic<int> times{0}; std::atomic<uint32_t> batch{0}; };
static std::vector<Done> done(kMessages);                              // by message: its address is its number
static std::vector<std::atomic<uint32_t>> need(kMessages);             // operations of the stream enqueued before it
static std::atomic<uint32_t> operations{0}, batches{0};
static std::atomic<int> early{0};

static void block(Ring* r, uint32_t next, uint32_t generation) {       // k_ring
  const double begun = us();
  double last = begun;
  bool closing = false;
  while (true) {
    uint64_t v[16][3];
    int count = 0;
    for (int i = 0; i < 16; ++i)
      for (int k = 0; k < 3; ++k) v[i][k] = word(r->slot[(next + i) % kRingSlots].w[k]).load(std::memory_order_relaxed);
    const uint64_t stop = word(r->stop).load(std::memory_order_relaxed);
    spin(1);
    while (count < 16 && ring_arrived(v[count][0], v[count][1], v[count][2], next + count, generation) &&
           !(count && (v[count][2] & kRingOrdered))) ++count;
    std::atomic_thread_fence(std::memory_order_acq_rel);
    const double now = us();
    if (count) last = now;
    const int over = closing ? (count ? 0 : 2) : ring_stopped(stop, generation) || now - begun > 100 || now - last > 5 ? 1 : 0;
    if (count) {
      const uint32_t b = ++batches;
      for (int i = 0; i < count; ++i) {
        const uint64_t id = v[i][0] & ((1ull << 48) - 1);
        if (operations.load() < need[id].load()) ++early;
        done[id].batch = b;
        ++done[id].times;
      }
      next += count;
      word(r->consumed).store(next, std::memory_order_release);
    }
    if (over == 2) break;
    if (over == 1) {
      closing = true;
      word(r->closed).store(generation, std::memory_order_relaxed);
      std::atomic_thread_fence(std::memory_order_seq_cst);
    }
  }
  word(r->final).store((uint64_t)generation << 32 | next, std::memory_order_release);
}

struct Context {
  Stream stream;
  Ring ring;
  RingWriter writer;
  Context() { memset(&ring, 0, sizeof(ring)); writer.open(&ring); }
  int message(uint32_t id) {
    return writer.message((uint64_t)id, (uint64_t)id + (1ull << 40), 1,
                          [&](uint32_t from, uint32_t g) { spin(2); stream.enqueue([=, this] { block(&ring, from, g); }); return 0; },
                          [&](auto arrived) {
                            for (int i = 0; i < 2000; ++i) { if (arrived()) return 0; std::this_thread::yield(); }
                            stream.sync();
                            return 0;
                          });
  }
  void operation(double t, std::atomic<int>* over = nullptr) {
    const auto held = writer.stop();
    spin(3);
    stream.enqueue([t, over] { spin(t); ++operations; if (over) *over = 1; });
  }
  void quiet() {
    uint32_t head;
    if (writer.serving(&head))
      for (int i = 0; i < 2000; ++i) { if (writer.done(head)) return; std::this_thread::yield(); }
    (void)writer.stop();
    stream.sync();
  }
};

// windows of messages before and behind an operation that the caller does not wait for
static int windows(int before, int behind, double length, int rounds) {
  Context c;
  uint32_t id = 0, enqueued = 0;
  int left = 0, unordered = 0;
  for (int r = 0; r < rounds; ++r) {
    for (int i = 0; i < before; ++i) { need[id] = enqueued; if (c.message(id++)) return 1; }
    c.operation(length);
    ++enqueued;
    c.writer.fence();
    const uint32_t at = id;
    for (int i = 0; i < behind; ++i) { need[id] = enqueued; if (c.message(id++)) return 1; }
    c.quiet();
    if (operations.load() != enqueued) ++left;
    for (uint32_t k = at - before; k < id; ++k) left += done[k].times != 1;
    for (uint32_t k = at - before; k < at; ++k) unordered += done[k].batch >= done[at].batch;
  }
  c.quiet();
  c.stream.sync();
  int repeated = 0;
  for (uint32_t k = 0; k < id; ++k) repeated += done[k].times != 1;
  printf("early %d left %d unordered %d repeated %d\n", early.load(), left, unordered, repeated);
  return 0;
}

// One thread's operations and quiets beside another thread's messages in the same context.
static int shared(int rounds) {
  Context c;
  std::atomic<bool> end{false};
  std::thread other([&] { for (uint32_t id = 0; !end && id < kMessages; ++id) { c.message(id); spin(3); } });
  int left = 0;
  for (int r = 0; r < rounds; ++r) {
    std::atomic<int> over{0};
    c.operation(30, &over);
    c.quiet();
    if (!over) { ++left; c.stream.sync(); }
  }
  end = true;
  other.join();
  c.stream.sync();
  printf("left %d\n", left);
  return 0;
}

// Nobody takes the messages: an error once the slots are full, and none of them is written over.
static int full() {
  Ring ring;
  memset(&ring, 0, sizeof(ring));
  RingWriter w;
  w.open(&ring);
  int launched = 0, rc = 0;
  uint32_t sent = 0;
  auto message = [&] { return w.message(sent, 1ull << 40, 1, [&](uint32_t, uint32_t) { return ++launched, 0; }, [](auto) { return 0; }); };
  while (sent < 2 * kRingSlots && !(rc = message())) ++sent;
  Ring before = ring;
  const int again = message();
  printf("%u %d %d %d %d\n", sent, launched, rc == BSHMEM_ERR_STATE, again == rc, memcmp(&before, &ring, sizeof(ring)));
  // the block ended without a word of how far it got
  ring.closed = 1;
  ring.consumed = sent;
  const int lost = message();
  printf("%d\n", lost == BSHMEM_ERR_STATE);
  return 0;
}

int main(int n, char** a) {
  if (n == 1) return full();
  if (n == 2) return shared(atoi(a[1]));
  return windows(atoi(a[1]), atoi(a[2]), atof(a[3]), atoi(a[4]));
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs a C++ compiler")
    d = tmp_path_factory.mktemp("ring")
    (d / "model.cc").write_text(MODEL)
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-I", str(CUDA), "-o", str(d / "model"), str(d / "model.cc"), "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return lambda *a: subprocess.run([str(d / "model")] + [str(x) for x in a], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("before,behind,length,rounds", [(1, 1, 20, 2000), (3, 40, 50, 500), (64, 400, 300, 150), (0, 700, 100, 80)])
def test_messages_around_an_operation(model, before, behind, length, rounds):
    r = model(before, behind, length, rounds)
    assert r.returncode == 0 and r.stdout == "early 0 left 0 unordered 0 repeated 0\n", r.stdout + r.stderr


def test_two_threads_on_a_context(model):
    """A quiet covers its own thread's operation, also where another thread's message launched a block meanwhile."""
    r = model(2000)
    assert r.returncode == 0 and r.stdout == "left 0\n", r.stdout + r.stderr


def test_a_ring_that_nobody_empties(model):
    r = model()
    assert r.returncode == 0 and r.stdout == "256 1 1 1 0\n1\n", r.stdout + r.stderr
