"""The protocol of served calls (csrc/cuda/call_service.h): the host's side as it is, the serving block (k_calls) as host threads that end
when they please.  Every request is carried out once and answered, or refused and not carried out."""
import shutil
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <thread>
#include <vector>
#include "call_service.h"
using namespace bshmem;

static CallSlot slot;
static std::atomic<uint64_t> answer{0};
static std::vector<std::atomic<int>> times(1 << 20);
static auto& word(uint64_t& w) { return reinterpret_cast<std::atomic<uint64_t>&>(w); }

static void block(uint32_t seq, uint32_t generation, int looks) {      // k_calls: ends after `looks` looks without a request
  while (true) {
    uint32_t req[kCallWords];
    bool here = false;
    for (int i = 0; i < looks && !here; ++i) {
      here = true;
      for (unsigned k = 0; k < kCallWords; ++k) {
        const uint64_t v = word(slot.w[k]).load(std::memory_order_relaxed);
        req[k] = (uint32_t)v;
        here = here && (uint32_t)(v >> 32) == seq;
      }
      if (!here) std::this_thread::yield();
    }
    if (!here) break;
    ++times[req[CALL_VALUE]];
    answer.store((uint64_t)req[CALL_TOKEN] << 32 | (req[CALL_VALUE] ^ req[CALL_HEAD]), std::memory_order_release);
    ++seq;
  }
  word(slot.final).store((uint64_t)generation << 32 | (seq - 1), std::memory_order_release);
}

int main(int, char** a) {
  const int n = atoi(a[1]), looks = atoi(a[2]), refuse = atoi(a[3]);
  std::vector<std::thread> blocks;
  CallWriter w;
  w.slot = &slot;
  std::mt19937 rng(looks);
  int wrong = 0, refused = 0;
  for (int i = 0; i < n; ++i) {
    Call call(CALL_AMO, 1, 2, 8);
    call.set(CALL_VALUE, (uint64_t)i).set(CALL_TOKEN, (uint64_t)i + 1);
    const bool done = w.run(call,
        [&](uint32_t first, uint32_t generation) {
          if (refuse && (int)(rng() % refuse) == 0) return (int)BSHMEM_ERR_CUDA;
          blocks.emplace_back(block, first, generation, 1 + (int)(rng() % looks));
          return (int)BSHMEM_OK;
        },
        [&] { return (answer.load(std::memory_order_acquire) >> 32) == (uint64_t)i + 1; },
        [&] { for (auto& t : blocks) if (t.joinable()) t.join(); return (int)BSHMEM_OK; });
    if (done) wrong += times[i] != 1 || (uint32_t)answer.load() != ((uint32_t)i ^ call.w[CALL_HEAD]);
    else { ++refused; wrong += times[i] != 0; }
    if (rng() % 8 == 0) for (unsigned k = rng() % 400; k; --k) std::this_thread::yield();
  }
  for (auto& t : blocks) if (t.joinable()) t.join();
  for (int i = 0; i < n; ++i) wrong += times[i] > 1;
  printf("wrong %d refused %s\n", wrong, refused ? "some" : "none");
  return 0;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs a C++ compiler")
    d = tmp_path_factory.mktemp("calls")
    (d / "model.cc").write_text(MODEL)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CUDA), "-o", str(d / "model"), str(d / "model.cc"), "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return lambda *a: subprocess.run([str(d / "model")] + [str(x) for x in a], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("calls,looks,refuse,expect", [(3000, 300, 0, "none"), (3000, 20000, 0, "none"), (2000, 200, 3, "some")])
def test_every_call_once(model, calls, looks, refuse, expect):
    r = model(calls, looks, refuse)
    assert r.returncode == 0 and r.stdout == f"wrong 0 refused {expect}\n", r.stdout + r.stderr


# ---- a block that is launched ahead, on a device that may have no place for it ----
AHEAD = MODEL[:MODEL.index("int main(")].replace("static void block(uint32_t seq", """static std::atomic<bool> place{true};
static std::atomic<int> blocks_there{0};
static void block_body(uint32_t, uint32_t, int);
static void block(uint32_t seq, uint32_t generation, int looks) {
  while (!place.load()) std::this_thread::yield();
  ++blocks_there;
  word(slot.begun).store(generation, std::memory_order_relaxed);
  block_body(seq, generation, looks);
}
static void block_body(uint32_t seq""") + r"""
int main(int, char** a) {
  const int n = atoi(a[1]), looks = atoi(a[2]), full = atoi(a[3]);     // full: calls in a row without a place for a block
  std::vector<std::thread> blocks;
  CallWriter w;
  w.slot = &slot;
  std::mt19937 rng(looks);
  int wrong = 0, served = 0, waited = 0;
  for (int i = 0; i < n; ++i) {
    if (full) place = i / full % 2 == 0;
    Call call(CALL_AMO, 1, 2, 8);
    call.set(CALL_VALUE, (uint64_t)i).set(CALL_TOKEN, (uint64_t)i + 1);
    bool done = false;
    if (w.ready()) {
      done = w.run(call, [](uint32_t, uint32_t) { return (int)BSHMEM_ERR_STATE; },
                   [&] { return (answer.load(std::memory_order_acquire) >> 32) == (uint64_t)i + 1; },
                   [&] { waited += blocks_there.load() < (int)blocks.size(); std::this_thread::yield(); return (int)BSHMEM_OK; });
      if (done) wrong += times[i] != 1 || (uint32_t)answer.load() != ((uint32_t)i ^ call.w[CALL_HEAD]);
    }
    if (done) ++served;
    else {
      wrong += times[i]++ != 0;                                          // by a launch
      w.prepare([&](uint32_t first, uint32_t generation) {
        blocks.emplace_back(block, first, generation, 1 + (int)(rng() % looks));
        return (int)BSHMEM_OK;
      });
      for (unsigned k = rng() % 50; k; --k) std::this_thread::yield();
    }
  }
  place = true;
  for (auto& t : blocks) if (t.joinable()) t.join();
  for (int i = 0; i < n; ++i) wrong += times[i] != 1;
  printf("wrong %d waited %d served %s\n", wrong, waited, served ? "some" : "none");
  return 0;
}
"""


@pytest.mark.parametrize("calls,looks,full", [(3000, 3000, 0), (3000, 3000, 100), (500, 20000, 500)])
def test_no_call_waits_for_a_block_to_begin(tmp_path, calls, looks, full):
    """Each call once, by the block or by a launch, also while a block that was launched has no place to run."""
    if shutil.which("g++") is None:
        pytest.skip("needs a C++ compiler")
    (tmp_path / "ahead.cc").write_text(AHEAD)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CUDA), "-o", str(tmp_path / "ahead"), str(tmp_path / "ahead.cc"), "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(tmp_path / "ahead")] + [str(x) for x in (calls, looks, full)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "wrong 0 waited 0 served some\n", r.stdout + r.stderr


# ---- when a call asks ----
POLICY = r"""
#include <cstdio>
#include <cstdlib>
#include "call_service.h"
using namespace bshmem;
int main(int, char** a) {
  // `calls` calls `gap` ns apart, a kernel before every `every`-th of them (0: none), a block for every series that ends after `taken` requests
  const int calls = atoi(a[1]), gap = atoi(a[2]), every = atoi(a[3]), taken = atoi(a[4]);
  CallSeries s;
  int asked = 0, refused = 0, blocks = 0, left = 0;
  for (int i = 0; i < calls; ++i) {
    if (!s.long_enough((long long)i * gap + 1000000)) continue;
    ++asked;
    if (every && i % every == 0) { s.refused(); ++refused; continue; }
    if (left == 0) { ++blocks; left = taken; }
    else if (--left == 0) s.ended((unsigned)taken);
  }
  AskAhead w;
  int useless = 0;
  for (int i = 0; i < calls; ++i)
    if (w.now()) { ++useless; w.told(false); }
  w.told(true);
  printf("%d %d %d %d %d\n", asked, refused, blocks, useless, (int)w.now());
  return 0;
}
"""


@pytest.mark.parametrize("calls,gap,every,taken,most_asked,most_refused,most_blocks", [
    (10000, 20000, 0, 90, 0, 0, 0),             # no series
    (10000, 8000, 0, 90, 10000, 0, 120),        # a loop of calls: a block for every 90 of them
    (10000, 8000, 1, 90, 180, 180, 0),          # a kernel before each: asked every 65th time
    (10000, 8000, 0, 3, 700, 0, 170),           # blocks that end after 3: one for some 65 calls
])
def test_a_program_that_has_no_use_for_blocks_does_not_pay_for_them(tmp_path, calls, gap, every, taken, most_asked, most_refused, most_blocks):
    if shutil.which("g++") is None:
        pytest.skip("needs a C++ compiler")
    (tmp_path / "policy.cc").write_text(POLICY)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CUDA), "-o", str(tmp_path / "policy"), str(tmp_path / "policy.cc")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([str(tmp_path / "policy")] + [str(x) for x in (calls, gap, every, taken)], capture_output=True, text=True, timeout=60).stdout
    asked, refused, blocks, useless, again = map(int, out.split())
    assert asked <= most_asked and refused <= most_refused and blocks <= most_blocks, out
    assert most_blocks != 120 or (asked > 9900 and blocks > 100), out
    assert useless <= calls // 60 and again == 1, out
