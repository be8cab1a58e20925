"""How several blocks share a batch of messages (k_ring_wide in csrc/cuda/gpu_backend.cu), with host threads in the place of blocks: the first to come
hands the batches out, the others take part from when they have come, and any number of them may come late or when all is over.  Every piece once,
no batch before the last one is done, and an end for all; and by the source, that nothing in the kernel asks for blocks that run together."""
import shutil
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"

MODEL = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <thread>
#include <vector>
static std::atomic<unsigned long long> batch_word{0};
static std::atomic<unsigned> came{0}, done{0}, left_{0};
static int shared_count;                                   // the batch: so many pieces
static std::vector<std::atomic<int>> times(1 << 16);       // of a piece of the batch
static std::atomic<int> wrong{0}, helped{0};
static const unsigned long long kOver = ~0ull;

static void copy_part(int count, unsigned me, unsigned blocks) {
  for (int p = (int)me; p < count; p += (int)blocks) ++times[p];
}
static void block(int batches, int grid, unsigned seed) {
  std::mt19937 rng(seed);
  const unsigned me = came.fetch_add(1);
  if (me == 0) {
    unsigned parts = 0, number = 0;
    for (int b = 0; b < batches; ++b) {
      for (unsigned k = rng() % 20; k; --k) std::this_thread::yield();     // looks
      const int count = 1 + (int)(rng() % 300);
      unsigned here = 1;
      if (count > 8) {
        shared_count = count;
        here = came.load(std::memory_order_relaxed);
        if (here > 1) batch_word.store((unsigned long long)++number << 32 | here, std::memory_order_release);
      }
      copy_part(count, 0, here);
      parts += here - 1;
      helped += here > 1;
      while (here > 1 && done.load(std::memory_order_acquire) != parts) std::this_thread::yield();
      for (int p = 0; p < (1 << 10); ++p) wrong += times[p].exchange(0) != (p < count);
    }
    batch_word.store(kOver, std::memory_order_release);
  } else {
    unsigned seen = 0;
    while (true) {
      unsigned long long v = 0;
      do {
        v = batch_word.load(std::memory_order_acquire);
        if (v != kOver && me >= (unsigned)v) seen = (unsigned)(v >> 32);
        if ((unsigned)(v >> 32) == seen) std::this_thread::yield();
      } while ((unsigned)(v >> 32) == seen);
      seen = (unsigned)(v >> 32);
      if (v == kOver) break;
      copy_part(shared_count, me, (unsigned)v);
      done.fetch_add(1, std::memory_order_release);
    }
  }
  if (left_.fetch_add(1) == (unsigned)grid - 1) {
    batch_word = 0;
    came = done = left_ = 0;
  }
}
int main(int, char** a) {
  const int grid = atoi(a[1]), batches = atoi(a[2]), late = atoi(a[3]), launches = atoi(a[4]);      // late: blocks that find a place at the end only
  for (int l = 0; l < launches; ++l) {
    std::vector<std::thread> t;
    for (int i = 0; i < grid - late; ++i) t.emplace_back(block, batches, grid, l * 100 + i);
    std::atomic<bool> over{false};
    if (late == grid - 1) for (auto& x : t) x.join();
    for (int i = grid - late; i < grid; ++i) t.emplace_back(block, batches, grid, l * 100 + i);
    for (auto& x : t) if (x.joinable()) x.join();
    wrong += batch_word.load() != 0 || came.load() != 0 || done.load() != 0;
  }
  printf("wrong %d helped %s\n", wrong.load(), helped ? "some" : "none");
  return 0;
}
"""


@pytest.mark.parametrize("grid,batches,late,launches,helped", [(4, 50, 0, 20, "some"), (8, 100, 3, 10, "some"), (8, 100, 7, 20, "none")])
def test_blocks_that_come_when_they_please(tmp_path, grid, batches, late, launches, helped):
    if shutil.which("g++") is None:
        pytest.skip("needs a C++ compiler")
    (tmp_path / "share.cc").write_text(MODEL)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-o", str(tmp_path / "share"), str(tmp_path / "share.cc"), "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(tmp_path / "share")] + [str(x) for x in (grid, batches, late, launches)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == f"wrong 0 helped {helped}\n", r.stdout + r.stderr


def test_no_block_of_a_message_kernel_needs_another():
    text = (CUDA / "gpu_backend.cu").read_text()
    assert "barrier.cluster" not in text and "cudaLaunchAttributeClusterDimension" not in text and "cudaLaunchAttributeCooperative" not in text
