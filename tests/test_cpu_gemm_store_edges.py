"""The direct stores of the split GEMM forms, on the CPU: the two device functions that write a result's columns are compiled as
plain C++ and run over every N around a store's width; they must write all columns below N and none at or behind it."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"


def _function(text: str, start: str) -> str:
    """The function whose signature begins with `start`, braces included."""
    i = text.index(start)
    j = text.index("{", text.index(")", i))
    depth, k = 1, j + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        k += 1
    return text[i:k]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_split_forms_stay_inside_their_columns(tmp_path):
    pair = _function((CUDA / "gemm_bf16.cu").read_text(), "__device__ static __forceinline__ void store_row16")
    few = _function((CUDA / "gemm_skinny.cuh").read_text(), "__device__ __forceinline__ void add_partials")
    few = re.sub(r"asm volatile.*?;", "", few)
    (tmp_path / "t.cc").write_text(r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <vector>
using std::min;
#define __device__
#define __forceinline__ inline
struct float4 { float x, y, z, w; };
struct uint2 { uint32_t a, b; };
struct uint4 { uint32_t a, b, c, d; };
static uint2 make_uint2(uint32_t a, uint32_t b) { return {a, b}; }
static uint4 make_uint4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) { return {a, b, c, d}; }
typedef uint16_t __nv_bfloat16;                      // every value is 1: the test looks at where, not at what
static uint32_t pack_bf16(float, float) { return 0x00010001u; }
static __nv_bfloat16 __float2bfloat16_rn(float) { return 1; }
struct Core { int M, N; };
struct Params { Core core; __nv_bfloat16* out; long long ldc, ldo; int M, N; };
constexpr int ROWS = 128, NUM_THREADS = 192;
static uint32_t mapa(uint32_t a, uint32_t) { return a; }
static float4 ld_cluster_f4(uint32_t) { return {1, 1, 1, 1}; }
""" + pair.replace("static __forceinline__", "static") + "\ntemplate <int S>\n" + few + r"""
int main() {
  for (int N = 1; N <= 280; ++N) {
    const int ld = (N + 7) / 8 * 8 + 8, M = 3;
    for (int form = 0; form < 2; ++form) {
      std::vector<uint16_t> buf((M + 1) * ld + 512, 0);
      Params p{{M, N}, buf.data(), ld, ld, M, N};
      if (form == 0) {
        float4 v[4] = {};
        for (int row = 0; row < 4; ++row)
          for (int col = 0; col < (N + 255) / 256 * 256; col += 16) store_row16(p, row, col, v);
      } else {
        for (int n0 = 0; n0 < N; n0 += ROWS)
          for (int rank = 0; rank < 2; ++rank)
            for (int warp = 0; warp < 6; ++warp)
              for (int lane = 0; lane < 32; ++lane)
                if (n0 + lane * 4 < N) add_partials<2>(p, 0, rank, warp, lane, n0);
      }
      for (size_t i = 0; i < buf.size(); ++i) {
        const bool mine = i < (size_t)M * ld && (int)(i % ld) < N;
        if ((buf[i] != 0) != mine) { printf("form %d N %d: element %zu\n", form, N, i); return 1; }
      }
    }
  }
  puts("ok");
}
""")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
