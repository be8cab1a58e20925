"""Which collectives ask for the 128 KiB ring of the bulk moves: the host's rule, compiled as plain C++, against what the kernels
of the data-movement unit use."""
import shutil
import subprocess
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda" / "coll_kernels.h"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_ring_only_where_it_is_used(tmp_path):
    text = HEADER.read_text()
    args = text[text.index("struct CollArgs {"):text.index("};", text.index("struct CollArgs {")) + 2]
    rule = text[text.index("inline bool wants_move_ring"):]
    rule = rule[:rule.index("\n}\n") + 3]
    (tmp_path / "t.cc").write_text("#include <cstdint>\n#include <cstdio>\n#include <initializer_list>\n" + args + "\n" + rule + r"""
int main() {
  const uint64_t big = 1 << 22, min = 32 << 10;
  for (int kind = 0; kind < 9; ++kind)
    for (int staged = 0; staged < 2; ++staged)
      for (int ctas = 1; ctas <= 64; ctas *= 4)
        for (uint64_t n : {uint64_t(0), min - 16, min, 4 * min, big, big + 8, ~uint64_t(0) - 15})
          for (uint64_t off : {0, 8, 16}) {
            CollArgs a{};
            a.kind = kind; a.n = n; a.stage_seq = staged; a.dst_off = off; a.src_off = 4096;
            // kinds 5 and 6: fcollect and alltoall.  (An exchange keeps a payload word in n, a broadcast never uses the ring.)
            const bool used = (kind == 5 || kind == 6) && !staged && n % 16 == 0 && off % 16 == 0 && n / ctas >= min;
            if (wants_move_ring(a, ctas, min) != used) { printf("kind %d staged %d n %llu\n", kind, staged, (unsigned long long)n); return 1; }
          }
  puts("ok");
}
""")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-w", "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
    impl = (HEADER.parent / "coll_kernels_impl.cuh").read_text()
    assert "wants_move_ring(a, ctas, coll::kMoveMinBytes)" in impl          # what the launches ask
