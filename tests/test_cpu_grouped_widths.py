"""Grouped products with counts on the device take both accumulators per tile only where whole waves of tiles agree (csrc/cuda/pair_plan.h)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"
# (row blocks, columns, depth): width
PLANS = {(16 * 5, 1024, 2048): 256, (16 * 7, 1024, 2048): 256, (8 * 8, 2048, 4096): 256, (8 * 3, 2048, 4096): 256, (8 * 9, 2048, 4096): 512,
         (8 * 6, 2048, 8192): 512, (8 * 16, 4096, 14336): 512}


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_plan(tmp_path):
    calls = "".join(f"w = plan_width({m}, {n}, {k}, 74, 64, false, false); std::printf(\"%d \", w.cols[0] + w.cols[1]);" for m, n, k in PLANS)
    (tmp_path / "t.cc").write_text(f"#include <cstdio>\n#include \"pair_plan.h\"\nusing namespace bshmem::gemm2;\nint main() {{ Width w; {calls} }}\n")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-I", str(CUDA), "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert [int(v) for v in subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.split()] == list(PLANS.values())
