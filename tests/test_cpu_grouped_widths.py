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
def test_a_device_without_pairs(tmp_path):
    """A plan for no pair at all is a plan, not a division by zero."""
    (tmp_path / "t.cc").write_text("#include <cstdio>\n#include <cstdlib>\n#include \"pair_plan.h\"\nusing namespace bshmem::gemm2;\n"
                                   "int main(int, char** a) { int p = atoi(a[1]); Width x = plan_width(4, 1024, 1024, p, 32, false), y = plan_width(4, 1024, 1024, p, 64, "
                                   "false, false); std::printf(\"%d %d\", x.cols[0] > 0, y.cols[0] > 0); }\n")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-I", str(CUDA), "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    for pairs in ("0", "-1", "1"):
        r = subprocess.run([str(exe), pairs], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0 and r.stdout == "1 1"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_plan(tmp_path):
    calls = "".join(f"w = plan_width({m}, {n}, {k}, 74, 64, false, false); std::printf(\"%d \", w.cols[0] + w.cols[1]);" for m, n, k in PLANS)
    (tmp_path / "t.cc").write_text(f"#include <cstdio>\n#include \"pair_plan.h\"\nusing namespace bshmem::gemm2;\nint main() {{ Width w; {calls} }}\n")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-I", str(CUDA), "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert [int(v) for v in subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.split()] == list(PLANS.values())
