"""The few-token GEMM prefetches weights only where that is known to pay (csrc/cuda/prefetch_plan.h)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"
# (tokens, weight row in elements, blocks per CTA): blocks
PLANS = {(1, 512, 8): 4, (16, 4096, 8): 4, (128, 3584, 28): 4, (129, 3584, 28): 0, (200, 2048, 8): 0, (16, 4104, 8): 0, (50, 8200, 16): 0,
         (8, 1504, 6): 4, (8, 1504, 7): 4, (8, 1504, 8): 0, (8, 64, 1): 4,
         (64, 3584, 14): 7, (65, 3584, 14): 4, (64, 3584, 9): 4}


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_plan(tmp_path):
    calls = "".join(f"std::printf(\"%d \", bshmem::skinny::prefetch_blocks({m}, 2ll * {k}, {n}));" for m, k, n in PLANS)
    (tmp_path / "t.cc").write_text(f"#include <cstdio>\n#include \"prefetch_plan.h\"\nint main() {{ {calls} }}\n")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-I", str(CUDA), "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert [int(v) for v in subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.split()] == list(PLANS.values())
