"""A launch whose preferred form the device refuses runs in its general form (csrc/cuda/launch_choice.h)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_a_refused_form_falls_back(tmp_path):
    (tmp_path / "t.cc").write_text("""#include <cstdio>
#include "launch_choice.h"
int main() {
  // fits, what the preferred and the general form answer: the call's answer, and how often each was launched
  const int cases[][3] = {{1, 0, 0}, {1, 7, 0}, {1, 7, 9}, {0, 0, 0}, {0, 0, 9}};
  for (auto& c : cases) {
    int first = 0, second = 0;
    const int rc = bshmem::launch_preferred(c[0] != 0, 0, [&] { ++first; return c[1]; }, [&] { ++second; return c[2]; });
    std::printf("%d%d%d ", rc, first, second);
  }
}
""")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-I", str(CUDA), "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.split() == ["010", "011", "911", "001", "901"]
