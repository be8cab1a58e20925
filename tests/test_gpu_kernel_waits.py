"""A host thread that answers a kernel which waits for it, on another stream: the first series of blocking calls and the first long messages of
a process, whose kernels have to be there without the device falling quiet.  The waiting kernel gives up after half a second."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import time
import torch
import roc_shmem_b200 as shmem

rt = shmem.init("device", rank=0, world_size=1, heap_bytes=64 << 20, timeout_ms=500)
ctx = rt.ctx_create()
side = torch.cuda.Stream()
flag, word, box = rt.zeros((1,), torch.int64), rt.zeros((1,), torch.int64), rt.zeros((8, 65536), torch.uint8)
src = torch.full((8, 65536), 3, dtype=torch.uint8, device="cuda")
torch.cuda.synchronize()
for i in (1, 2):
    rt.set_stream(side)
    rt.set_blocking(False)
    rt.wait_until(flag, "ge", i)          # a kernel on `side`, not waited for
    rt.set_stream(None)
    rt.set_blocking(True)
    t0 = time.perf_counter()
    if i == 1:
        for k in range(20):
            assert rt.atomic_fetch_add(word, 1, 0) == k
    else:
        for k in range(8):
            ctx.put(box[k], src[k], 0, nbi=True)
        ctx.quiet()
    assert not side.query()
    rt.put_signal(word, word, flag, i, 0)
    side.synchronize()
    assert time.perf_counter() - t0 < 0.4
    assert rt.error_record()["code"] == 0
assert bool((box == 3).all())
ctx.destroy()
rt.finalize()
print("answered")
"""


def test_a_waiting_kernel_is_answered():
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=120, cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0 and r.stdout.strip() == "answered", r.stderr[-2000:]
