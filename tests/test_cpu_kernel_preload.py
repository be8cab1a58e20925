"""Every kernel that the runtime launches is loaded when a PE is created, by the source: a first launch that loads its kernel may need a quiet device,
which a kernel that waits for what is launched does not leave."""
import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda" / "gpu_backend.cu"


def test_every_kernel_is_loaded_at_the_start():
    text = SOURCE.read_text()
    kernels = set(re.findall(r"__global__ void (?:__launch_bounds__\([\w, ]+\) )?(\w+)\(", text))
    loaded = set(re.findall(r"cudaFuncGetAttributes\(&fa, (\w+)\)", text))
    assert len(kernels) > 10 and kernels == loaded
