"""Waits of a whole warp, by the kernels' source (lanes that disagree cannot be staged): what a lane saw by itself (ptx::mbar_test) decides nothing
before all lanes have voted on it, because the waits behind such a decision are votes of all lanes."""
import re
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"
USERS = [f for f in sorted(CUDA.glob("*.cu*")) if "ptx::mbar_test(" in f.read_text()]


@pytest.mark.parametrize("path", USERS, ids=lambda p: p.name)
def test_what_a_lane_saw_is_voted_on(path):
    text = re.sub(r"//.*", "", path.read_text())
    names = set(re.findall(r"(\w+)\s*=\s*ptx::mbar_test\(", text))
    assert len(names) and text.count("ptx::mbar_test(") == len(re.findall(r"\w+\s*=\s*ptx::mbar_test\(", text))
    for name in names:
        for use in re.finditer(rf"\b{name}\b", text):
            before, behind = text[:use.start()], text[use.end():]
            made = re.match(r"\s*=\s*(ptx::mbar_test\(|false)", behind)
            assert made or re.search(r"__all_sync\(0xffffffffu, [\w &]*$", before), f"{name}: {text[use.start() - 40:use.end() + 20]}"
