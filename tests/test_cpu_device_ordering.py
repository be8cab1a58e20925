"""Scopes of the device API's ordering calls, by its source (an order that memory may or may not show cannot be run into):
quiet publishes to the host too, whatever the PEs share; a fence orders for the PEs, so GPU scope does where they share a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc"
HEADER = CSRC / "include" / "bshmem_device.cuh"


def _body(name: str) -> str:
    text = HEADER.read_text()
    i = text.index(f"void {name}(const State& s) {{")
    depth, j = 1, text.index("{", i) + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
    return text[i:j]


def test_quiet_is_system_scope():
    assert re.findall(r"fence\.acq_rel\.(\w+)", _body("quiet")) == ["sys"] and "one_gpu" not in _body("quiet")
    assert "fence_peers" not in _body("quiet")


def test_fence_has_the_scope_of_its_peers():
    assert "fence_peers" in _body("fence")
    peers = _body("fence_peers")
    assert peers.index("one_gpu") < peers.index("fence.acq_rel.gpu") < peers.index("else") < peers.index("fence.acq_rel.sys")


def test_a_served_signal_is_there_before_its_answer():
    """k_calls answers from a stream of its own: payload, fence, signal, fence, answer."""
    text = (CSRC / "cuda" / "gpu_backend.cu").read_text()
    case = text[text.index("case CALL_PUT_SIGNAL:\n"):]
    case = case[:case.index("break;")]
    steps = re.findall(r"copy_bytes<|__syncthreads|fence_peers|signal_update|signal_done", case)
    assert steps == ["copy_bytes<", "__syncthreads", "fence_peers", "signal_update", "fence_peers", "signal_done"]


def test_a_contexts_words_are_cleared_where_they_are_used():
    """A context's stream does not wait for the default stream: what its kernels find zeroed is zeroed in that stream."""
    text = (CSRC / "cuda" / "gpu_backend.cu").read_text()
    body = text[text.index("int ctx_open("):text.index("void ctx_close(")]
    assert re.findall(r"cudaMalloc\(&L\.(\w+)", body) == re.findall(r"cudaMemsetAsync\(L\.(\w+), 0, sizeof\(\w+\), L\.stream\)", body)
    assert "cudaMemset(" not in body
