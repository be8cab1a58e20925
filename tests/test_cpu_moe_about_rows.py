"""A MoE layer plans its grouped products for the tokens of the call, not for the capacity that it was built with."""
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"


@pytest.mark.parametrize("P,tokens,topk", [(1, 500, 2), (2, 300, 2), (1, 4096, 1)])
@pytest.mark.parametrize("training", [False, True])
def test_products_are_told_the_rows(P, tokens, topk, training, monkeypatch):
    from roc_shmem_b200.ops import moe
    E, H, F, max_tokens = 4 * P, 256, 256, 4096
    G, cap = E // P, 256 * 20
    seen = []

    class Native:
        def __getattr__(self, name):
            return lambda *a: 0

    def record(*a, about_rows=0, **k):
        seen.append(about_rows)

    monkeypatch.setattr(moe, "_fast", Native())
    monkeypatch.setattr(moe, "_stream", lambda: 0)
    for n in ("grouped_gemm", "grouped_gemm_act", "grouped_gemm_swiglu_bwd", "grouped_gemm_tn"):
        monkeypatch.setattr(moe, n, record)
    monkeypatch.setattr(moe, "zero_pad_rows", lambda *a: None)
    layer = object.__new__(moe.MoELayer)
    layer.P, layer.G, layer.E, layer.H, layer.F, layer.cap, layer.T, layer.topk = P, G, E, H, F, cap, max_tokens, topk
    layer.training, layer.timeout_ms, layer.ctas, layer.launches, layer.parity, layer.tn_gemm = training, 1000, 1, 0, 0, True
    layer._plan_a = layer._state_a = layer.err_word = 0
    for n in ("topk_idx", "topk_w", "pos", "recv", "meta", "gu", "hact", "yexp", "ybuf", "out", "recv_count", "send_to", "expect_from",
              "arrive", "counts", "counts_all", "ticket", "recv_bwd", "dtopk_w", "dlogit", "dwr_f32", "dwr", "dgu", "dh", "xsave", "dxe", "dx",
              "ybuf_bwd", "meta_bwd", "dxbuf"):
        setattr(layer, n, torch.zeros(max_tokens, 1))
    layer.wr = torch.zeros(E, H)
    layer.w13, layer.w2 = torch.zeros(G, 2 * F, H), torch.zeros(G, H, F)
    layer.w13_t, layer.w2_t, layer.dw13, layer.dw2 = torch.zeros(G, H, 2 * F), torch.zeros(G, F, H), torch.zeros(G, 2 * F, H), torch.zeros(G, H, F)
    layer.route = lambda x: None
    x = torch.zeros(tokens, H)
    layer.forward(x)
    assert seen == [P * tokens * topk // E] * 2
    if training:
        layer.backward(x)
        assert seen == [P * tokens * topk // E] * 6


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_rows_of_a_plan(tmp_path):
    (tmp_path / "t.cc").write_text("#include <cstdio>\n#include \"pair_plan.h\"\nusing namespace bshmem::gemm2;\n"
                                   "int main() { std::printf(\"%d %d %d %d %d\", group_rows(2560, 0), group_rows(2560, 215), group_rows(2560, 9999), "
                                   "group_rows(256, 0), group_rows(2560, 1)); }\n")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-I", str(CUDA), "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout == "2048 215 2560 205 1"
