"""What the MoE layer tells the few-row GEMM about its groups, with several PEs that bring different numbers of tokens: the
launch shape is chosen for the counts that can arrive, not for those this PE would expect from its own tokens."""
import pytest
import torch


@pytest.mark.parametrize("P,mine,other,topk", [(2, 1, 64, 2), (8, 1, 64, 1), (4, 3, 17, 8), (1, 5, 5, 2)])
@pytest.mark.parametrize("training", [False, True])
def test_bounds_hold_for_unequal_tokens(P, mine, other, topk, training, monkeypatch):
    from roc_shmem_b200.ops import moe
    E, H, F, max_tokens, cap = 8 * P, 256, 256, 64, 256 * P
    G = E // P
    seen = []

    class Native:
        def __getattr__(self, name):
            return lambda *a: 0

    monkeypatch.setattr(moe, "_fast", Native())
    monkeypatch.setattr(moe, "_stream", lambda: 0)
    monkeypatch.setattr(moe, "grouped_gemm", lambda *a, few=None, **k: seen.append(few))
    monkeypatch.setattr(moe, "grouped_gemm_act", lambda *a, **k: None)
    layer = object.__new__(moe.MoELayer)
    layer.P, layer.G, layer.E, layer.H, layer.F, layer.cap, layer.T, layer.topk = P, G, E, H, F, cap, max_tokens, topk
    layer.training, layer.timeout_ms, layer.ctas, layer.launches, layer.parity = training, 1000, 1, 0, 0
    layer._plan_a = layer._state_a = layer.err_word = 0
    names = ("topk_idx", "topk_w", "pos", "recv", "meta", "gu", "hact", "yexp", "ybuf", "out", "recv_count", "send_to", "expect_from",
             "arrive", "counts", "counts_all", "ticket")
    for n in names:
        setattr(layer, n, torch.zeros(max_tokens, 1))
    layer.w13, layer.w2 = torch.zeros(G, 2 * F, H), torch.zeros(G, H, F)
    layer.route = lambda x: None
    layer.forward(torch.zeros(mine, H))
    hints = [f for f in seen if f is not None]
    assert hints                                             # few enough tokens for the form at all
    tokens = [mine] + [other] * (P - 1)
    for rows, active in hints:
        assert rows >= min(cap, sum(tokens))                 # every token picks the same group
        assert active >= min(G, sum(tokens) * topk)          # ... or they spread as far as they can
