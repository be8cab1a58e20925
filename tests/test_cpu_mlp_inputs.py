"""What the gated MLP hands to its kernels on one PE, on the CPU with recorders in the kernels' place: whatever the caller passes,
they get bf16 matrices of the layer's own shape with rows they can address, and a wrong shape is refused before a launch."""
import pytest
import torch

M, H, F = 256, 256, 256


def _linear(n, k):
    from types import SimpleNamespace
    buf = torch.zeros(M, k, dtype=torch.bfloat16)
    layer = SimpleNamespace(x_shard=buf, gathered=buf, out=torch.zeros(M, n, dtype=torch.bfloat16))
    return layer


@pytest.fixture
def make(monkeypatch):
    from roc_shmem_b200.models import llama

    def block(training, fills):
        seen = []
        record = lambda name: lambda *a, **k: seen.append((name, a[0].clone()))  # noqa: E731
        for n in ("gemm_bf16", "grouped_gemm", "grouped_gemm_act", "grouped_gemm_swiglu_bwd", "grouped_gemm_tn"):
            monkeypatch.setattr(llama, n, record(n) if n != "gemm_bf16" else lambda a, b, out, **k: (seen.append(("gemm_bf16", a.clone())), out)[1])
        monkeypatch.setattr(llama, "current_stream", lambda: 0)
        monkeypatch.setattr(llama, "moe_fast", type("Native", (), {"__getattr__": lambda s, n: lambda *a: 0})())
        b = object.__new__(llama.LlamaMLP)
        b.P, b.M, b.H, b.F, b.Fp, b.training, b.launches = 1, M, H, F, F, training, 0
        b.up, b.dgrad_h = _linear(2 * F, H), _linear(F, H)
        b.w13, b.w2_t, b.gu, b.h, b.rows = torch.zeros(2 * F, H), torch.zeros(F, H), b.up.out, torch.zeros(M, F), torch.zeros(1)
        b.dgu, b.dw2, b.dw13, b.w13_t = torch.zeros(M, 2 * F), torch.zeros(H, F), torch.zeros(2 * F, H), torch.zeros(H, 2 * F)
        b.down = b.dgrad_x = lambda x, **k: x
        b._fills = lambda cols: fills
        return b, seen
    return block


def _bad_layouts(v):
    yield "fp32", v.float()
    yield "columns first", v.t().contiguous().t()
    wide = torch.zeros(M, H + 1, dtype=torch.bfloat16)
    wide[:, :H] = v
    yield "odd row pitch", wide[:, :H]
    off = torch.zeros(M * H + 1, dtype=torch.bfloat16)[1:]
    yield "misaligned", off.copy_(v.reshape(-1)).view(M, H)


@pytest.mark.parametrize("fills", [False, True])
def test_inputs_are_converted(make, fills):
    v = (torch.arange(M * H) % 251).view(M, H).to(torch.bfloat16)
    for name, x in [("as it is", v), *_bad_layouts(v)]:
        for training, call in ((False, "forward"), (True, "backward")):
            b, seen = make(training, fills)
            getattr(b, call)(x)
            first = seen[0][1]
            assert first.dtype == torch.bfloat16 and torch.equal(first, v), (name, call)
    row = v[:1].expand(M, H)
    b, seen = make(False, fills)
    b.forward(row)
    assert torch.equal(seen[0][1], row)


@pytest.mark.parametrize("fills", [False, True])
def test_in_place_and_none(make, fills):
    v = torch.randn(M, H).to(torch.bfloat16)
    b, seen = make(False, fills)
    b.up.x_shard.copy_(v)
    b.forward(None)                                          # the caller has written its rows into the layer's buffer
    assert torch.equal(seen[0][1], v)
    b, seen = make(True, fills)
    b.dgrad_h.x_shard.copy_(v)
    b.backward(None)
    assert torch.equal(seen[0][1], v)


@pytest.mark.parametrize("fills", [False, True])
@pytest.mark.parametrize("shape", [(M // 2, H), (2 * M, H), (M, H // 2), (3, M, H)])
def test_wrong_shapes_are_refused(make, fills, shape):
    for training, call in ((False, "forward"), (True, "backward")):
        b, seen = make(training, fills)
        with pytest.raises((RuntimeError, ValueError)):
            getattr(b, call)(torch.zeros(shape, dtype=torch.bfloat16))
        assert not seen


@pytest.mark.parametrize("bad", ["type", "rows", "columns", "order"])
@pytest.mark.parametrize("which", range(4))
@pytest.mark.parametrize("backward", [False, True])
def test_fused_products_check_their_matrices(monkeypatch, backward, which, bad):
    from roc_shmem_b200.ops import moe
    launched = []
    monkeypatch.setattr(moe, "_fast", type("Native", (), {"__getattr__": lambda s, n: lambda *a: launched.append(n) or 0})())
    monkeypatch.setattr(moe, "_stream", lambda: 0)
    G, R, K, N = 2, 512, 64, 256
    shapes = [(R, K), (G * N, K), (R, 2 * N), (R, 2 * N)] if backward else [(R, K), (G * N, K), (R, N), (R, N // 2)]
    run = moe.grouped_gemm_swiglu_bwd if backward else moe.grouped_gemm_act
    ts = [torch.zeros(s, dtype=torch.bfloat16) for s in shapes]
    run(*ts, G)
    assert len(launched) == 1
    r, c = shapes[which]
    ts[which] = {"type": torch.zeros(r, c), "rows": torch.zeros(r // 2, c, dtype=torch.bfloat16),
                 "columns": torch.zeros(r, 2 * c, dtype=torch.bfloat16), "order": torch.zeros(c, r, dtype=torch.bfloat16).t()}[bad]
    if (which, bad) == (1, "rows"):
        ts[which] = ts[which][:r // 2 - 1]                   # (half the weights are the weights of a smaller problem)
    with pytest.raises(ValueError):
        run(*ts, G)
    assert len(launched) == 1
