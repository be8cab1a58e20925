"""Grouped GEMM for few rows per group and the one-PE MoE data movement at the sizes where they can go wrong: empty groups,
counts around the MMA's steps of 16 and the chunk of 128, one group only, both epilogues."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("rows", [[0, 0, 1], [16, 17, 0], [127, 128, 129], [256, 3, 0], [0, 250, 15]])
@pytest.mark.parametrize("N,K", [(256, 64), (512, 1000), (512, 8192), (2048, 2048), (9472, 1024)])
def test_grouped_gemm_few_rows(rows, gated, N, K):
    from roc_shmem_b200.ops.moe import grouped_gemm, moe_lib
    torch.manual_seed(sum(rows) + N)
    G, cap = len(rows), 256
    a = torch.randn(G * cap, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(G * N, K, device="cuda") * 0.1).to(torch.bfloat16)
    cnt = torch.tensor(rows, dtype=torch.int32, device="cuda")
    out = torch.full((G * cap, N // 2 if gated else N), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm(a, b, out, G, rows=cnt, gated=gated, few=(max(rows), sum(r > 0 for r in rows)))
    torch.cuda.synchronize()
    assert moe_lib().bshmem_moe_gemm_error_site(1) == 0
    for g, n in enumerate(rows):
        assert bool((out[g * cap + n:(g + 1) * cap] == 7).all())                     # nothing beyond a group's rows
        ref = a[g * cap:g * cap + n].double() @ b[g * N:(g + 1) * N].double().t()
        tol = K * K * 2 ** -24 / K ** 0.5 * 0.1 + 1e-6                               # fp32 sums in another order
        if gated:                                                                    # 32 gate columns, then the 32 up columns
            pair = ref.view(n, N // 64, 2, 32)
            ref = (torch.nn.functional.silu(pair[:, :, 0]) * pair[:, :, 1]).reshape(n, N // 2)
            tol = tol * (1 + pair.abs().max().item() if n else 1) * 2 + 1e-4          # times the other factor; __expf
        err = (out[g * cap:g * cap + n].double() - ref).abs()
        assert bool((err <= ref.abs() * 2 ** -8 + tol).all()), (g, err.max().item())


@pytest.mark.parametrize("T,E,topk", [(1, 8, 2), (5, 64, 8), (129, 16, 1), (4096, 8, 2), (4099, 12, 3)])
def test_router_and_plan(T, E, topk):
    """Router forms on both sides of their limit, uneven expert counts, and the plan's positions in entry order."""
    from roc_shmem_b200.baseline.moe import route
    from roc_shmem_b200.ops.moe import moe_lib
    torch.manual_seed(T + E)
    lib, H = moe_lib(), 264
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    wr = torch.randn(E, H, device="cuda").to(torch.bfloat16)
    n = T * topk
    idx = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    w = torch.empty(n, dtype=torch.float32, device="cuda")
    probs = torch.empty(T, E, dtype=torch.float32, device="cuda")
    pos, cnt = torch.empty_like(idx), torch.empty(E, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert lib.bshmem_moe_router_topk(x.data_ptr(), wr.data_ptr(), T, H, E, topk, idx.data_ptr(), w.data_ptr(), probs.data_ptr(), s) == 0
    assert lib.bshmem_moe_plan(idx.data_ptr(), n, E, pos.data_ptr(), cnt.data_ptr(), s) == 0
    torch.cuda.synchronize()
    ridx, rw = route(x, wr, topk)
    same = (idx.view(T, topk).long() == ridx).all(-1)
    assert same.float().mean() > 0.99                                                # fp32 order may flip near-ties
    assert torch.allclose(w.view(T, topk)[same], rw[same], atol=2e-3)
    assert torch.allclose(probs.sum(-1), torch.ones(T, device="cuda"), atol=1e-5)
    flat, p = idx.tolist(), pos.tolist()
    seen = [0] * E
    for i, e in enumerate(flat):
        assert p[i] == seen[e]
        seen[e] += 1
    assert cnt.tolist() == seen


@pytest.mark.parametrize("T,E,topk,H", [(1, 8, 2, 8), (17, 64, 8, 264), (300, 64, 8, 2048), (2400, 3, 1, 520), (8200, 16, 2, 1032)])
def test_router_backward(T, E, topk, H):
    """d_Wr on both sides of its token block, columns that do not fill one, more experts than warps and fewer, one expert that
    takes most tokens and one that takes none."""
    from roc_shmem_b200.ops.moe import moe_lib
    torch.manual_seed(T + E)
    lib = moe_lib()
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    score = torch.rand(T, E, device="cuda")
    score[: T * 3 // 4, 0] += 1
    if E > topk:
        score[:, E - 1] = -1
    idx = score.topk(topk, dim=1).indices.to(torch.int32).contiguous()
    dlog = torch.randn(T, topk, device="cuda")
    scratch = torch.full((E, H), 5.0, device="cuda")
    dwr = torch.empty(E, H, dtype=torch.bfloat16, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert lib.bshmem_moe_router_backward(x.data_ptr(), idx.data_ptr(), 0, 0, T, H, E, topk, dlog.data_ptr(), scratch.data_ptr(),
                                          dwr.data_ptr(), s) == 0
    torch.cuda.synchronize()
    d = torch.zeros(T, E, dtype=torch.float64, device="cuda").scatter_(1, idx.long(), dlog.double())
    ref, mag = d.t() @ x.double(), d.abs().t() @ x.double().abs()
    assert bool(((dwr.double() - ref).abs() <= ref.abs() * 2 ** -8 + mag * T * 2 ** -24).all())     # bf16; fp32 sums in any order


@pytest.mark.parametrize("T,E,topk", [(17, 24, 4), (2369, 64, 8), (2400, 32, 1)])
def test_router_and_plan_more_forms(T, E, topk):
    """Expert counts that leave a tile partly empty and the largest, with eight and with sixteen warps to a block."""
    test_router_and_plan(T, E, topk)


@pytest.mark.parametrize("T,H,E,topk", [(1, 256, 8, 1), (32, 512, 64, 8), (33, 512, 24, 8), (37, 768, 8, 3), (100, 256, 64, 8), (2500, 2048, 8, 2), (4800, 1024, 12, 5)])
def test_local_rows(T, H, E, topk):
    """Plans of few entries and of more, dispatch, combine and their backward forms on one PE for every rounding of top-k, one
    token and four per warp, a capacity that some entries exceed."""
    import roc_shmem_b200 as shmem
    from roc_shmem_b200.ops.moe import MoELayer, _fast
    rt = shmem.init("device", rank=0, world_size=1, heap_bytes=512 << 20, timeout_ms=5000)
    try:
        torch.manual_seed(T + H)
        layer = MoELayer(rt, H, 256, E, topk, T, capacity_factor=8.0 if T == 1 else 1.0, training=True)
        for t in (layer.wr, layer.w13, layer.w2):
            t.normal_(std=0.05)
        layer.sync_transposes()
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        layer.forward(x)
        torch.cuda.synchronize()
        cap, s = layer.cap, torch.cuda.current_stream().cuda_stream
        idx, pos = layer.topk_idx[:T * topk].view(T, topk).long(), layer.pos[:T * topk].view(T, topk).long()
        live = pos < cap
        seen = [0] * E
        for e, q in zip(idx.view(-1).tolist(), pos.view(-1).tolist()):               # positions in entry order
            assert q == seen[e]
            seen[e] += 1
        assert layer.recv_count.tolist() == [min(c, cap) for c in seen]
        row = (idx * cap + pos.clamp(max=cap - 1))
        assert torch.equal(layer.recv[row[live]], x.view(T, 1, H).expand(T, topk, H)[live])
        y = torch.randn(E * cap, H, device="cuda").to(torch.bfloat16)
        w = torch.randn(T, topk, device="cuda")
        wr = torch.randn(E, H, device="cuda").to(torch.bfloat16)
        picked = y[row].double() * live.unsqueeze(-1)
        out = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
        p = (layer._plan_a, y.data_ptr(), w.data_ptr(), layer.topk_idx.data_ptr(), layer.pos.data_ptr(), T, topk, H, out.data_ptr())
        for with_wr in (0, wr.data_ptr()):
            assert _fast.combine_local(*p, with_wr, s) == 0
            torch.cuda.synchronize()
            parts = torch.cat([picked, w.double().unsqueeze(-1) * wr[idx].double()], 1) if with_wr else picked * w.double().unsqueeze(-1)
            ref, mag = parts.sum(1), parts.abs().sum(1)
            assert bool(((out.double() - ref).abs() <= ref.abs() * 2 ** -8 + mag * 2 * topk * 2 ** -24).all())
        dout = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        g, dw, dlog = torch.zeros_like(y), torch.empty_like(w), torch.empty_like(w)
        assert _fast.dispatch_grad_local(layer._plan_a, dout.data_ptr(), layer.topk_idx.data_ptr(), layer.pos.data_ptr(), w.data_ptr(), T, topk, H,
                                         g.data_ptr(), y.data_ptr(), dw.data_ptr(), dlog.data_ptr(), s) == 0
        torch.cuda.synchronize()
        assert torch.equal(g[row[live]], (dout.float().view(T, 1, H) * w.unsqueeze(-1)).to(torch.bfloat16)[live])
        dref = (picked * dout.double().view(T, 1, H)).sum(-1)
        tol = (picked * dout.double().view(T, 1, H)).abs().sum(-1) * H * 2 ** -24 + 1e-12
        assert bool(((dw.double() - dref).abs() <= tol).all())
        wd = w.double()
        lref = wd * (dref - (wd * dref).sum(1, keepdim=True))
        ltol = wd.abs() * (tol + (wd.abs() * (tol + dref.abs() * topk * 2 ** -23)).sum(1, keepdim=True) + dref.abs() * 2 ** -22)
        assert bool(((dlog.double() - lref).abs() <= ltol + lref.abs() * 2 ** -22).all())
    finally:
        shmem.finalize()


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("rows,few", [([65, 0, 130], (1, 1)), ([17, 16, 1], (16, 1)), ([0, 0, 33], (2, 3)), ([5, 9, 2], (9, 3))])
@pytest.mark.parametrize("N,K", [(256, 8192), (1280, 2048)])
def test_more_rows_and_groups_than_expected(rows, few, gated, N, K):
    """Counts beyond the bounds that chose the launch: more tiles than clusters where the reduction is split, more chunks."""
    from roc_shmem_b200.ops.moe import grouped_gemm, moe_lib
    torch.manual_seed(sum(rows) + N)
    G, cap = len(rows), 256
    a = torch.randn(G * cap, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(G * N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    cnt = torch.tensor(rows, dtype=torch.int32, device="cuda")
    out = torch.full((G * cap, N // 2 if gated else N), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm(a, b, out, G, rows=cnt, gated=gated, few=few)
    torch.cuda.synchronize()
    assert moe_lib().bshmem_moe_gemm_error_site(1) == 0
    for g, n in enumerate(rows):
        assert bool((out[g * cap + n:(g + 1) * cap] == 7).all())
        x, w = a[g * cap:g * cap + n].double(), b[g * N:(g + 1) * N].double()
        ref, tol = x @ w.t(), K * 2 ** -24 * (x.abs() @ w.abs().t())                 # fp32 sums in any order
        if gated:
            (gate, up), (tg, tu) = ref.view(n, N // 64, 2, 32).unbind(2), tol.view(n, N // 64, 2, 32).unbind(2)
            s = torch.sigmoid(gate)
            # slope of silu at most 1.1; 2^-18 for __expf; the factors' own errors
            ref, tol = gate * s * up, (1.1 * tg * (up.abs() + tu) + tu * gate.abs() + (gate * up).abs() * 2 ** -18)
            ref, tol = ref.reshape(n, N // 2), tol.reshape(n, N // 2)
        err = (out[g * cap:g * cap + n].double() - ref).abs()
        assert bool((err <= ref.abs() * 2 ** -8 + tol + 1e-30).all()), (g, (err - tol).max().item())


@pytest.mark.parametrize("T,H,E,topk", [(2048, 4096, 8, 2), (2048, 4096, 16, 2), (2048, 4096, 32, 2), (4096, 2048, 64, 8)])
@pytest.mark.parametrize("scale", [0.02, 0.1])
def test_router_keeps_fp32_sums(T, H, E, topk, scale):
    """The probabilities against fp64: the logits' sums have to be fp32 additions, not a tensor-core chain over the reduction,
    which truncates as it adds and was 2 to 4 times as far off.  In units of 2^-25, the mean size of an fp32 rounding: about three
    for exponential, normalisation and result, and two of the logits' size for their 40 or so additions of partial sums."""
    from roc_shmem_b200.ops.moe import moe_lib
    torch.manual_seed(T + E)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    wr = (torch.randn(E, H, device="cuda") * scale).to(torch.bfloat16)
    idx = torch.empty(T * topk, dtype=torch.int32, device="cuda")
    w, probs = torch.empty(T * topk, device="cuda"), torch.empty(T, E, device="cuda")
    assert moe_lib().bshmem_moe_router_topk(x.data_ptr(), wr.data_ptr(), T, H, E, topk, idx.data_ptr(), w.data_ptr(), probs.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    logits = x.double() @ wr.double().t()
    ref = torch.softmax(logits, -1)
    err = (probs.double() - ref).norm() / ref.norm()
    assert err <= 2 ** -25 * (3 + logits.std().item() * 2), err.item()
