"""The gated MLP's training kernels, SwiGLU in the projection's epilogue and its derivative in the gradient's, at tile edges:
empty groups, one row, rows that end inside, at and behind a warp's 32 rows and a tile's 256, ragged K, one tile and several."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _split(gu):
    """Interleaved pre-activations [R, 2F] (32 gate columns, 32 up columns, ...) as (gate, up), [R, F] each."""
    v = gu.view(gu.shape[0], gu.shape[1] // 64, 2, 32)
    return v[:, :, 0].reshape(gu.shape[0], -1), v[:, :, 1].reshape(gu.shape[0], -1)


@pytest.mark.parametrize("rows", [[256, 0, 1], [31, 32, 33], [255, 512, 257]])
@pytest.mark.parametrize("F,K", [(256, 64), (512, 200), (1024, 1032)])
def test_fused_swiglu_forward_and_backward(rows, F, K):
    from roc_shmem_b200.ops.moe import grouped_gemm_act, grouped_gemm_swiglu_bwd, moe_lib
    torch.manual_seed(sum(rows) + F)
    G, cap, bf = len(rows), 512, torch.bfloat16
    cnt = torch.tensor(rows, dtype=torch.int32, device="cuda")
    a = torch.randn(G * cap, K, device="cuda").to(bf)
    w = (torch.randn(G * 2 * F, K, device="cuda") * K ** -0.5).to(bf)
    gu, act = torch.full((G * cap, 2 * F), 7.0, dtype=bf, device="cuda"), torch.full((G * cap, F), 7.0, dtype=bf, device="cuda")
    grouped_gemm_act(a, w, gu, act, G, rows=cnt)
    dy, w2t = torch.randn(G * cap, K, device="cuda").to(bf), (torch.randn(G * F, K, device="cuda") * K ** -0.5).to(bf)
    dgu = torch.full((G * cap, 2 * F), 7.0, dtype=bf, device="cuda")
    grouped_gemm_swiglu_bwd(dy, w2t, gu, dgu, G, rows=cnt)
    torch.cuda.synchronize()
    assert moe_lib().bshmem_moe_gemm_error_site(1) == 0
    for g, n in enumerate(rows):
        used, rest = slice(g * cap, g * cap + n), slice(g * cap + -(-n // 32) * 32, (g + 1) * cap)     # stored by 32 rows
        assert bool((gu[rest] == 7).all()) and bool((act[rest] == 7).all()) and bool((dgu[rest] == 7).all())
        if not n:
            continue
        u = 2.0 ** -8                                                     # one rounding to bf16; fp32 sums of K products: K / 2^24
        ref = a[used].double() @ w[g * 2 * F:(g + 1) * 2 * F].double().t()
        sums = K * 2 ** -24 * (a[used].double().abs() @ w[g * 2 * F:(g + 1) * 2 * F].double().abs().t())
        assert bool(((gu[used].double() - ref).abs() <= ref.abs() * u + sums).all())
        # activations and gradients start from the stored, rounded pre-activations; 2^-18: __expf
        gate, up = _split(gu[used].double())
        s = torch.sigmoid(gate)
        h = gate * s * up
        assert bool(((act[used].double() - h).abs() <= h.abs() * (u + 2 ** -18) + 1e-30).all())
        b = w2t[g * F:(g + 1) * F].double()
        d = dy[used].double() @ b.t()
        dtol = d.abs() * u + K * 2 ** -24 * (dy[used].double().abs() @ b.abs().t())      # d is rounded to bf16 on the way
        dgate, dup = _split(dgu[used].double())
        # the factor 1 + g (1 - s) cancels near its zero: its error is absolute, up to |g| 2^-18 (fp32 and __expf)
        fg, fu = up * s * (1 + gate * (1 - s)), gate * s
        fg_err, fu_err = up.abs() * s * (1 + gate.abs()) * 2 ** -18, fu.abs() * 2 ** -18
        for got, f, ferr in ((dgate, fg, fg_err), (dup, fu, fu_err)):
            tol = (d * f).abs() * u + (dtol * f.abs() + (d.abs() + dtol) * ferr) * (1 + u) + 1e-30
            assert bool(((got - d * f).abs() <= tol).all()), ((got - d * f).abs() - tol).max().item()
