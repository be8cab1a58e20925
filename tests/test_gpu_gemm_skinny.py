"""The few-token form of the bf16 GEMM (weight tiles, split reduction) at the edges of its tiles: token counts around the
MMA's steps of 16 and the limits between its launch shapes, ragged column counts and reduction lengths."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 15, 16, 17, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 72), (736, 1000), (2048, 4096), (14336, 512)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_few_tokens(M, N, K, b_mn):
    from roc_shmem_b200.ops.gemm import gemm_bf16, gemm_error_site
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda").to(torch.bfloat16)
    buf = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    for _ in range(2):
        gemm_bf16(a, b, buf[:M], b_mn=b_mn)
    torch.cuda.synchronize()
    assert gemm_error_site() == 0
    assert bool((buf[M] == 7).all())                         # nothing beyond the last token's row
    # bf16 rounds the result to 2^-9 of its size; fp32 sums of K products of unit variance differ by their order:
    # at most K * 2^-24 of the sum of the magnitudes (about K), against a result of about sqrt(K)
    ref = a.double() @ (b.double() if b_mn else b.double().t())
    err = (buf[:M].double() - ref).abs()
    assert bool((err <= ref.abs() * 2 ** -8 + K * K * 2 ** -24 / K ** 0.5 + 1e-6).all()), err.max().item()


def test_few_tokens_reproducible_and_strided():
    """Same bits every time (fixed summation order), with leading dimensions larger than the rows."""
    from roc_shmem_b200.ops.gemm import gemm_bf16
    torch.manual_seed(0)
    a = torch.randn(40, 1024, device="cuda").to(torch.bfloat16)[:, :968]
    b = torch.randn(1032, 1000, device="cuda").to(torch.bfloat16)[:, :968]
    out = torch.zeros(40, 1200, dtype=torch.bfloat16, device="cuda")
    first = gemm_bf16(a, b, out[:, :1032]).clone()
    for _ in range(5):
        assert torch.equal(gemm_bf16(a, b, out[:, :1032]), first)
    assert int((out[:, 1032:] != 0).sum()) == 0
    assert torch.equal(first, gemm_bf16(a.contiguous(), b.contiguous()))
