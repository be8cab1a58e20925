"""bf16 products whose tiles of 128 columns are one wave: on both sides of the depths from which a tile's reduction is split over two and four
CTA pairs instead, in every operand layout, with rows and columns that end inside a tile and inside a 16-byte piece of it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(512, 2048), (768, 1024), (272, 136), (520, 1000), (264, 9464), (2048, 1144)])
@pytest.mark.parametrize("K", [64, 1544, 2560, 2624, 3776, 3840])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_one_wave(M, N, K, a_mn, b_mn):
    from roc_shmem_b200.ops.gemm import gemm_bf16, gemm_error_site
    torch.manual_seed(M + N + K)
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.randn(N, K, device="cuda").to(torch.bfloat16)
    buf = torch.full((M + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm_bf16(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, buf[:M, :N], a_mn=a_mn, b_mn=b_mn)
    torch.cuda.synchronize()
    assert gemm_error_site() == 0
    assert bool((buf[:, N:] == 7).all()) and bool((buf[M:] == 7).all())
    a, b = a.double(), b.double()
    ref = a @ b.t()
    # bf16 rounding of the result, plus fp32 sums of K products in any order
    tol = ref.abs() * 2 ** -8 + K * 2 ** -24 * (a.abs() @ b.abs().t())
    assert bool(((buf[:M, :N].double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("kb,tokens", [(4, 106), (8, 124), (12, 142), (20, 178), (32, 232), (32, 256), (33, 256)])
@pytest.mark.parametrize("N", [128, 1032, 9472, 9473])
@pytest.mark.parametrize("b_mn", [False, True])
def test_few_tokens_on_pairs(kb, tokens, N, b_mn):
    """Both sides of the line between the few-token form and pairs on one wave of tiles of 128 columns."""
    from roc_shmem_b200.ops.gemm import gemm_bf16, gemm_error_site
    if b_mn and N % 8:
        pytest.skip("refused: TMA needs rows of a multiple of 16 bytes")
    K = 64 * kb - 8
    for M in (tokens - 1, tokens):
        torch.manual_seed(M + N + K)
        a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.randn(N, K, device="cuda").to(torch.bfloat16)
        buf = torch.full((M + 1, (N + 15) // 8 * 8), 7.0, dtype=torch.bfloat16, device="cuda")
        gemm_bf16(a, b.t().contiguous() if b_mn else b, buf[:M, :N], b_mn=b_mn)
        torch.cuda.synchronize()
        assert gemm_error_site() == 0
        assert bool((buf[:, N:] == 7).all()) and bool((buf[M:] == 7).all())
        a, b = a.double(), b.double()
        ref = a @ b.t()
        tol = ref.abs() * 2 ** -8 + K * 2 ** -24 * (a.abs() @ b.abs().t())
        assert bool(((buf[:M, :N].double() - ref).abs() <= tol).all())
