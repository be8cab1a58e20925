"""Column counts of the bf16 GEMM that are no multiple of a store's width, into a wider buffer: the forms (few tokens, split
or not, CTA pairs, split) write their N columns and nothing behind them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# N = 13, 1001 and 1002 end inside a store of 4 and of 8 columns; the last ones make 2, 8, 32 and 112 tiles of 256 x 256
@pytest.mark.parametrize("M,N,K", [(16, 13, 4096), (16, 1001, 4096), (40, 1002, 72), (100, 1003, 2048), (129, 1001, 4096), (256, 1005, 8192),
                                   (300, 13, 2048), (300, 1001, 2048), (512, 4001, 2056), (1000, 7144, 72)])
def test_nothing_behind_the_last_column(M, N, K):
    from roc_shmem_b200.ops.gemm import gemm_bf16, gemm_error_site
    torch.manual_seed(M + N + K)
    wide = -(-N // 8) * 8 + 8
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.randn(N, K, device="cuda").to(torch.bfloat16)
    buf = torch.full((M + 1, wide), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm_bf16(a, b, buf[:M, :N])
    torch.cuda.synchronize()
    assert gemm_error_site() == 0
    assert bool((buf[:, N:] == 7).all()) and bool((buf[M] == 7).all())
    # bf16 result, and fp32 sums of K products of unit variance in any order
    ref = a.double() @ b.double().t()
    err = (buf[:M, :N].double() - ref).abs()
    assert bool((err <= ref.abs() * 2 ** -8 + K * 2 ** -24 * (a.double().abs() @ b.double().abs().t())).all()), err.max().item()


@pytest.mark.parametrize("M,N,K", [(1000, 7143, 72), (1000, 7142, 72), (520, 1, 64), (300, 257, 136)])
def test_nothing_behind_the_last_column_of_whole_tiles(M, N, K):
    """CTA pairs that do not split their tiles (asked for with an explicit number of CTAs): a TMA store would pad a row's last
    16 bytes with zeros."""
    from roc_shmem_b200.ops.gemm import gemm_bf16, gemm_error_site
    torch.manual_seed(M + N + K)
    wide = -(-N // 8) * 8 + 8
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.randn(N, K, device="cuda").to(torch.bfloat16)
    buf = torch.full((M + 1, wide), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm_bf16(a, b, buf[:M, :N], max_ctas=148)
    torch.cuda.synchronize()
    assert gemm_error_site() == 0
    assert bool((buf[:, N:] == 7).all()) and bool((buf[M] == 7).all())
    ref = a.double() @ b.double().t()
    err = (buf[:M, :N].double() - ref).abs()
    assert bool((err <= ref.abs() * 2 ** -8 + K * 2 ** -24 * (a.double().abs() @ b.double().abs().t())).all()), err.max().item()
