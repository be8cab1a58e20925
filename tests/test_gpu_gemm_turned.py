"""bf16 products whose operands change places because that leaves fewer empty rows in the tiles (the result is stored transposed): one and two
accumulators per tile, rows and columns that end inside a tile, a store box and a 16-byte piece, in every operand layout; and their neighbours
that are multiplied as they are."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(261, 8192), (264, 14336), (272, 9480), (320, 14344), (384, 8200), (385, 14328), (577, 8192), (640, 8168), (808, 4096),
                                 (1152, 4104), (1304, 7168), (272, 9481), (512, 14336)])
@pytest.mark.parametrize("K", [64, 200, 1544])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_turned(M, N, K, a_mn, b_mn):
    from roc_shmem_b200.ops.gemm import gemm_bf16, gemm_error_site
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("refused: TMA needs rows of a multiple of 16 bytes")
    torch.manual_seed(M + N + K)
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.randn(N, K, device="cuda").to(torch.bfloat16)
    buf = torch.full((M + 1, (N + 15) // 8 * 8), 7.0, dtype=torch.bfloat16, device="cuda")
    for out, before in ((buf[:M, :N], 7.0), (torch.zeros(M, (N + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")[:, :N], 0.0)):
        gemm_bf16(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, out, a_mn=a_mn, b_mn=b_mn)
        torch.cuda.synchronize()
        assert gemm_error_site() == 0
        ref = a.float() @ b.float().t()
        # bf16 rounding of the result, plus fp32 sums of K products in any order on both sides
        tol = ref.abs() * 2 ** -8 + 2 * K * 2 ** -24 * (a.float().abs() @ b.float().abs().t())
        assert bool(((out.float() - ref).abs() <= tol).all())
    assert bool((buf[:, N:] == 7).all()) and bool((buf[M:] == 7).all())


def test_the_bits_do_not_depend_on_it():
    """A row of the result is the same whichever way the product was multiplied: 320 rows are turned, 512 are not."""
    from roc_shmem_b200.ops.gemm import gemm_bf16
    torch.manual_seed(5)
    a, b = torch.randn(512, 3584, device="cuda").to(torch.bfloat16), torch.randn(8192, 3584, device="cuda").to(torch.bfloat16)
    assert torch.equal(gemm_bf16(a[:320], b), gemm_bf16(a, b)[:320])
