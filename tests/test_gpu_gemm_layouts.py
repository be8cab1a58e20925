"""The three operand layouts of the bf16 GEMM on CTA pairs (forward, data gradient, weight gradient), whole tiles and
tiles split over the pairs of a cluster, at ragged edges and around the tile counts where the form changes, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(out, ref, K):
    # bf16 result: half a unit in the last place (2^-9), doubled for a sum near a tie; fp32 sums of K products of unit
    # variance in two different orders: at most K * 2^-24 of the sum of the magnitudes (about K)
    err = (out.double() - ref).abs()
    assert bool((err <= ref.abs() * 2 ** -8 + K * K * 2 ** -24 / K ** 0.5 + 1e-6).all()), err.max().item()


# rows, columns, reduction of the output; tiles: 2, 6 (split over four pairs), 24 and 32 (over two), 74, 112, 9, 4
@pytest.mark.parametrize("M,N,K", [(264, 8, 8), (257, 520, 7640), (1000, 1288, 2048), (512, 4096, 2056), (512, 9472, 1024),
                                   (1000, 7168, 1040), (8, 2056, 4096), (300, 264, 72), (264, 264, 1536), (264, 264, 1528)])
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
def test_layouts(M, N, K, layout):
    from roc_shmem_b200.ops.gemm import gemm_bf16, gemm_error_site
    a_mn, b_mn = layout == "tn", layout != "nt"
    if a_mn:
        M = M // 8 * 8
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda").to(torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda").to(torch.bfloat16)
    buf = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    first = gemm_bf16(a, b, buf[:M], a_mn=a_mn, b_mn=b_mn).clone()
    for _ in range(3):                                       # the parts of a split tile always add up in the same order
        assert torch.equal(gemm_bf16(a, b, buf[:M], a_mn=a_mn, b_mn=b_mn), first)
    torch.cuda.synchronize()
    assert gemm_error_site() == 0 and bool((buf[M] == 7).all())
    _check(first, (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t()), K)


def test_odd_token_counts_in_the_weight_gradient():
    """The reduction of a weight gradient is the token count: any number, the rest of the last block counts as zero."""
    from roc_shmem_b200.ops.gemm import gemm_bf16
    for tokens in (1, 63, 65, 1001):
        dy = torch.randn(tokens, 264, device="cuda").to(torch.bfloat16)
        x = torch.randn(tokens, 520, device="cuda").to(torch.bfloat16)
        _check(gemm_bf16(dy, x, a_mn=True, b_mn=True), dy.double().t() @ x.double(), tokens)
