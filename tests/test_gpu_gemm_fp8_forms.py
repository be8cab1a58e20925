"""Forms of the block-scaled fp8 product and its quantiser at the sizes where they can go wrong: tiles split over clusters of
two, four and eight CTAs with uneven shares of the k-blocks, the last size that is not split, more k-blocks than the ring of
scales and than a warp has lanes, rows and columns that leave the quantiser's 32 x 512 block partly empty."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 256, 128 * 32), (128, 512, 128 * 37), (128, 2560, 128 * 17), (256, 4096, 128 * 9),
                                   (128, 256, 128 * 7), (1152, 4096, 128 * 8), (128 * 37, 1024, 128 * 33)])
def test_gemm_fp8_split_and_plain(M, N, K):
    from roc_shmem_b200.ops.gemm_fp8 import fp8_error_site, gemm_fp8, quantize_act, quantize_weight
    torch.manual_seed(M + N + K)
    x = (torch.randn(M, K, device="cuda") * (1 + torch.arange(M, device="cuda").view(M, 1) % 7)).to(torch.bfloat16)
    x[:, :128] *= 16                                         # k-blocks of different weight: a share taken twice shows
    w = (torch.randn(N, K, device="cuda") * (0.02 * (1 + torch.arange(N, device="cuda").view(N, 1) // 128 % 5))).to(torch.bfloat16)
    qa, qw = quantize_act(x), quantize_weight(w)
    buf = torch.full((M, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm_fp8(qa, qw, buf[:, :N])
    torch.cuda.synchronize()
    assert fp8_error_site() == 0
    assert bool((buf[:, N:] == 7).all())
    a, b = qa.dequantize().double(), qw.dequantize().double()
    ref = a @ b.t()
    # bf16 rounding of the result, plus fp32 sums of K products in any order
    tol = ref.abs() * 2 ** -8 + K * 2 ** -24 * (a.abs() @ b.abs().t())
    assert bool(((buf[:, :N].double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("M,K,pad", [(1, 128, 0), (31, 512, 8), (33, 640, 0), (130, 1152, 8), (64, 384, 4)])
def test_quantiser_edges(M, K, pad):
    """Every block against the definition: scale = absmax / 448 (1 for an all-zero block), payload within half a step of e4m3."""
    from roc_shmem_b200.ops.gemm_fp8 import quantize_act
    torch.manual_seed(M + K)
    x = (torch.randn(M, K + pad, device="cuda") * 5).to(torch.bfloat16)[:, :K]
    x[M // 2, :128] = 0
    qa = quantize_act(x)
    torch.cuda.synchronize()
    amax = x.float().view(M, K // 128, 128).abs().amax(-1)
    scale = torch.where(amax > 0, amax / 448, torch.ones_like(amax))
    assert torch.allclose(qa.scales.t(), scale, rtol=2 ** -22)
    step = x.float().abs().view(M, K // 128, 128) * 2 ** -4 + scale.view(M, K // 128, 1) * 2 ** -10   # normal, subnormal
    assert bool(((qa.dequantize() - x.float()).abs().view(M, K // 128, 128) <= step * 1.001).all())


@pytest.mark.parametrize("M", [0, 65535 * 32, 65535 * 32 + 1])
def test_quantiser_row_counts(M):
    """No rows at all, and the last count of the tiled kernel's grid and the first beyond it."""
    from roc_shmem_b200.ops.gemm_fp8 import quantize_act
    x = torch.randint(-3, 4, (M, 128), device="cuda").to(torch.bfloat16)
    qa = quantize_act(x)
    torch.cuda.synchronize()
    assert qa.q.shape == (M, 128) and qa.scales.shape == (1, M)
    amax = x.abs().amax(1).float() if M else x.new_empty(0).float()
    assert torch.allclose(qa.scales[0], torch.where(amax > 0, amax / 448, torch.ones_like(amax)), rtol=2 ** -22)
    for at in (0, M // 2, M - 3):
        if M:
            part = (qa.q[at:at + 3].view(torch.float8_e4m3fn).float() * qa.scales[0, at:at + 3].unsqueeze(1))
            assert torch.allclose(part, x[at:at + 3].float(), rtol=2 ** -4, atol=1e-6)       # e4m3: half a step is 2^-4


# 152 and 200 tiles on 148 SMs: four tiles of the last wave on clusters of four and eight, 52 on clusters of two; too few k-blocks
@pytest.mark.parametrize("M,N,K", [(128 * 38, 1024, 128 * 16), (128 * 38, 1024, 128 * 33), (128 * 25, 2048, 128 * 25), (128 * 25, 2048, 128 * 9)])
def test_gemm_fp8_last_wave_split(M, N, K):
    test_gemm_fp8_split_and_plain(M, N, K)


def test_gemm_fp8_last_wave_in_a_chain():
    """What follows a product in the stream waits for all of it: each product's result becomes the next one's activations."""
    from roc_shmem_b200.ops.gemm_fp8 import fp8_error_site, gemm_fp8, quantize_act, quantize_weight
    M, N, K = 128 * 38, 1024, 4096
    torch.manual_seed(1)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w, back = (quantize_weight((torch.randn(*s, device="cuda") * 0.03).to(torch.bfloat16)) for s in ((N, K), (K, N)))
    first = None
    for _ in range(5):
        y = x
        for _ in range(4):
            y = gemm_fp8(quantize_act(gemm_fp8(quantize_act(y), w, torch.zeros(M, N, dtype=torch.bfloat16, device="cuda"))), back,
                         torch.zeros(M, K, dtype=torch.bfloat16, device="cuda"))
        if first is None:
            torch.cuda.synchronize()
            first = y.clone()
        assert torch.equal(y, first) and bool(torch.isfinite(y.float()).all())
    assert fp8_error_site() == 0
