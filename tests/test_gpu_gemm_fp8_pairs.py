"""The block-scaled fp8 product on CTA pairs: the shortest reductions it takes, tiles that reach behind the matrix, several tiles per pair,
a last wave that goes to the split form, and the same bits as the form on single CTAs (which scales off a 16-byte boundary get)."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K):
    from roc_shmem_b200.ops.gemm_fp8 import quantize_act, quantize_weight
    torch.manual_seed(M + N + K)
    x = (torch.randn(M, K, device="cuda") * (1 + torch.arange(M, device="cuda").view(M, 1) % 7)).to(torch.bfloat16)
    x[:, :128] *= 16                                         # k-blocks of different weight: a scale of another k-block shows
    w = (torch.randn(N, K, device="cuda") * (0.02 * (1 + torch.arange(N, device="cuda").view(N, 1) // 128 % 5))).to(torch.bfloat16)
    return quantize_act(x), quantize_weight(w)


def _product(qa, qw, M, N):
    from roc_shmem_b200.ops.gemm_fp8 import fp8_error_site, gemm_fp8
    buf = torch.full((M + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm_fp8(qa, qw, buf[:M, :N])
    torch.cuda.synchronize()
    assert fp8_error_site() == 0
    assert bool((buf[:, N:] == 7).all()) and bool((buf[M:] == 7).all())
    return buf[:M, :N]


# 2 tiles of 128 rows per tile of a pair; 74 pairs
@pytest.mark.parametrize("M,N,K", [(256, 256, 512), (128, 256, 512), (384, 512, 512), (2560, 2304, 1536), (128 * 33, 1280, 512), (640, 10240, 7168),
                                   (4096, 1280, 4096), (128 * 33, 1280, 4096)])
def test_gemm_fp8_pairs(M, N, K):
    qa, qw = _operands(M, N, K)
    out = _product(qa, qw, M, N)
    a, b = qa.dequantize().double(), qw.dequantize().double()
    ref = a @ b.t()
    # bf16 rounding of the result, plus fp32 sums of K products in any order
    tol = ref.abs() * 2 ** -8 + K * 2 ** -24 * (a.abs() @ b.abs().t())
    assert bool(((out.double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("M,N,K", [(256, 512, 512), (384, 512, 512), (2560, 2304, 1536), (18 * 256, 1024, 7168)])
def test_same_bits_as_single_ctas(M, N, K):
    qa, qw = _operands(M, N, K)
    shifted = torch.empty(qa.scales.numel() + 1, dtype=torch.float32, device="cuda")[1:].view_as(qa.scales)
    shifted.copy_(qa.scales)
    assert torch.equal(_product(qa, qw, M, N), _product(dataclasses.replace(qa, scales=shifted), qw, M, N))
