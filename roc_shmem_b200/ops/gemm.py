"""Hand-written tcgen05 GEMM (sm_100a): ``C = A @ B.T`` with A [M, K], B [N, K].

This is the compute core under the fused tensor-parallel kernels; the reference
contains no GEMM (it is a communication runtime only), so there is no parity
citation — the layout convention is torch's ``F.linear(x, w)``.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from .. import _native

_declared = False
_run = None                                            # bshmem_gemm_bf16_ex without ctypes (see _native.fast)
_raw_stream = torch._C._cuda_getCurrentRawStream
_BF16 = torch.bfloat16


def current_stream() -> int:
    """Handle of the current CUDA stream of the current device (torch.cuda.current_stream() builds an object)."""
    return _raw_stream(torch._C._cuda_getDevice())


def gemm_lib() -> C.CDLL:
    global _declared, _run
    lib = _native.load("libbshmem_gemm.so")
    if not _declared:
        lib.bshmem_gemm_last_error.restype = C.c_char_p
        lib.bshmem_gemm_bf16.restype = C.c_int
        lib.bshmem_gemm_bf16.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int,
                                         C.c_int, C.c_void_p, C.c_int, C.c_int]
        lib.bshmem_gemm_error_site.restype = C.c_int
        lib.bshmem_gemm_error_site.argtypes = [C.c_int]
        lib.bshmem_gemm_bf16_ex.restype = C.c_int
        lib.bshmem_gemm_bf16_ex.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p] + [C.c_int] * 8 + [C.c_void_p, C.c_int, C.c_int]
        _run = _native.fast(lib, "bshmem_gemm_bf16_ex")
        _declared = True
    return lib


def gemm_bf16(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None, *, max_ctas: int = 0,
              timeout_ms: int = 2000, a_mn: bool = False, b_mn: bool = False) -> torch.Tensor:
    """out[M, N] = a[M, K] @ b[N, K].T in bf16 with fp32 accumulation (tcgen05 + TMEM).
    With ``a_mn`` the first operand is stored [K, M], with ``b_mn`` the second one [K, N] (the gradient products of a
    linear layer); the tensor core reads them as they are, nothing is transposed in memory.

    Launches on the current CUDA stream.  Fails loudly if the native library is
    missing — there is no eager fallback."""
    if not (a.is_cuda and b.is_cuda):
        raise ValueError("gemm_bf16 needs CUDA tensors")
    if a.dtype is not _BF16 or b.dtype is not _BF16:
        raise ValueError("gemm_bf16 needs bf16 operands")
    sa, sb = a.shape, b.shape
    if len(sa) != 2 or len(sb) != 2 or sa[not a_mn] != sb[not b_mn]:
        raise ValueError(f"shape mismatch: a {tuple(sa)} b {tuple(sb)}")
    lda, ka = a.stride()
    ldb, kb = b.stride()
    if ka != 1 or kb != 1:
        raise ValueError("operands must be K-major (last dimension contiguous)")
    K, M = sa if a_mn else sa[::-1]
    N = sb[b_mn]
    if out is None:
        out = a.new_empty((M, N))
        ldc = N
    else:
        if out.shape != (M, N) or out.dtype is not _BF16 or out.stride(1) != 1:
            raise ValueError("bad output tensor")
        ldc = out.stride(0)
    if _run is None:
        gemm_lib()
    st = _run(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, lda, ldb, ldc, a_mn, b_mn,
              _raw_stream(torch._C._cuda_getDevice()), max_ctas, timeout_ms)
    if st != 0:
        raise RuntimeError(f"bshmem_gemm_bf16 failed ({st}): {gemm_lib().bshmem_gemm_last_error().decode()}")
    return out


def gemm_error_site(clear: bool = True) -> int:
    """0 if no in-kernel bounded wait ran out since the last clear, else the site code."""
    return int(gemm_lib().bshmem_gemm_error_site(int(clear)))
