"""PyTorch operator registration for the hand-written kernels.

``torch.ops.bshmem.linear(x, w)`` is ``x @ w.T`` on the tcgen05 GEMM with a registered fake (meta)
implementation and an autograd formula whose two gradients also run on the tcgen05 kernels
(data gradient: MN-major weight operand; weight gradient: both operands MN-major; nothing is
transposed).  ``torch.ops.bshmem.linear_fp8`` quantises both operands to block-scaled e4m3 and runs
the fp8 kernel (forward only).  The reference has no PyTorch layer.
"""
from __future__ import annotations

import torch
from torch.utils._device import DeviceContext

from .gemm import gemm_bf16
from .gemm_fp8 import gemm_fp8, quantize_act, quantize_weight


def _check_linear(x: torch.Tensor, w: torch.Tensor) -> None:
    if x.dim() != 2 or w.dim() != 2 or x.shape[1] != w.shape[1]:
        raise ValueError(f"linear: shape mismatch {tuple(x.shape)} x {tuple(w.shape)}")
    if x.dtype != torch.bfloat16 or w.dtype != torch.bfloat16:
        raise ValueError("linear: bf16 operands only")


@torch.library.custom_op("bshmem::linear", mutates_args=())
def linear(x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    _check_linear(x, w)
    return gemm_bf16(x.contiguous(), w.contiguous())


@linear.register_fake
def _(x, w):
    return x.new_empty((x.shape[0], w.shape[0]))


@torch.library.custom_op("bshmem::linear_wgrad", mutates_args=())
def linear_wgrad(dy: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """dW[N, K] = dy[M, N].T @ x[M, K] on token-major operands, for any number of tokens."""
    return gemm_bf16(dy.contiguous(), x.contiguous(), a_mn=True, b_mn=True)


@linear_wgrad.register_fake
def _(dy, x):
    return x.new_empty((dy.shape[1], x.shape[1]))


@torch.library.custom_op("bshmem::linear_dgrad", mutates_args=())
def linear_dgrad(dy: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """dX[M, K] = dy[M, N] @ w[N, K]; the weight is read as it is stored."""
    return gemm_bf16(dy.contiguous(), w.contiguous(), b_mn=True)


@linear_dgrad.register_fake
def _(dy, w):
    return dy.new_empty((dy.shape[0], w.shape[1]))


def _save_inputs(ctx, inputs, output):
    ctx.save_for_backward(*inputs)


def _linear_backward(ctx, dy):
    x, w = ctx.saved_tensors
    dy = dy.contiguous()
    dx = torch.ops.bshmem.linear_dgrad(dy, w) if ctx.needs_input_grad[0] else None
    dw = torch.ops.bshmem.linear_wgrad(dy, x) if ctx.needs_input_grad[1] else None
    return dx, dw


def _dgrad_backward(ctx, g):
    dy, w = ctx.saved_tensors
    g = g.contiguous()
    return (torch.ops.bshmem.linear(g, w) if ctx.needs_input_grad[0] else None,
            torch.ops.bshmem.linear_wgrad(dy, g) if ctx.needs_input_grad[1] else None)


linear.register_autograd(_linear_backward, setup_context=_save_inputs)
linear_dgrad.register_autograd(_dgrad_backward, setup_context=_save_inputs)      # second order through dX; dW has none


@torch.library.custom_op("bshmem::linear_fp8", mutates_args=())
def linear_fp8(x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """x @ w.T with both operands quantised on the fly to block-scaled e4m3 (1x128 / 128x128 scales)."""
    _check_linear(x, w)
    return gemm_fp8(quantize_act(x.contiguous()), quantize_weight(w.contiguous()))


@linear_fp8.register_fake
def _(x, w):
    return x.new_empty((x.shape[0], w.shape[0]))


class _LinearFn(torch.autograd.Function):
    """The same layer without the dispatcher: a custom operator costs 60 to 100 us of host time per call (fake-tensor
    and schema machinery), a training step of the layer makes three of them."""

    @staticmethod
    def forward(ctx, x, w):
        _check_linear(x, w)
        ctx.save_for_backward(x, w)          # the inputs themselves: second-order gradients go through them
        return gemm_bf16(x.contiguous(), w.contiguous())

    @staticmethod
    def backward(ctx, dy):
        # the registered operators where the gradients are differentiated or batched themselves, or watched
        if torch.is_grad_enabled() or not _unwatched() or type(dy) is not torch.Tensor or torch._C._functorch.is_legacy_batchedtensor(dy):
            return _linear_backward(ctx, dy)
        x, w = ctx.saved_tensors
        x, w, dy = x.contiguous(), w.contiguous(), dy.contiguous()
        need_x, need_w = ctx.needs_input_grad
        return (gemm_bf16(dy, w, b_mn=True) if need_x else None, gemm_bf16(dy, x, a_mn=True, b_mn=True) if need_w else None)


_PLAIN = (torch.Tensor, torch.nn.Parameter)


def _unwatched() -> bool:
    """Nobody watches or rewrites operators: no compilation or tracing, no dispatch or function mode (fake tensors, make_fx,
    counters; the one of a default device only adds an argument to factories), no functorch transform (vmap, grad, jvp)."""
    C = torch._C
    modes = C._len_torch_function_stack()
    return (C._len_torch_dispatch_stack() == 0 and C._functorch.peek_interpreter_stack() is None and C._get_tracing_state() is None
            and (modes == 0 or modes == 1 and type(C._get_function_stack_at(0)) is DeviceContext) and not torch.compiler.is_compiling())


class Linear(torch.nn.Module):
    """Drop-in bf16 ``nn.Linear`` (no bias) whose forward and both gradients run on the tcgen05 kernels."""

    def __init__(self, in_features: int, out_features: int, device=None):
        super().__init__()
        self.weight = torch.nn.Parameter(torch.empty((out_features, in_features), dtype=torch.bfloat16, device=device))
        torch.nn.init.normal_(self.weight, std=0.02)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        w = self.weight
        # the registered operator for everything but plain tensors in GPU memory (meta, fake and other subclasses)
        if not (x.is_cuda and w.is_cuda and type(x) in _PLAIN and type(w) in _PLAIN and _unwatched()):
            lead = x.shape[:-1]
            return torch.ops.bshmem.linear(x.reshape(-1, x.shape[-1]), w).reshape(*lead, -1)
        if x.dim() == 2:
            return _LinearFn.apply(x, w)
        return _LinearFn.apply(x.reshape(-1, x.shape[-1]), w).reshape(*x.shape[:-1], -1)


# ---- collectives on the calling PE's runtime (roc_shmem_b200.current()) --------------------------------
# Arbitrary tensors are staged through symmetric scratch that is cached per (shape, dtype); symmetric
# tensors (rt.empty / rt.zeros) are used in place.  Works on the NVLink and on the CPU backend.
_scratch: dict = {}


def _sym(rt, key: str, shape, dtype) -> torch.Tensor:
    k = (id(rt), key, tuple(shape), dtype)
    t = _scratch.get(k)
    if t is None:
        t = rt.empty(tuple(shape), dtype)
        _scratch[k] = t
    return t


def release_scratch() -> None:
    """Free the cached symmetric staging buffers (collective: every PE must call it)."""
    from .. import current
    rt = current()
    for k in [k for k in _scratch if k[0] == id(rt)]:
        rt.free(_scratch.pop(k))


@torch.library.custom_op("bshmem::all_reduce", mutates_args=())
def all_reduce(x: torch.Tensor, op: str = "sum") -> torch.Tensor:
    """Reduction over all PEs (`to_all`); every PE gets the result."""
    from .. import current
    rt = current()
    src, dst = _sym(rt, "ar_src", x.shape, x.dtype), _sym(rt, "ar_dst", x.shape, x.dtype)
    src.copy_(x)
    rt.reduce(dst, src, op)
    return dst.clone()


@all_reduce.register_fake
def _(x, op="sum"):
    return torch.empty_like(x)


@torch.library.custom_op("bshmem::all_gather", mutates_args=())
def all_gather(x: torch.Tensor) -> torch.Tensor:
    """Concatenation of every PE's `x` along dimension 0 (`fcollect`)."""
    from .. import current
    rt = current()
    src = _sym(rt, "ag_src", x.shape, x.dtype)
    dst = _sym(rt, "ag_dst", (rt.n_pes * x.shape[0],) + tuple(x.shape[1:]), x.dtype)
    src.copy_(x)
    rt.fcollect(dst, src)
    return dst.clone()


@all_gather.register_fake
def _(x):
    from .. import current
    return x.new_empty((current().n_pes * x.shape[0],) + tuple(x.shape[1:]))


@torch.library.custom_op("bshmem::reduce_scatter", mutates_args=())
def reduce_scatter(x: torch.Tensor, op: str = "sum") -> torch.Tensor:
    """This PE's 1/n slice (dimension 0) of the reduction of every PE's `x`."""
    from .. import current
    rt = current()
    if x.shape[0] % rt.n_pes:
        raise ValueError("reduce_scatter: dimension 0 must divide by the number of PEs")
    src = _sym(rt, "rs_src", x.shape, x.dtype)
    dst = _sym(rt, "rs_dst", (x.shape[0] // rt.n_pes,) + tuple(x.shape[1:]), x.dtype)
    src.copy_(x)
    rt.reduce_scatter(dst, src, op)
    return dst.clone()


@reduce_scatter.register_fake
def _(x, op="sum"):
    from .. import current
    return x.new_empty((x.shape[0] // current().n_pes,) + tuple(x.shape[1:]))


@torch.library.custom_op("bshmem::all_to_all", mutates_args=())
def all_to_all(x: torch.Tensor) -> torch.Tensor:
    """Block k (dimension 0 split in n equal blocks) of PE j's `x` becomes block j of PE k's result."""
    from .. import current
    rt = current()
    if x.shape[0] % rt.n_pes:
        raise ValueError("all_to_all: dimension 0 must divide by the number of PEs")
    src, dst = _sym(rt, "a2a_src", x.shape, x.dtype), _sym(rt, "a2a_dst", x.shape, x.dtype)
    src.copy_(x)
    rt.alltoall(dst, src)
    return dst.clone()


@all_to_all.register_fake
def _(x):
    return torch.empty_like(x)


def _ar_backward(ctx, g):
    return torch.ops.bshmem.all_reduce(g.contiguous(), "sum"), None


def _ag_backward(ctx, g):
    return torch.ops.bshmem.reduce_scatter(g.contiguous(), "sum")


def _rs_backward(ctx, g):
    return torch.ops.bshmem.all_gather(g.contiguous()), None


def _a2a_backward(ctx, g):
    return torch.ops.bshmem.all_to_all(g.contiguous())


# gradients of the sum-collectives are the matching collectives (valid for op == "sum")
all_reduce.register_autograd(_ar_backward)
all_gather.register_autograd(_ag_backward)
reduce_scatter.register_autograd(_rs_backward)
all_to_all.register_autograd(_a2a_backward)
