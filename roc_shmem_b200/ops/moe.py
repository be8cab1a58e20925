"""Expert-parallel MoE layer on the device API: router, dispatch / combine over NVLink
with put + signal semantics, grouped tcgen05 expert GEMMs, forward and backward.

Mixtral-style: E experts spread over P PEs (E/P per PE), top-k routing with softmax
over all experts and renormalisation over the chosen ones, SwiGLU experts
(w1 = gate, w3 = up, w2 = down).  The kernels are in csrc/cuda/moe_kernels.cu and
moe_gemm.cu; the NCCL all_to_all + cuBLAS equivalent is roc_shmem_b200/baseline/moe.py.
The reference has no MoE layer — this is a north-star workload built on its device API
shape (put, signal, wait).
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from .. import _native
from ..gpu import DevState
from .gemm import current_stream

_declared = False
SIG_FWD_DISPATCH, SIG_FWD_COMBINE, SIG_BWD_DISPATCH, SIG_BWD_COMBINE = range(4)
# Average rows per expert up to which the weight-streaming GEMM is the faster one.  It is up to about 110 rows in a group (8
# groups, N x K = 28672 x 4096, 100 rows: 325 us against 373), but a router spreads the tokens of a batch unevenly and a group
# beyond 128 reads its weights twice.  Where its tiles of 128 columns do not occupy the chip and each is split over a cluster,
# the reduction grows with the rows (16 groups, 1024 x 2048: 24 us against 23 with 24 rows, 30 against 24 with 64).
FEW_ROWS, FEW_ROWS_SPLIT, FEW_TILES = 80, 32, 148


class PlanDev(C.Structure):
    """Mirror of MoePlanDev."""
    _fields_ = [("P", C.c_int), ("E", C.c_int), ("me", C.c_int), ("cap", C.c_int), ("base_me", C.c_void_p),
                ("src_start", C.c_void_p), ("recv_count", C.c_void_p), ("expect_from", C.c_void_p), ("send_to", C.c_void_p),
                ("dropped", C.c_void_p), ("arrive_sig", C.c_void_p)]


def moe_lib() -> C.CDLL:
    global _declared
    lib = _native.load("libbshmem_moe.so")
    if not _declared:
        VP, I = C.c_void_p, C.c_int
        PS, PP = C.POINTER(DevState), C.POINTER(PlanDev)

        def f(name, *args, res=I):
            fn = getattr(lib, name)
            fn.restype, fn.argtypes = res, list(args)
        f("bshmem_moe_last_error", res=C.c_char_p)
        f("bshmem_moe_gemm_last_error", res=C.c_char_p)
        f("bshmem_moe_router_topk", VP, VP, I, I, I, I, VP, VP, VP, VP)
        f("bshmem_moe_plan", VP, I, I, VP, VP, VP)
        f("bshmem_moe_offsets", PP, VP, I, VP)
        f("bshmem_moe_plan_local", PP, VP, I, VP, VP, VP, VP, I, VP)
        f("bshmem_moe_dispatch_local", PP, VP, VP, VP, I, I, I, VP, VP)
        f("bshmem_moe_dispatch_grad_local", PP, VP, VP, VP, VP, I, I, I, VP, VP, VP, VP, VP)
        f("bshmem_moe_combine_local", PP, VP, VP, VP, VP, I, I, I, VP, VP, VP)
        f("bshmem_moe_dispatch", PS, PP, VP, VP, VP, VP, I, I, I, VP, VP, I, I, I, VP)
        f("bshmem_moe_wait_arrivals", PP, I, I, VP, I, VP, VP)
        f("bshmem_moe_combine_send", PS, PP, VP, VP, I, VP, I, I, I, VP)
        f("bshmem_moe_combine_reduce", PP, VP, VP, VP, VP, I, I, I, VP, VP)
        f("bshmem_moe_router_weight_grad", PP, VP, VP, VP, VP, I, I, I, VP, VP)
        f("bshmem_moe_router_backward", VP, VP, VP, VP, I, I, I, I, VP, VP, VP, VP)
        f("bshmem_moe_combine_reduce_router", PP, VP, VP, VP, I, I, I, VP, VP, VP, VP)
        f("bshmem_moe_swiglu_fwd", VP, VP, I, I, I, VP, VP)
        f("bshmem_moe_swiglu_bwd", VP, VP, VP, I, I, I, VP, VP)
        f("bshmem_moe_transpose_pad", VP, VP, I, I, I, VP, VP)
        f("bshmem_moe_grouped_gemm", VP, VP, VP, I, I, I, I, I, I, I, I, VP, I, VP, I, VP, VP, I, VP, I, I)
        f("bshmem_moe_grouped_gemm_act", VP, VP, VP, VP, I, I, I, I, I, I, I, I, VP, VP, VP, I, VP, I, I)
        f("bshmem_moe_grouped_gemm_swiglu_bwd", VP, VP, VP, VP, I, I, I, I, I, I, I, I, VP, VP, VP, I, VP, I, I)
        f("bshmem_moe_grouped_gemm_few", VP, VP, VP, I, I, I, I, I, I, I, VP, I, I, I, VP, VP, I, VP, I)
        f("bshmem_moe_grouped_gemm_tn", VP, VP, VP, I, I, I, I, I, I, I, VP, VP, I, I, I)
        f("bshmem_moe_zero_pad_rows", VP, I, VP, I, VP, I, VP, I, VP, I, I, VP)
        f("bshmem_moe_gemm_error_site", I)
        f("bshmem_moe_gemm_error_word", res=VP)
        _declared = True
    return lib


class _Fast:
    """The library's entry points as plain callables of integers (see _native.fast), bound on first use."""

    def __getattr__(self, name):
        fn = _native.fast(moe_lib(), "bshmem_moe_" + name)
        setattr(self, name, fn)
        return fn


_fast = _Fast()
_stream = current_stream


def _p(t: Optional[torch.Tensor]) -> int:
    return 0 if t is None else t.data_ptr()


def interleave_gate_up(w1: torch.Tensor, w3: torch.Tensor) -> torch.Tensor:
    """[F, H] gate and [F, H] up weights → [2F, H] with 32 gate rows followed by the matching 32 up rows,
    the layout the gated epilogue and the SwiGLU kernels expect."""
    F, H = w1.shape
    assert F % 32 == 0 and w3.shape == w1.shape
    return torch.stack((w1.view(F // 32, 32, H), w3.view(F // 32, 32, H)), dim=1).reshape(2 * F, H).contiguous()


def grouped_gemm(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor, groups: int, *, rows: Optional[torch.Tensor] = None,
                 fixed_rows: int = 0, klen: Optional[torch.Tensor] = None, gated: bool = False, arrive=None, expected=None,
                 n_arrive: int = 0, timeout_ms: int = 4000, max_ctas: int = 0, few: Optional[tuple] = None, about_rows: int = 0) -> None:
    """out_g = a_g @ b_g.T per group on the tcgen05 grouped kernel.  a: [G*Ra, K], b: [G*Rb, K], out: [G*Ra, N or N/2].
    `few` = (most rows of a group, most groups with rows): the caller expects about 100 rows per group or less; the
    weight-streaming form takes such problems.  The two numbers set its launch shape; a call whose counts exceed them is
    slower and as right.  `about_rows`: about how many rows a group has, where `rows` says it on the device only (0: not
    known); it sets the width of the tiles, and any counts are right."""
    G = groups
    ra, rb = a.shape[0] // G, b.shape[0] // G
    if few is not None and rows is not None and G <= 64:
        st = _fast.grouped_gemm_few(a.data_ptr(), b.data_ptr(), out.data_ptr(), G, ra, rb, a.shape[1], a.stride(0), b.stride(0),
                                    out.stride(0), rows.data_ptr(), few[0], few[1], 1 if gated else 0, arrive, _p(expected), n_arrive,
                                    _stream(), timeout_ms)
        if st != 0:
            raise RuntimeError(f"grouped gemm failed ({st}): {moe_lib().bshmem_moe_gemm_last_error().decode()}")
        return
    st = _fast.grouped_gemm(a.data_ptr(), b.data_ptr(), out.data_ptr(), G, ra, rb, rb, a.shape[1], a.stride(0), b.stride(0), out.stride(0),
                            _p(rows), about_rows if rows is not None else fixed_rows, _p(klen), 1 if gated else 0, arrive, _p(expected), n_arrive, _stream(), timeout_ms,
                            max_ctas)
    if st != 0:
        raise RuntimeError(f"grouped gemm failed ({st}): {moe_lib().bshmem_moe_gemm_last_error().decode()}")


def _check_matrices(what: str, **matrices) -> None:
    """Name = (tensor, rows, columns): bf16 matrices of that size with contiguous rows (the kernels get addresses only)."""
    for name, (t, rows, cols) in matrices.items():
        if t.dtype is not torch.bfloat16 or t.shape != (rows, cols) or t.stride(1) != 1:
            raise ValueError(f"{what}: {name} must be a bf16 [{rows}, {cols}] matrix with contiguous rows, got {t.dtype} {tuple(t.shape)}")


def grouped_gemm_act(a: torch.Tensor, b: torch.Tensor, gu: torch.Tensor, act: torch.Tensor, groups: int, *,
                     rows: Optional[torch.Tensor] = None, arrive=None, expected=None, n_arrive: int = 0, timeout_ms: int = 4000,
                     about_rows: int = 0) -> None:
    """Training forward of the gated MLP in one kernel: gu_g = a_g @ b_g.T (interleaved gate / up pre-activations, kept for
    the backward pass) and act_g = silu(gate) * up.  a: [G*R, K], b: [G*N, K], gu: [G*R, N], act: [G*R, N/2]."""
    G = groups
    R, K, N = a.shape[0], a.shape[1], b.shape[0] // G
    _check_matrices("grouped_gemm_act", a=(a, R, K), b=(b, G * N, K), gu=(gu, R, N), act=(act, R, N // 2))
    st = _fast.grouped_gemm_act(a.data_ptr(), b.data_ptr(), gu.data_ptr(), act.data_ptr(), G, a.shape[0] // G, b.shape[0] // G, a.shape[1],
                                a.stride(0), b.stride(0), gu.stride(0), act.stride(0), _p(rows), arrive, _p(expected), n_arrive, _stream(),
                                timeout_ms, about_rows)
    if st != 0:
        raise RuntimeError(f"grouped gemm (act) failed ({st}): {moe_lib().bshmem_moe_gemm_last_error().decode()}")


def grouped_gemm_swiglu_bwd(dy: torch.Tensor, w2_t: torch.Tensor, gu: torch.Tensor, dgu: torch.Tensor, groups: int, *,
                            rows: Optional[torch.Tensor] = None, arrive=None, expected=None, n_arrive: int = 0,
                            timeout_ms: int = 4000, about_rows: int = 0) -> None:
    """d_gu_g = SwiGLU backward of (dy_g @ w2_t_g.T) at the pre-activations gu_g, in one kernel: the gradient of the
    activations never goes to memory.  dy: [G*R, K], w2_t: [G*N, K], gu and dgu: [G*R, 2N] (interleaved)."""
    G = groups
    R, K, N = dy.shape[0], dy.shape[1], w2_t.shape[0] // G
    _check_matrices("grouped_gemm_swiglu_bwd", dy=(dy, R, K), w2_t=(w2_t, G * N, K), gu=(gu, R, 2 * N), dgu=(dgu, R, 2 * N))
    st = _fast.grouped_gemm_swiglu_bwd(dy.data_ptr(), w2_t.data_ptr(), gu.data_ptr(), dgu.data_ptr(), G, dy.shape[0] // G,
                                       w2_t.shape[0] // G, dy.shape[1], dy.stride(0), w2_t.stride(0), gu.stride(0), dgu.stride(0), _p(rows),
                                       arrive, _p(expected), n_arrive, _stream(), timeout_ms, about_rows)
    if st != 0:
        raise RuntimeError(f"grouped gemm (swiglu) failed ({st}): {moe_lib().bshmem_moe_gemm_last_error().decode()}")


def grouped_gemm_tn(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor, groups: int, counts: torch.Tensor, *,
                    timeout_ms: int = 4000, max_ctas: int = 0, about_rows: int = 0) -> None:
    """out_g[M, N] = a_g.T @ b_g per group with token-major operands a: [G*cap, M], b: [G*cap, N] and
    `counts[g]` tokens per group; both operands go to the tensor core MN-major, no transpose is materialised.
    Token rows [counts[g], next multiple of 64) of a and b must be zero (see zero_pad_rows).  `about_rows` as in grouped_gemm."""
    G = groups
    cap = a.shape[0] // G
    st = _fast.grouped_gemm_tn(a.data_ptr(), b.data_ptr(), out.data_ptr(), G, cap, a.shape[1], b.shape[1], a.stride(0), b.stride(0),
                               out.stride(0), counts.data_ptr(), _stream(), timeout_ms, max_ctas, about_rows)
    if st != 0:
        raise RuntimeError(f"grouped gemm (tn) failed ({st}): {moe_lib().bshmem_moe_gemm_last_error().decode()}")


def zero_pad_rows(buf, groups: int, counts: torch.Tensor) -> None:
    """Zero rows [counts[g], next multiple of 64) of every group of a contiguous [G*cap, cols] bf16 buffer, or of up to four
    buffers with the same number of rows in one launch."""
    bufs = [buf] if isinstance(buf, torch.Tensor) else list(buf)
    rows = bufs[0].shape[0]
    assert all(b.is_contiguous() and b.shape[0] == rows for b in bufs)
    args = [v for b in bufs for v in (b.data_ptr(), b.shape[1])] + [0, 0] * (4 - len(bufs))
    st = _fast.zero_pad_rows(*args, counts.data_ptr(), groups, rows // groups, _stream())
    if st != 0:
        raise RuntimeError(f"zero_pad_rows failed ({st}): {moe_lib().bshmem_moe_gemm_last_error().decode()}")


def few_bounds(P: int, G: int, cap: int, tokens: int, topk: int, max_tokens: int) -> tuple:
    """(most rows a group of this PE can get, most of its G groups that can get any).  A token sends at most one row to a
    group.  One PE knows the call's tokens; with several, the others may bring up to the layer's limit, whatever this one brings."""
    if P == 1:
        return min(cap, tokens), min(G, tokens * topk)
    return min(cap, P * max_tokens), G


class _Addresses:
    """Addresses of a layer's buffers by name, as they are at the moment of the call: a caller may put others in their place."""

    __slots__ = ("_of",)

    def __init__(self, of):
        self._of = of

    def __getitem__(self, name: str) -> int:
        return getattr(self._of, name).data_ptr()


class MoELayer:
    """One MoE block: y[T, H] = combine(experts(dispatch(x)))  with forward and backward.

    Weights per local expert: `w13` [G, 2F, H] (interleaved gate/up, see interleave_gate_up), `w2` [G, H, F];
    router `wr` [E, H].  Transposed copies used by the backward data-gradient GEMMs are kept in sync by
    `sync_transposes()` (all operands of the tcgen05 kernels are K-major)."""

    def __init__(self, rt, hidden: int, ffn: int, n_experts: int, topk: int, max_tokens: int, capacity_factor: float = 1.25,
                 training: bool = True, timeout_ms: int = 4000, tn_gemm: bool = True):
        self.tn_gemm = tn_gemm          # weight gradients on MN-major operands (False: explicit transposes)
        self.rt, self.H, self.F, self.E, self.topk, self.T = rt, hidden, ffn, n_experts, topk, max_tokens
        self.lib = moe_lib()
        P = rt.n_pes
        assert n_experts % P == 0 and hidden % 256 == 0 and ffn % 256 == 0
        self.P, self.G = P, n_experts // P
        cap = int(max_tokens * topk * P / n_experts * capacity_factor)
        self.cap = (cap + 255) // 256 * 256
        self.training, self.timeout_ms = training, timeout_ms
        dev, bf = rt.device, torch.bfloat16
        G, cap, H, F, T = self.G, self.cap, hidden, ffn, max_tokens
        n_entries = T * topk
        # ---- weights (random init by the caller) ----
        self.wr = torch.empty((n_experts, H), dtype=bf, device=dev)
        self.w13 = torch.empty((G, 2 * F, H), dtype=bf, device=dev)
        self.w2 = torch.empty((G, H, F), dtype=bf, device=dev)
        # ---- routing state ----
        self.topk_idx = torch.empty((n_entries,), dtype=torch.int32, device=dev)
        self.topk_w = torch.empty((n_entries,), dtype=torch.float32, device=dev)
        self.pos = torch.empty((n_entries,), dtype=torch.int32, device=dev)
        self.counts = rt.zeros((n_experts,), torch.int32)                     # symmetric: gathered below
        self.counts_all = rt.zeros((P * n_experts,), torch.int32)
        self.base_me = torch.zeros((n_experts,), dtype=torch.int32, device=dev)
        self.src_start = torch.zeros((G * (P + 1),), dtype=torch.int32, device=dev)
        self.recv_count = torch.zeros((G,), dtype=torch.int32, device=dev)
        self.expect_from = torch.zeros((P,), dtype=torch.int32, device=dev)
        self.send_to = torch.zeros((P,), dtype=torch.int32, device=dev)
        self.dropped = torch.zeros((1,), dtype=torch.int32, device=dev)
        self.arrive = rt.zeros((2 * 4 * P,), torch.int64)
        # ---- symmetric data buffers ----
        self.recv = rt.empty((G * cap, H), bf, align=1024)                    # dispatched tokens (kept for dW13 in training)
        self.meta = rt.empty((G * cap,), torch.int32)
        self.ybuf = rt.empty((n_entries, H), bf, align=1024)                  # expert outputs per entry, back at the source
        # ---- expert-side activations ----
        self.gu = torch.empty((G * cap, 2 * F), dtype=bf, device=dev)
        self.hact = torch.empty((G * cap, F), dtype=bf, device=dev)
        self.yexp = torch.empty((G * cap, H), dtype=bf, device=dev)
        self.out = torch.empty((T, H), dtype=bf, device=dev)
        if training:
            # the backward pass dispatches gradients into a receive buffer of its own, so the forward's dispatched
            # inputs stay where they landed until dW13 has read them (no copy)
            self.recv_bwd = rt.empty((G * cap, H), bf, align=1024)
            self.xsave = self.recv
            self.w13_t = torch.empty((G, H, 2 * F), dtype=bf, device=dev)
            self.w2_t = torch.empty((G, F, H), dtype=bf, device=dev)
            self.dh = torch.empty((G * cap, F), dtype=bf, device=dev)             # used where experts have few rows
            self.dgu = torch.empty((G * cap, 2 * F), dtype=bf, device=dev)
            self.dxe = torch.empty((G * cap, H), dtype=bf, device=dev)
            if not tn_gemm:
                self.t_a = torch.empty((G * 2 * F * cap,), dtype=bf, device=dev)  # transposed operands, reused
                self.t_b = torch.empty((G * max(F, H) * cap,), dtype=bf, device=dev)
            self.dw13 = torch.empty((G, 2 * F, H), dtype=bf, device=dev)
            self.dw2 = torch.empty((G, H, F), dtype=bf, device=dev)
            self.dxbuf = rt.empty((n_entries, H), bf, align=1024)
            self.dx = torch.empty((T, H), dtype=bf, device=dev)
            self.dtopk_w = torch.empty((n_entries,), dtype=torch.float32, device=dev)
            self.dlogit = torch.empty((n_entries,), dtype=torch.float32, device=dev)   # gradient of the chosen experts' logits
            self.dwr_f32 = torch.empty((n_experts, H), dtype=torch.float32, device=dev)
            self.dwr = torch.empty((n_experts, H), dtype=bf, device=dev)             # router weight gradient
            self._x_in = None
        self.plan = PlanDev(P=P, E=n_experts, me=rt.my_pe, cap=self.cap, base_me=self.base_me.data_ptr(),
                            src_start=self.src_start.data_ptr(), recv_count=self.recv_count.data_ptr(),
                            expect_from=self.expect_from.data_ptr(), send_to=self.send_to.data_ptr(),
                            dropped=self.dropped.data_ptr(), arrive_sig=self.arrive.data_ptr())
        self.state = rt.device_state()
        self.ticket = torch.zeros((1,), dtype=torch.int32, device=dev)        # of the one-PE plan kernel
        self._plan_a, self._state_a = C.addressof(self.plan), C.addressof(self.state)
        self.err_word = self.lib.bshmem_moe_gemm_error_word()
        self.calls = 0
        self.launches = 0
        self.ctas = 128
        rt.barrier_all()

    # ------------------------------------------------------------------------------------
    def sync_transposes(self) -> None:
        """Refresh the transposed weight copies the backward data-gradient GEMMs read."""
        if self.training:
            self.w13_t.copy_(self.w13.transpose(1, 2))
            self.w2_t.copy_(self.w2.transpose(1, 2))

    def _chk(self, st: int, what: str) -> None:
        if st != 0:
            raise RuntimeError(f"{what} failed ({st}): {self.lib.bshmem_moe_last_error().decode()}")
        self.launches += 1

    def _sig_ptr(self, parity: int, which: int) -> int:
        return self.arrive.data_ptr() + 8 * (parity * 4 * self.P + which * self.P)

    def route(self, x: torch.Tensor) -> None:
        """Router, plan, count exchange and offsets for this call's tokens."""
        T, s, a = x.shape[0], _stream(), _Addresses(self)
        n_entries = T * self.topk
        self.calls += 1
        self.parity = self.calls & 1
        self._chk(_fast.router_topk(x.data_ptr(), self.wr.data_ptr(), T, self.H, self.E, self.topk, a["topk_idx"], a["topk_w"], 0, s), "router")
        if self.P == 1:
            self._chk(_fast.plan_local(self._plan_a, a["topk_idx"], n_entries, a["pos"], a["counts"], a["counts_all"], a["ticket"],
                                       self.parity, s), "plan")
            return
        self._chk(_fast.plan(a["topk_idx"], n_entries, self.E, a["pos"], a["counts"], s), "plan")
        self.rt.fcollect(self.counts_all, self.counts)            # all-gather of the per-expert counts (device collective)
        self.launches += 1
        self._chk(_fast.offsets(self._plan_a, a["counts_all"], self.parity, s), "offsets")

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        T, s, a = x.shape[0], _stream(), _Addresses(self)
        n_entries = T * self.topk
        G, cap, H, F, P = self.G, self.cap, self.H, self.F, self.P
        local = P == 1                                             # no row leaves this GPU: no signals, no return buffer
        bounds = few_bounds(P, G, cap, T, self.topk, self.T)

        def few(cols):
            """The bounds if the product with `cols` columns is one for the weight-streaming GEMM, else None.  The choice goes by
            the expected rows (every PE brings about as many tokens)."""
            limit = FEW_ROWS if G * cols // 128 > FEW_TILES else FEW_ROWS_SPLIT
            return bounds if P * n_entries <= limit * self.E else None

        few_up, few_down = few(2 * F), few(H)
        about = max(1, P * n_entries // self.E)                    # rows of an expert
        self.route(x)
        par = self.parity
        if local:
            self._chk(_fast.dispatch_local(self._plan_a, x.data_ptr(), a["topk_idx"], a["pos"], T, self.topk, H, a["recv"], s), "dispatch")
            wait = {}
        else:
            self._chk(_fast.dispatch(self._state_a, self._plan_a, x.data_ptr(), 0, a["topk_idx"], a["pos"], n_entries, self.topk, H,
                                     a["recv"], a["meta"], par, SIG_FWD_DISPATCH, self.ctas, s), "dispatch")
            wait = dict(arrive=self._sig_ptr(par, SIG_FWD_DISPATCH), expected=self.expect_from, n_arrive=P)
        # gate/up projection (waits on the arrival words inside the kernel), then SwiGLU, then down projection
        if self.training:
            if few_up is None:
                grouped_gemm_act(self.recv, self.w13.view(G * 2 * F, H), self.gu, self.hact, G, rows=self.recv_count,
                                 timeout_ms=self.timeout_ms, about_rows=about, **wait)
            else:
                grouped_gemm(self.recv, self.w13.view(G * 2 * F, H), self.gu, G, rows=self.recv_count, timeout_ms=self.timeout_ms,
                             few=few_up, about_rows=about, **wait)
                self._chk(_fast.swiglu_fwd(a["gu"], a["recv_count"], G, cap, F, a["hact"], s), "swiglu")
            self._x_in = x                                         # the router's backward needs the layer input
            self._few_h, self._few_x = few(F), few_down
        else:
            grouped_gemm(self.recv, self.w13.view(G * 2 * F, H), self.hact, G, rows=self.recv_count, gated=True,
                         timeout_ms=self.timeout_ms, few=few_up, about_rows=about, **wait)
        self.launches += 1
        grouped_gemm(self.hact, self.w2.view(G * H, F), self.yexp, G, rows=self.recv_count, timeout_ms=self.timeout_ms, few=few_down,
                     about_rows=about)
        self.launches += 1
        if local:
            self._chk(_fast.combine_local(self._plan_a, a["yexp"], a["topk_w"], a["topk_idx"], a["pos"], T, self.topk, H, a["out"], 0, s),
                      "combine")
            return self.out[:T]
        self._chk(_fast.combine_send(self._state_a, self._plan_a, a["yexp"], a["meta"], H, a["ybuf"], par, SIG_FWD_COMBINE, self.ctas, s),
                  "combine_send")
        self._chk(_fast.wait_arrivals(self._plan_a, par, SIG_FWD_COMBINE, a["send_to"], self.timeout_ms, self.err_word, s), "wait")
        self._chk(_fast.combine_reduce(self._plan_a, a["ybuf"], a["topk_w"], a["topk_idx"], a["pos"], T, self.topk, H, a["out"], s),
                  "combine_reduce")
        return self.out[:T]

    def backward(self, dout: torch.Tensor) -> torch.Tensor:
        """Gradients w.r.t. the layer input (returned; expert path and router path), the expert weights (self.dw13,
        self.dw2), the routing weights (self.dtopk_w) and, through the softmax over the chosen experts, the router
        weights (self.dwr).  Must follow forward() of the same tokens; the forward's input must still be intact."""
        assert self.training
        T, s, a = dout.shape[0], _stream(), _Addresses(self)
        n_entries = T * self.topk
        G, cap, H, F, P = self.G, self.cap, self.H, self.F, self.P
        local = P == 1
        par = self.parity
        rc = self.recv_count
        dy = self.recv_bwd
        about = max(1, P * n_entries // self.E)                    # rows of an expert
        if local:
            # w * d_out into the experts' gradient buffers, and in the same pass the gradients of the routing weights and of
            # the chosen experts' logits
            self._chk(_fast.dispatch_grad_local(self._plan_a, dout.data_ptr(), a["topk_idx"], a["pos"], a["topk_w"], T, self.topk, H,
                                                a["recv_bwd"], a["yexp"], a["dtopk_w"], a["dlogit"], s), "dispatch(bwd)")
            self._chk(_fast.router_backward(self._x_in.data_ptr(), a["topk_idx"], 0, 0, T, H, self.E, self.topk, a["dlogit"], a["dwr_f32"],
                                            a["dwr"], s), "router backward")
            self.launches += 1
            wait = {}
        else:
            self._chk(_fast.router_weight_grad(self._plan_a, a["ybuf"], dout.data_ptr(), a["topk_idx"], a["pos"], n_entries, self.topk, H,
                                               a["dtopk_w"], s), "router weight grad")
            # router backward: d_logits of the chosen experts and d_Wr = d_logits^T · x
            self._chk(_fast.router_backward(self._x_in.data_ptr(), a["topk_idx"], a["topk_w"], a["dtopk_w"], T, H, self.E, self.topk,
                                            a["dlogit"], a["dwr_f32"], a["dwr"], s), "router backward")
            self.launches += 2
            # combine-backward = dispatch of w * d_out into the experts' gradient receive buffers (same slots as forward)
            self._chk(_fast.dispatch(self._state_a, self._plan_a, dout.data_ptr(), a["topk_w"], a["topk_idx"], a["pos"], n_entries, self.topk,
                                     H, a["recv_bwd"], 0, par, SIG_BWD_DISPATCH, self.ctas, s), "dispatch(bwd)")
            wait = dict(arrive=self._sig_ptr(par, SIG_BWD_DISPATCH), expected=self.expect_from, n_arrive=P)
        # d_hact = d_y · W2 (B operand = W2^T [F, H], K = H) and through SwiGLU to d_gu
        if self._few_h is None:
            grouped_gemm_swiglu_bwd(dy, self.w2_t.view(G * F, H), self.gu, self.dgu, G, rows=rc, timeout_ms=self.timeout_ms,
                                    about_rows=about, **wait)
        else:
            grouped_gemm(dy, self.w2_t.view(G * F, H), self.dh, G, rows=rc, timeout_ms=self.timeout_ms, few=self._few_h,
                         about_rows=about, **wait)
            self._chk(_fast.swiglu_bwd(a["gu"], a["dh"], rc.data_ptr(), G, cap, F, a["dgu"], s), "swiglu bwd")
        # dW2 = d_y^T · hact: token-major operands straight into the MN-major tensor-core path
        if self.tn_gemm:
            zero_pad_rows((dy, self.hact, self.dgu, self.xsave), G, rc)
            grouped_gemm_tn(dy, self.hact, self.dw2.view(G * H, F), G, rc, timeout_ms=self.timeout_ms, about_rows=about)
        else:                          # explicit transposes + ragged-K K-major GEMM
            ta = self.t_a[: G * H * cap].view(G * H, cap)
            tb = self.t_b[: G * F * cap].view(G * F, cap)
            self._chk(_fast.transpose_pad(dy.data_ptr(), rc.data_ptr(), G, cap, H, ta.data_ptr(), s), "transpose")
            self._chk(_fast.transpose_pad(a["hact"], rc.data_ptr(), G, cap, F, tb.data_ptr(), s), "transpose")
            grouped_gemm(ta, tb, self.dw2.view(G * H, F), G, fixed_rows=H, klen=rc, timeout_ms=self.timeout_ms)
        # dW13 = d_gu^T · x and d_x = d_gu · W13
        if self.tn_gemm:
            grouped_gemm_tn(self.dgu, self.xsave, self.dw13.view(G * 2 * F, H), G, rc, timeout_ms=self.timeout_ms, about_rows=about)
        else:
            ta2 = self.t_a[: G * 2 * F * cap].view(G * 2 * F, cap)
            tb2 = self.t_b[: G * H * cap].view(G * H, cap)
            self._chk(_fast.transpose_pad(a["dgu"], rc.data_ptr(), G, cap, 2 * F, ta2.data_ptr(), s), "transpose")
            self._chk(_fast.transpose_pad(self.xsave.data_ptr(), rc.data_ptr(), G, cap, H, tb2.data_ptr(), s), "transpose")
            grouped_gemm(ta2, tb2, self.dw13.view(G * 2 * F, H), G, fixed_rows=2 * F, klen=rc, timeout_ms=self.timeout_ms)
        grouped_gemm(self.dgu, self.w13_t.view(G * H, 2 * F), self.dxe, G, rows=rc, timeout_ms=self.timeout_ms, few=self._few_x,
                     about_rows=about)
        self.launches += 4
        if local:
            # d_x = sum over k of the experts' rows + the router path (d_logits · Wr), written once
            self._chk(_fast.combine_local(self._plan_a, a["dxe"], a["dlogit"], a["topk_idx"], a["pos"], T, self.topk, H, a["dx"], self.wr.data_ptr(), s),
                      "combine(bwd)")
            return self.dx[:T]
        # dispatch-backward = combine of the d_x rows back to their source entries, summed over k
        self._chk(_fast.combine_send(self._state_a, self._plan_a, a["dxe"], a["meta"], H, a["dxbuf"], par, SIG_BWD_COMBINE, self.ctas, s),
                  "combine_send(bwd)")
        self._chk(_fast.wait_arrivals(self._plan_a, par, SIG_BWD_COMBINE, a["send_to"], self.timeout_ms, self.err_word, s), "wait")
        # d_x = sum over k of the returned rows + the router path (d_logits · Wr), written once
        self._chk(_fast.combine_reduce_router(self._plan_a, a["dxbuf"], a["topk_idx"], a["pos"], T, self.topk, H, a["dx"], a["dlogit"],
                                              self.wr.data_ptr(), s), "combine_reduce(bwd)")
        return self.dx[:T]

    def check(self) -> None:
        site = self.lib.bshmem_moe_gemm_error_site(1)
        if site:
            raise RuntimeError(f"moe: a bounded in-kernel wait ran out (site {site})")
        if int(self.dropped.item()):
            raise RuntimeError(f"moe: {int(self.dropped.item())} rows exceeded the expert capacity {self.cap}")
