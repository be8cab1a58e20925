"""Performance cases of roc_shmem_b200 on one GPU: the calls a program makes, from a one-word message to a full
mixture-of-experts training step.

``listed()`` names twelve cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` builds what a program
holds before the call (its PE, buffers, layers, weights), ``run`` is one pass through the public entry points, ``work``
is what the pass cannot do without and ``tolerance`` how far two correct implementations may lie apart.

Kinds of case and what each stands for:

  window        a host thread fills a window of 64 non-blocking puts (or gets) on a context and waits for it
  signal        request / reply of a host thread: fetch-add, put with signal, wait on the signal, read a word
  device_copy   device-initiated put / get of one message, striped over the GPU
  collective    a collective over the PEs of a local group (all PEs on this GPU)
  linear        forward of a (tensor-parallel) linear layer on bf16: decode with few tokens, prefill with many
  linear_train  forward and both gradients of a bf16 linear layer through autograd
  linear_fp8    activations quantised on the fly, times a weight that is kept in block-scaled fp8
  mlp           gated MLP block (one rank's share of a tensor-parallel Llama block), inference or forward + backward
  moe           mixture-of-experts block, inference (decode and prefill) or forward + backward
"""
from __future__ import annotations

import math
import weakref

import torch

import roc_shmem_b200 as shmem
from roc_shmem_b200 import gpu
from roc_shmem_b200.models import LlamaMLP, MixtralMoEBlock
from roc_shmem_b200.ops.gemm_fp8 import gemm_fp8, quantize_act, quantize_weight
from roc_shmem_b200.ops.torch_ops import Linear
from roc_shmem_b200.parallel.tp import RowParallelLinear
from roc_shmem_b200.utils import dtypes as D

WINDOW = 64
HEAP_BYTES = 16 << 30            # symmetric heap of the program's PE
GROUP_HEAP_BYTES = 1 << 30       # symmetric heap of each PE of a local group

# (in features, out features) of linear layers: shards of the 70B Llama MLP at eight ranks, Mixtral's expert matrices,
# and the square problems of the GEMM benchmark
LINEAR_SHAPES = [(3584, 8192), (8192, 7168), (4096, 4096), (8192, 8192), (4096, 14336), (14336, 4096), (2048, 2048)]
# (hidden, ffn of this rank)
MLP_SHAPES = [(8192, 3584), (8192, 7168), (4096, 3584), (2048, 4096)]
# (hidden, ffn, experts, top-k)
MOE_SHAPES = [(4096, 14336, 8, 2), (2048, 4096, 8, 2), (2048, 1024, 64, 8), (1024, 2048, 16, 2)]


def listed() -> list[dict]:
    return [
        # message-rate loop of a communication library: 64 small puts in flight, then quiet
        {"name": "put window 64 B", "kind": "window", "get": False, "nbytes": 64},
        # a control message between two services: counter, payload with flag, wait, read back
        {"name": "signalled message 4 KiB", "kind": "signal", "nbytes": 4096},
        # bulk transfer started from the device (parameter or KV-cache block), size not a power of two
        {"name": "device get 96 MB", "kind": "device_copy", "get": True, "scope": "bulk", "nbytes": 96_000_000},
        # a latency-bound allreduce: gradient norms, routing counts, small tensors
        {"name": "allreduce fp32 16 KiB", "kind": "collective", "op": "allreduce", "pes": 4, "dtype": "float32",
         "nbytes": 16384, "ctas": 1},
        # a bandwidth-bound gradient bucket
        {"name": "reduce-scatter bf16 32 MiB", "kind": "collective", "op": "reduce_scatter", "pes": 8, "dtype": "bfloat16",
         "nbytes": 32 << 20, "ctas": 16},
        # decode step of a serving engine: a batch of 16 sequences through the down-projection shard
        {"name": "linear decode 16", "kind": "linear", "tokens": 16, "k": 3584, "n": 8192},
        # prefill / training forward of the same layer at the benchmark's size
        {"name": "linear prefill 8192", "kind": "linear", "tokens": 8192, "k": 3584, "n": 8192},
        # fine-tuning on a packed batch whose token count is no multiple of a tile
        {"name": "linear train 1000", "kind": "linear_train", "tokens": 1000, "k": 8192, "n": 7168},
        # fp8 serving of the gate + up shard
        {"name": "linear fp8 4096", "kind": "linear_fp8", "tokens": 4096, "k": 8192, "n": 7168},
        # training step of one rank's MLP block
        {"name": "mlp train 8192", "kind": "mlp", "tokens": 8192, "hidden": 8192, "ffn": 3584, "train": True},
        # decode step of a Mixtral-style layer
        {"name": "moe decode 32", "kind": "moe", "tokens": 32, "max_tokens": 64, "hidden": 4096, "ffn": 14336, "experts": 8,
         "topk": 2, "train": False},
        # training step of the same layer at the benchmark's size
        {"name": "moe train 16384", "kind": "moe", "tokens": 16384, "max_tokens": 16384, "hidden": 4096, "ffn": 14336,
         "experts": 8, "topk": 2, "train": True},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _linear_shape(rng) -> tuple[int, int]:
    if rng.random() < 0.6:
        return rng.choice(LINEAR_SHAPES)
    return 8 * rng.randint(64, 1024), 8 * rng.randint(64, 1024)


def draw(rng) -> dict:
    kind = rng.choice(["window", "signal", "device_copy", "collective", "linear", "linear", "linear_train", "linear_fp8", "mlp",
                       "moe", "moe"])
    if kind == "window":
        return {"kind": kind, "get": rng.random() < 0.4, "nbytes": _log_int(rng, 8, 262144)}
    if kind == "signal":
        return {"kind": kind, "nbytes": _log_int(rng, 8, 1 << 20)}
    if kind == "device_copy":
        scope = rng.choice(["bulk", "bulk", "block"])
        n = _log_int(rng, 65536, 256 << 20)
        return {"kind": kind, "get": rng.random() < 0.5, "scope": scope, "nbytes": n - n % 16 if scope == "bulk" else n}
    if kind == "collective":
        pes = rng.choice([2, 4, 8])
        dtype = rng.choice(["float32", "bfloat16", "int32"])
        nbytes = _log_int(rng, 1024, 64 << 20)
        nbytes -= nbytes % (16 * pes)
        ctas = max(1, min(128 // pes, nbytes >> 16))
        return {"kind": kind, "op": rng.choice(["allreduce", "allreduce", "reduce_scatter", "fcollect", "alltoall"]), "pes": pes,
                "dtype": dtype, "nbytes": nbytes, "ctas": ctas}
    if kind == "linear":
        k, n = _linear_shape(rng)
        return {"kind": kind, "tokens": _log_int(rng, 1, 8192), "k": k, "n": n}
    if kind == "linear_train":
        k, n = _linear_shape(rng)
        return {"kind": kind, "tokens": 8 * _log_int(rng, 8, 1024), "k": k, "n": n}
    if kind == "linear_fp8":
        k, n = rng.choice(LINEAR_SHAPES)
        return {"kind": kind, "tokens": 128 * _log_int(rng, 1, 64), "k": k, "n": n}
    if kind == "mlp":
        hidden, ffn = rng.choice(MLP_SHAPES)
        return {"kind": kind, "tokens": 256 * _log_int(rng, 1, 32), "hidden": hidden, "ffn": ffn, "train": rng.random() < 0.6}
    hidden, ffn, experts, topk = rng.choice(MOE_SHAPES)
    train = rng.random() < 0.5
    tokens = _log_int(rng, 256 if train else 1, 16384)
    # a serving layer is built for the largest batch of its tier; a training layer for the step's own token count
    top = tokens if train else next(m for m in (64, 1024, 16384) if tokens <= m)
    return {"kind": kind, "tokens": tokens, "max_tokens": top, "hidden": hidden, "ffn": ffn, "experts": experts, "topk": topk,
            "train": train}


# ---- the program around the calls -------------------------------------------------------------------------------
_programs: dict = {}


def _pe():
    """This process's PE: a program initialises the runtime once."""
    if "pe" not in _programs:
        _programs["pe"] = shmem.init("device", rank=0, world_size=1, heap_bytes=HEAP_BYTES)
    return _programs["pe"]


def _group(pes: int) -> gpu.LocalGroup:
    """The local group of `pes` PEs: created once as well."""
    if pes not in _programs:
        _programs[pes] = gpu.LocalGroup(pes, heap_bytes=GROUP_HEAP_BYTES)
    return _programs[pes]


class _Symmetric:
    """Symmetric tensors of one state; they go back to the heap with the state."""

    def __init__(self, owned):
        owned = [(rt, t) for rt, t in owned]
        self._release = weakref.finalize(self, _Symmetric._free, owned)

    @staticmethod
    def _free(owned):
        for rt, t in owned:
            if not rt.finalized:
                rt.free(t, collective=False)


def _layer_buffers(rt, before: set) -> _Symmetric:
    """What a layer's constructor allocated in the heap since `before`."""
    return _Symmetric([(rt, t) for p, t in rt._live.items() if p not in before])


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, shape, std=1.0, dtype=torch.bfloat16) -> torch.Tensor:
    t = torch.empty(shape, dtype=dtype, device="cuda")
    return t.normal_(0.0, std, generator=g)


def _bytes(g, n: int) -> torch.Tensor:
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=g)


def prepare(case: dict, seed: int) -> dict:
    kind, g = case["kind"], _generator(seed)
    st = {"case": case}
    if kind == "window":
        rt, n = _pe(), case["nbytes"]
        sym, local = rt.empty((WINDOW, n), torch.uint8), torch.empty((WINDOW, n), dtype=torch.uint8, device="cuda")
        src, dst = (sym, local) if case["get"] else (local, sym)
        src.copy_(_bytes(g, WINDOW * n).view(WINDOW, n))
        dst.zero_()
        if "ctx" not in _programs:
            _programs["ctx"] = rt.ctx_create(shmem.CTX_SERIALIZED)
        st.update(ctx=_programs["ctx"], pairs=list(zip(dst.unbind(0), src.unbind(0))), out=dst, owned=_Symmetric([(rt, sym)]))
    elif kind == "signal":
        rt, n = _pe(), case["nbytes"]
        box, flag, counter = rt.empty((n,), torch.uint8), rt.zeros((1,), torch.int64), rt.zeros((1,), torch.int64)
        counter.fill_(int(seed) % 1009)
        st.update(rt=rt, box=box, flag=flag, counter=counter, message=_bytes(g, n),
                  owned=_Symmetric([(rt, box), (rt, flag), (rt, counter)]))
    elif kind == "device_copy":
        rt, n = _pe(), case["nbytes"]
        sym, local = rt.empty((n,), torch.uint8), torch.empty(n, dtype=torch.uint8, device="cuda")
        src, dst = (sym, local) if case["get"] else (local, sym)
        src.copy_(_bytes(g, n))
        dst.zero_()
        st.update(rt=rt, sym=sym, local=local, out=dst, owned=_Symmetric([(rt, sym)]))
    elif kind == "collective":
        group, dt = _group(case["pes"]), getattr(torch, case["dtype"])
        elems = case["nbytes"] // (2 if dt == torch.bfloat16 else 4)
        out_elems = elems // case["pes"] if case["op"] == "reduce_scatter" else elems
        in_elems = elems // case["pes"] if case["op"] == "fcollect" else elems
        srcs, dsts = group.empty((in_elems,), dt), group.empty((out_elems,), dt)
        for s, d in zip(srcs, dsts):
            if dt == torch.int32:
                s.random_(-(1 << 20), 1 << 20, generator=g)
            else:
                s.normal_(generator=g)
            d.zero_()
        st.update(group=group, srcs=srcs, dsts=dsts, dtype=dt, owned=_Symmetric(list(zip(group.pes * 2, srcs + dsts))))
    elif kind == "linear":
        layer = RowParallelLinear(_pe(), case["k"], case["n"], case["tokens"])
        layer.weight.copy_(_normal(g, (case["n"], case["k"]), 0.02))
        st.update(layer=layer, x=_normal(g, (case["tokens"], case["k"])))
    elif kind == "linear_train":
        layer = Linear(case["k"], case["n"], device="cuda")
        with torch.no_grad():
            layer.weight.copy_(_normal(g, (case["n"], case["k"]), 0.02))
        st.update(layer=layer, x=_normal(g, (case["tokens"], case["k"])).requires_grad_(True),
                  dy=_normal(g, (case["tokens"], case["n"])))
    elif kind == "linear_fp8":
        st.update(w=quantize_weight(_normal(g, (case["n"], case["k"]), 0.02)), x=_normal(g, (case["tokens"], case["k"])),
                  out=torch.empty((case["tokens"], case["n"]), dtype=torch.bfloat16, device="cuda"))
    elif kind == "mlp":
        h, f, t = case["hidden"], case["ffn"], case["tokens"]
        block = LlamaMLP(_pe(), h, f, t, training=case["train"])
        block.load(_normal(g, (f, h), 0.02), _normal(g, (f, h), 0.02), _normal(g, (h, f), 0.02))
        st.update(block=block, x=_normal(g, (t, h)), dy=_normal(g, (t, h)) if case["train"] else None)
    elif kind == "moe":
        rt = _pe()
        h, f, e, t = case["hidden"], case["ffn"], case["experts"], case["tokens"]
        before = set(rt._live)
        block = MixtralMoEBlock(rt, h, f, e, case["topk"], case["max_tokens"], training=case["train"])
        st["owned"] = _layer_buffers(rt, before)
        # weights straight into the layer's own layout (gate and up rows interleaved in groups of 32)
        block.wr.copy_(_normal(g, (e, h), 0.02))
        block.w13.normal_(0.0, 0.02, generator=g)
        block.w2.normal_(0.0, 0.02, generator=g)
        block.sync_transposes()
        st.update(block=block, x=_normal(g, (t, h)), dy=_normal(g, (t, h)) if case["train"] else None)
    else:
        raise ValueError(f"unknown kind of case: {kind!r}")
    torch.cuda.synchronize()
    return st


_COLLECTIVES = {"allreduce": gpu.COLL_REDUCE, "reduce_scatter": gpu.COLL_REDUCE_SCATTER, "fcollect": gpu.COLL_FCOLLECT,
                "alltoall": gpu.COLL_ALLTOALL}


def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "window":
        ctx = st["ctx"]
        move = ctx.get if case["get"] else ctx.put
        for dst, src in st["pairs"]:
            move(dst, src, 0, nbi=True)
        ctx.quiet()
        return st["out"]
    if kind == "signal":
        rt, flag, counter = st["rt"], st["flag"], st["counter"]
        ticket = rt.atomic_fetch_add(counter, 1, 0) + 1
        rt.put_signal(st["box"], st["message"], flag, ticket, 0)
        rt.wait_until(flag, "ge", ticket)
        return {"box": st["box"], "flag": flag, "ticket": ticket, "count": rt.g(counter, 0)}
    if kind == "device_copy":
        st["rt"].rma_kernel(st["sym"], st["local"], 0, put=not case["get"], scope=case["scope"], ctas=132,
                            threads=128 if case["scope"] == "bulk" else 512)
        return st["out"]
    if kind == "collective":
        d, op = st["dsts"], case["op"]
        es = st["srcs"][0].element_size()
        # elements of a reduced vector (allreduce), of the result (reduce-scatter), bytes of a block (fcollect, alltoall)
        count = {"allreduce": d[0].numel(), "reduce_scatter": d[0].numel(), "fcollect": st["srcs"][0].numel() * es,
                 "alltoall": case["nbytes"] // case["pes"]}[op]
        st["group"].collective(_COLLECTIVES[op], d, st["srcs"], count, dtype=st["dtype"], op=D.SUM, ctas=case["ctas"])
        return d
    if kind == "linear":
        return st["layer"](st["x"])
    if kind == "linear_train":
        x, w = st["x"], st["layer"].weight
        y = st["layer"](x)
        dx, dw = torch.autograd.grad(y, (x, w), st["dy"])
        return {"y": y, "dx": dx, "dw": dw}
    if kind == "linear_fp8":
        return gemm_fp8(quantize_act(st["x"]), st["w"], st["out"])
    block = st["block"]
    y = block.forward(st["x"])
    if not case["train"]:
        return y
    dx = block.backward(st["dy"])
    out = {"y": y, "dx": dx, "dw13": block.dw13, "dw2": block.dw2}
    if kind == "moe":
        out["dwr"] = block.dwr
    return out


def work(case: dict) -> dict:
    """Bytes that have to be read or written and operations that have to be done; weights count once, and of a
    mixture's experts only as many as the tokens can reach."""
    kind = case["kind"]
    if kind == "window":
        return {"bytes": 2 * WINDOW * case["nbytes"], "flops": 0}
    if kind in ("signal", "device_copy"):
        return {"bytes": 2 * case["nbytes"], "flops": 0}
    if kind == "collective":
        n, p = case["nbytes"], case["pes"]
        es = 2 if case["dtype"] == "bfloat16" else 4
        src, dst = (n // p if case["op"] == "fcollect" else n), (n // p if case["op"] == "reduce_scatter" else n)
        adds = {"allreduce": 1, "reduce_scatter": 1}.get(case["op"], 0) * (p - 1) * (n // es)
        return {"bytes": p * (src + dst), "flops": adds}
    if kind.startswith("linear"):
        t, k, n = case["tokens"], case["k"], case["n"]
        if kind == "linear_fp8":
            return {"bytes": 2 * t * k + n * k + 2 * t * n, "flops": 2 * t * k * n}
        once = {"bytes": 2 * (t * k + n * k + t * n), "flops": 2 * t * k * n}
        if kind == "linear":
            return once
        # forward, plus dy in and both gradients out
        return {"bytes": once["bytes"] + 2 * (t * n + t * k + n * k), "flops": 3 * once["flops"]}
    t, h, f = case["tokens"], case["hidden"], case["ffn"]
    if kind == "mlp":
        weights, flops = 2 * 3 * h * f, 6 * t * h * f
        if not case["train"]:
            return {"bytes": weights + 4 * t * h, "flops": flops}
        return {"bytes": 2 * weights + 8 * t * h, "flops": 3 * flops}
    e, k = case["experts"], case["topk"]
    weights = 2 * 3 * h * f * min(e, t * k) + 2 * e * h
    flops = 6 * t * k * h * f + 2 * t * e * h
    if not case["train"]:
        return {"bytes": weights + 4 * t * h, "flops": flops}
    return {"bytes": 2 * (2 * 3 * h * f * e + 2 * e * h) + 8 * t * h, "flops": 3 * flops}


def tolerance(case: dict):
    """Copies are exact, 32-bit sums differ by their order, a bf16 result by its rounding, and a chain of bf16 steps (or
    a gradient behind one) by the rounding of every intermediate."""
    kind = case["kind"]
    if kind in ("window", "signal", "device_copy"):
        return "exact"
    if kind == "collective":
        if case["op"] in ("fcollect", "alltoall") or case["dtype"] == "int32":
            return "exact"
        return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 5e-3}
    if kind in ("linear", "linear_train", "linear_fp8"):
        return {"rel": 5e-3}
    return {"rel": 1e-2}
