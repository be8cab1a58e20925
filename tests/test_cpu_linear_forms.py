"""``Linear`` on anything but plain tensors in GPU memory is the registered operator: meta and fake tensors, transforms, tracing
and modes that watch operators, with an fp32 product in the kernel's place."""
import pytest
import torch


@pytest.fixture
def lin(monkeypatch):
    from roc_shmem_b200.ops import torch_ops

    def product(a, b, out=None, *, a_mn=False, b_mn=False):
        with torch.no_grad():
            return ((a.t() if a_mn else a).float() @ (b if b_mn else b.t()).float()).to(torch.bfloat16)
    monkeypatch.setattr(torch_ops, "gemm_bf16", product)
    return torch_ops.Linear(16, 24, device="cpu")


def _x(*shape):
    return torch.randn(*shape).to(torch.bfloat16)


def test_meta_and_fake():
    from torch._subclasses.fake_tensor import FakeTensorMode

    from roc_shmem_b200.ops.torch_ops import Linear
    y = Linear(16, 24, device="meta")(torch.empty(2, 8, 16, dtype=torch.bfloat16, device="meta"))
    assert y.shape == (2, 8, 24) and y.device.type == "meta"
    with FakeTensorMode():
        y = Linear(16, 24, device="cpu")(torch.empty(8, 16, dtype=torch.bfloat16))
    assert y.shape == (8, 24) and type(y).__name__ == "FakeTensor"


def test_transforms_and_tracing(lin):
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils._python_dispatch import TorchDispatchMode
    x = _x(3, 8, 16)
    assert torch.equal(torch.func.vmap(lin)(x), lin(x))
    names = [str(n.target) for n in make_fx(lin)(x[0]).graph.nodes if n.op == "call_function"]
    assert "bshmem.linear.default" in names
    assert "bshmem::linear" in str(torch.jit.trace(lin, (x[0],)).graph)
    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))
    with Watch():
        lin(x)
    assert "bshmem.linear.default" in seen


def test_who_is_watching():
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    from roc_shmem_b200.ops.torch_ops import _unwatched
    assert _unwatched()
    with torch.device("cpu"):                                # a default device is no observer
        assert _unwatched()
    for mode in (TorchFunctionMode, TorchDispatchMode):
        with mode():
            assert not _unwatched()
    inside = []
    torch.func.vmap(lambda v: (inside.append(_unwatched()), v)[1])(torch.zeros(2))
    assert inside == [False]


@pytest.mark.parametrize("form", ["operator", "layer"])
@pytest.mark.parametrize("noncontiguous", [False, True])
def test_second_order_and_batched_gradients(lin, form, noncontiguous):
    """Through dX as often as asked, against autograd's own product; dW has no formula and says so instead of dropping out."""
    from roc_shmem_b200.ops.torch_ops import _LinearFn
    run = torch.ops.bshmem.linear if form == "operator" else _LinearFn.apply
    w = lin.weight.detach().requires_grad_(True)
    v = _x(16, 8).t() if noncontiguous else _x(8, 16)
    x = v.requires_grad_(True)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)

    def penalty(a, b, f):
        dx, = torch.autograd.grad(f(a, b).float().pow(2).sum(), a, create_graph=True)
        return dx.float().pow(2).sum() + f(a, b).float().sum()
    got = torch.autograd.grad(penalty(x, w, run), (x, w))
    ref = torch.autograd.grad(penalty(xr, wr, lambda a, b: a @ b.t()), (xr, wr))
    for g, r in zip(got, ref):
        assert (g.float() - r).norm() <= 2e-2 * r.norm()     # a chain of four bf16 products
    dw, = torch.autograd.grad(run(x, w).float().pow(2).sum(), w, create_graph=True)
    with pytest.raises(RuntimeError, match="autograd formula"):
        torch.autograd.grad(dw.float().pow(2).sum(), x)
    dy = _x(3, 8, 24)
    dx, dw = torch.autograd.grad(run(x, w), (x, w), dy, is_grads_batched=True)
    for i in range(3):
        dxi, dwi = torch.autograd.grad(run(x, w), (x, w), dy[i])
        assert torch.equal(dx[i], dxi) and torch.equal(dw[i], dwi)
