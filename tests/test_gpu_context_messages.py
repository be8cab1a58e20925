"""put and get of a device context in every form of the call: those that are made at once (plain tensors, nbi by keyword) and those that
take the general method, with the same results and the same errors."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    import roc_shmem_b200 as shmem
    r = shmem.init("device", rank=0, world_size=1, heap_bytes=64 << 20)
    yield r
    r.finalize()


FORMS = {
    "plain": lambda f, d, s: f(d, s, 0),
    "nbi": lambda f, d, s: f(d, s, 0, nbi=True),
    "not nbi": lambda f, d, s: f(d, s, 0, nbi=False),
    "truthy nbi": lambda f, d, s: f(d, s, 0, nbi=1),
    "bytes": lambda f, d, s: f(d, s, 0, nbi=True, nbytes=s.nbytes),
    "keywords": lambda f, d, s: f(dest=d, src=s, pe=0, nbi=True),
    "pe keyword": lambda f, d, s: f(d, s, pe=0),
    "numpy pe": lambda f, d, s: f(d, s, np.int64(0)),
    "parameter": lambda f, d, s: f(d, torch.nn.Parameter(s, requires_grad=False), 0, nbi=True),
    "needs grad": lambda f, d, s: f(d, s.detach().requires_grad_(s.dtype.is_floating_point), 0, nbi=True),
}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.bfloat16, torch.float32, torch.int64])
def test_forms(rt, form, dtype):
    with rt.ctx_create() as ctx:
        sym, local = rt.zeros((4, 33), dtype), torch.zeros((4, 33), dtype=dtype, device="cuda")
        values = torch.randint(0, 2, (4, 33), device="cuda").to(dtype)
        values[1:3].fill_(1)
        for move, dst, src in ((ctx.put, sym, local), (ctx.get, local, sym)):
            dst.zero_()
            src.copy_(values)
            torch.cuda.synchronize()
            FORMS[form](move, dst[1:3], src[1:3])          # a view behind the start of its storage
            ctx.quiet()
            assert torch.equal(dst[1:3], values[1:3]) and not bool(dst[0].any()) and not bool(dst[3].any())
        rt.free(sym, collective=False)


def test_other_buffers_and_sizes(rt):
    with rt.ctx_create() as ctx:
        sym = rt.zeros((64,), torch.float32)
        ctx.put(sym[:0], torch.empty(0, device="cuda"), 0, nbi=True)                 # nothing
        ctx.put(sym, torch.arange(64.0), 0)                                          # a host buffer
        ctx.quiet()
        assert torch.equal(sym.cpu(), torch.arange(64.0))
        out = np.zeros(64, np.float32)
        ctx.get(out, sym, 0)
        ctx.quiet()
        assert (out == np.arange(64)).all()
        ctx.put(sym, torch.full((), 9.0, device="cuda"), 0, nbi=True)                # one element
        ctx.quiet()
        assert sym[:2].tolist() == [9, 1]


def test_errors(rt):
    import roc_shmem_b200 as shmem
    ctx = rt.ctx_create()
    sym, local = rt.zeros((8,), torch.int32), torch.zeros(8, dtype=torch.int32, device="cuda")
    for nbi in (True, False):
        with pytest.raises(shmem.ShmemError, match="PE out of range"):
            ctx.put(sym, local, 7, nbi=nbi)
        with pytest.raises(shmem.ShmemError, match="symmetric"):
            ctx.put(local, local, 0, nbi=nbi)
        with pytest.raises(shmem.ShmemError, match="symmetric"):
            ctx.get(local, local, 0, nbi=nbi)
    with pytest.raises(TypeError):
        ctx.put(sym, local)
    with pytest.raises(TypeError):
        ctx.put(sym, local, 0, now=True)
    put, get = ctx.put, ctx.get                              # kept beyond the context's end
    ctx.destroy()
    for move in (put, get):
        with pytest.raises(shmem.ShmemError, match="invalid context"):
            move(sym, local, 0, nbi=True)
    with rt.ctx_create() as other:                           # may have the number of the old one
        for move in (put, get):
            with pytest.raises(shmem.ShmemError, match="invalid context"):
                move(sym, local, 0, nbi=True)
        other.quiet()


def test_a_subclass_keeps_its_own_methods(rt):
    from roc_shmem_b200.gpu import DeviceContext

    class Counting(DeviceContext):
        puts = 0

        def put(self, dest, src, pe, **kw):
            self.puts += 1
            return super().put(dest, src, pe, **kw)
    with rt.ctx_create() as ctx:
        mine = Counting(rt, ctx.idx, ctx.options, ctx.team)
        sym, local = rt.zeros((8,), torch.int32), torch.ones(8, dtype=torch.int32, device="cuda")
        mine.put(sym, local, 0, nbi=True)
        mine.quiet()
        assert mine.puts == 1 and bool((sym == 1).all())
