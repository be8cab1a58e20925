"""Small host-issued messages on the NVLink backend: payload, signal and single-element paths at the sizes where the
kernel that moves them changes (a block's piece, the one-block limit of a signalled message, the copy-engine limit)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    import roc_shmem_b200 as shmem
    r = shmem.init("device", rank=0, world_size=1, heap_bytes=64 << 20, timeout_ms=5000)
    yield r
    shmem.finalize()


@pytest.mark.parametrize("n", [1, 63, 4095, 4096, 4097, 32768, 32769, 131072, 131073])
@pytest.mark.parametrize("shift", [0, 3])
def test_put_get_signal_sizes(rt, n, shift):
    sym = rt.zeros((n + 64,), torch.uint8)
    sig = rt.zeros((1,), torch.int64)
    src = torch.randint(0, 256, (n + 8,), dtype=torch.uint8, device="cuda")
    for nbi in (False, True):
        sym.zero_()
        rt.put(sym[shift:shift + n], src[:n], 0, nbi=nbi)
        rt.quiet()
        assert torch.equal(sym[shift:shift + n], src[:n])
        assert int(sym[shift + n:].sum()) == 0 and int(sym[:shift].sum()) == 0       # nothing outside the message
        back = torch.zeros(n + 8, dtype=torch.uint8, device="cuda")
        rt.get(back[:n], sym[shift:shift + n], 0, nbi=nbi)
        rt.quiet()
        assert torch.equal(back[:n], src[:n]) and int(back[n:].sum()) == 0
        sym.zero_()
        rt.put_signal(sym[shift:shift + n], src[:n], sig, 7, 0, nbi=nbi)
        rt.wait_until(sig, "eq", 7)
        rt.quiet()
        assert torch.equal(sym[shift:shift + n], src[:n]) and int(sym[shift + n:].sum()) == 0
        sig.zero_()
    host = torch.zeros(n, dtype=torch.uint8)                                          # a host buffer takes the copy engine
    rt.get(host, sym[shift:shift + n], 0)
    assert torch.equal(host, src[:n].cpu())
    rt.free(sym)
    rt.free(sig)


@pytest.mark.parametrize("n", [131073, (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("to,frm", [(0, 0), (5, 5), (5, 0)])
def test_put_get_up_to_the_copy_engine(rt, n, to, frm):
    sym = rt.zeros((n + 64,), torch.uint8)
    src = torch.randint(0, 256, (n + 16,), dtype=torch.uint8, device="cuda")
    back = torch.zeros(n + 64, dtype=torch.uint8, device="cuda")
    rt.put(sym[to:to + n], src[frm:frm + n], 0)
    rt.get(back[frm:frm + n], sym[to:to + n], 0)
    for got, at in ((sym, to), (back, frm)):
        assert torch.equal(got[at:at + n], src[frm:frm + n])
        assert int(got[:at].sum()) == 0 and int(got[at + n:].sum()) == 0
    rt.free(sym)


@pytest.mark.parametrize("dtype,values", [(torch.uint8, (0, 255)), (torch.int8, (-128, 127)), (torch.int16, (-32768, 5)),
                                          (torch.int32, (-1, 2**31 - 1)), (torch.int64, (-2**63, 2**63 - 1)),
                                          (torch.float32, (-0.5, 3.25)), (torch.float64, (1e-300, -2.0)), (torch.bfloat16, (1.5, -3.0))])
def test_single_elements(rt, dtype, values):
    x = rt.zeros((4,), dtype)
    for i, v in enumerate(values):
        rt.p(x[i + 1:], v, 0)
        assert rt.g(x[i + 1:], 0) == v
    rt.quiet()
    assert x.tolist() == [0, *values, 0]
    rt.free(x)
