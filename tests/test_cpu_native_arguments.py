"""Direct native calls take what a ctypes call of the same entry point takes: anything that is an integer (numpy's, a one-element
tensor) where an integer is declared, None for an address only; flags of the Python methods are truth values."""
import numpy as np
import pytest
import torch

from roc_shmem_b200 import _native
from roc_shmem_b200.cpu import run_threads


def test_integers_of_every_kind():
    def body(rt):
        sym, src, back = rt.zeros((4,), torch.int64), torch.arange(4), torch.zeros(4, dtype=torch.int64)
        for pe in (0, np.int64(0), np.uint8(0), torch.tensor(0), False):
            for nbi in (True, False, np.bool_(True), 0, None, "yes"):
                rt.put(sym, src, pe, nbi=nbi)
                rt.get(back, sym, pe, nbi=nbi, nbytes=np.int32(32))
                assert torch.equal(back, src)
                sym.zero_()
                back.zero_()
            rt.p(sym, 5, pe)
            assert rt.g(sym, pe) == 5 and rt.atomic_fetch_add(sym, 2, pe) == 5
            sym.zero_()
        rt.put_signal(sym[:1], src[3:], sym[1:], np.int64(-1), np.int64(0))
        assert sym.tolist() == [3, -1, 0, 0]
    run_threads(1, body, heap_bytes=1 << 20)


def test_none_and_fractions_are_no_integers():
    def body(rt):
        sym, src = rt.zeros((4,), torch.int64), torch.arange(4)
        for bad in (None, 0.0, "0", np.bool_(False)):
            for call in (lambda: rt.put(sym, src, bad), lambda: rt.get(src, sym, bad), lambda: rt.p(sym, 1, bad), lambda: rt.g(sym, bad),
                         lambda: rt.atomic_fetch_add(sym, 1, bad), lambda: rt.put_signal(sym, src, sym, bad, 0)):
                with pytest.raises(TypeError):
                    call()
        assert sym.tolist() == [0] * 4
    run_threads(1, body, heap_bytes=1 << 20)


def test_addresses():
    put = _native.fast(_native.host_lib(), "bshmem_ctx_putmem")
    assert put(None, 0, None, None, 0, 0) != 0               # a null handle is refused by the call itself
    with pytest.raises(TypeError):
        put(np.int64(0), 0, None, None, 0, 0)                # an address is an int or None, as for a c_void_p
    with pytest.raises(TypeError):
        put(None, 0, None, None, 0)
