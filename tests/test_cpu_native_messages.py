"""put and get of a device context as the runtime makes it (csrc/host/pycall.cc, Mover), with recorders in place of the native calls."""
import ctypes as C

import pytest
import torch

from tests.test_cpu_tracing import _runtime, ranges  # noqa: F401  (ranges: a fixture)


def test_a_native_message_has_its_range(ranges):  # noqa: F811
    """put and get of a context as the runtime makes it: traced from when tracing is switched on, and called as before without it."""
    from roc_shmem_b200 import _native, gpu
    from roc_shmem_b200.utils import trace
    rt, ctx = _runtime(-1)
    lib = C.CDLL(None)                                       # any function's address: a CPU tensor is no call for it
    rt.lib, rt._check = type("Lib", (), {"bshmem_gpu_ctx_put_dev": lib.labs, "bshmem_gpu_ctx_get_dev": lib.labs}), None
    ctx = gpu.DeviceRuntime._context_type(rt, 1, 0, None)
    t = torch.zeros(4)
    for on in (True, False, True):
        trace.set_tracing(on)
        for call, name in ((ctx.put, "put"), (ctx.get, "get")):
            ranges.clear()
            call(t, t, 0)
            call(t, t, 0, nbi=True)
            assert ranges == [f"bshmem.{name}"] * (2 if on else 0)
    if hasattr(torch.Tensor, "__dlpack_c_exchange_api__"):
        assert type(ctx.put) is _native._pycall().Mover


class _Table(C.Structure):
    _fields_ = [("major", C.c_uint32), ("minor", C.c_uint32), ("older", C.c_void_p), ("allocate", C.c_void_p), ("owned_from", C.c_void_p),
                ("to", C.c_void_p), ("describe", C.c_void_p), ("work_stream", C.c_void_p)]


@pytest.mark.parametrize("fault", ["another version", "nothing to describe a tensor with", "another capsule"])
def test_a_context_without_a_table_for_it(ranges, monkeypatch, fault):  # noqa: F811
    """Where torch's table is not the one that is known, a context is created all the same, with the general methods."""
    from roc_shmem_b200 import gpu
    table = _Table(2 if fault == "another version" else 1, 0, describe=None if fault.startswith("nothing") else 1)
    new = C.pythonapi.PyCapsule_New
    new.restype, new.argtypes = C.py_object, [C.c_void_p, C.c_char_p, C.c_void_p]
    name = C.create_string_buffer(b"another" if fault == "another capsule" else b"dlpack_exchange_api")
    monkeypatch.setattr(torch.Tensor, "__dlpack_c_exchange_api__", new(C.addressof(table), name, None), raising=False)
    rt, _ = _runtime(-1)
    lib, calls = C.CDLL(None), []
    rt.lib, rt._check = type("Lib", (), {"bshmem_gpu_ctx_put_dev": lib.labs, "bshmem_gpu_ctx_get_dev": lib.labs}), None
    rt._c_put_dev, rt._c_get_dev = (lambda *a: calls.append("put")), (lambda *a: calls.append("get"))
    ctx = gpu.DeviceRuntime._context_type(rt, 1, 0, None)
    t = torch.zeros(4)
    ctx.put(t, t, 0)
    ctx.get(t, t, 0, nbi=True)
    assert calls == ["put", "get"] and not hasattr(ctx.put, "context")


class _Described(C.Structure):
    _fields_ = [("data", C.c_void_p), ("device_type", C.c_int32), ("device_id", C.c_int32), ("ndim", C.c_int32), ("code", C.c_uint8),
                ("bits", C.c_uint8), ("lanes", C.c_uint16), ("shape", C.POINTER(C.c_int64)), ("strides", C.c_void_p), ("offset", C.c_uint64)]


def test_tensors_without_memory_are_not_read(ranges):  # noqa: F811
    """A tensor that a transformation made up (functionalize) is described with a null address: it is for the general method, which refuses it."""
    from roc_shmem_b200 import _native
    shape, addresses, native, method = (C.c_int64 * 1)(4), {}, [], []

    def describe(tensor, out):
        d = C.cast(out, C.POINTER(_Described)).contents
        d.data, d.device_type, d.device_id, d.ndim, d.code, d.bits, d.lanes = addresses[id(tensor)], 2, 0, 1, 2, 32, 1
        d.shape, d.strides, d.offset = shape, None, 0
        return 0
    describe_c = C.PYFUNCTYPE(C.c_int, C.py_object, C.c_void_p)(describe)
    entry = C.CFUNCTYPE(C.c_int, *[C.c_uint64] * 7)(lambda *a: native.append(a) or 0)
    table = _Table(1, 0, describe=C.cast(describe_c, C.c_void_p).value)
    new = C.pythonapi.PyCapsule_New
    new.restype, new.argtypes = C.py_object, [C.c_void_p, C.c_char_p, C.c_void_p]
    name = C.create_string_buffer(b"dlpack_exchange_api")

    class Owner:
        def put(self, *a, **kw):
            method.append(a)
    owner = Owner()
    put = _native._pycall().Mover(C.cast(entry, C.c_void_p).value, 5, 1, 0, 1, torch.Tensor, new(C.addressof(table), name, None), owner, "put",
                                  Owner.put, None)
    a, b, none = torch.zeros(4), torch.zeros(4), torch.zeros(4)
    addresses.update({id(a): 4096, id(b): 8192, id(none): None})
    put(a, b, 0)
    assert len(native) == 1 and native[0][2:5] == (4096, 8192, 16) and not method
    put(a, none, 0)
    put(none, b, 0, nbi=True)
    assert len(native) == 1 and len(method) == 2
