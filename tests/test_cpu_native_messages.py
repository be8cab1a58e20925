"""put and get of a device context as the runtime makes it (csrc/host/pycall.cc, Mover), with recorders in place of the native calls."""
import ctypes as C

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
