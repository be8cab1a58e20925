"""Ranges of the host API on the device backend's classes, with recorders in place of the native calls and of NVTX: one range per
message, through the runtime or a context, on the direct path and on the general one."""
import contextlib

import pytest
import torch


@pytest.fixture
def ranges(monkeypatch):
    from roc_shmem_b200.utils import trace
    seen = []

    @contextlib.contextmanager
    def record(name):
        seen.append(name)
        yield
    monkeypatch.setattr(trace, "nvtx_range", record)
    trace.set_tracing(True)
    yield seen
    trace.set_tracing(False)


def _runtime(device_index):
    from roc_shmem_b200 import gpu
    rt = object.__new__(gpu.DeviceRuntime)
    rt._hv, rt._dev_index = 0, device_index                  # a CPU tensor's device index is -1
    for n in ("put_dev", "get_dev", "put_signal_dev", "put", "put_nbi", "get", "get_nbi", "put_signal", "put_signal_nbi"):
        setattr(rt, "_c_" + n, lambda *a: 0)
    return rt, gpu.DeviceContext(rt, 1, 0, None)


@pytest.mark.parametrize("direct", [True, False])
def test_one_range_per_message(ranges, direct):
    rt, ctx = _runtime(-1 if direct else 0)
    t = torch.zeros(4)
    for call, name in ((lambda: rt.put(t, t, 0), "put"), (lambda: ctx.put(t, t, 0), "put"), (lambda: rt.get(t, t, 0, nbi=True), "get"),
                       (lambda: ctx.get(t, t, 0), "get"), (lambda: rt.put_signal(t, t, t, 1, 0), "put_signal"),
                       (lambda: ctx.put_signal(t, t, t, 1, 0), "put_signal")):
        ranges.clear()
        call()
        assert ranges == [f"bshmem.{name}"]


def test_nothing_while_off(ranges):
    from roc_shmem_b200.utils import trace
    trace.set_tracing(False)
    rt, ctx = _runtime(-1)
    t = torch.zeros(4)
    ctx.put(t, t, 0)
    rt.get(t, t, 0)
    assert ranges == []
