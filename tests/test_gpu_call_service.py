"""Blocking calls of the default context that follow one another closely (served by one block, k_calls): every kind, between kernels of the
caller's stream that write what a call reads and read what it wrote, on both sides of the pause that ends a series, with a stream
that is busy, from several threads, and with a wait for what another stream has yet to bring about."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    import roc_shmem_b200 as shmem
    r = shmem.init("device", rank=0, world_size=1, heap_bytes=64 << 20)
    yield r
    r.finalize()


def test_series_between_kernels_of_the_stream(rt):
    box, flag, counter = rt.empty((9000,), torch.int32), rt.zeros((1,), torch.int64), rt.zeros((1,), torch.int64)
    src = torch.empty(9000, dtype=torch.int32, device="cuda")
    for i in range(1, 400):
        n = (1, 7, 1024, 2049, 8192)[i % 5]
        src.fill_(i)                                       # in the stream, not waited for
        assert rt.atomic_fetch_add(counter, 1, 0) == i - 1 + 2 * (i - 1)
        rt.put_signal(box[:n], src[:n], flag, i, 0)
        rt.wait_until(flag, "ge", i)
        counter.add_(2)                                    # a kernel behind one call and before the next
        assert rt.g(counter, 0) == 3 * i and rt.g(flag, 0) == i
        assert rt.g(box[n - 1:n], 0) == i
        if i % 3 == 0:
            assert bool((box[:n] == i).all())              # a kernel of the stream behind the calls
        assert all(rt.atomic_fetch_add(counter, 0, 0) == 3 * i for _ in range(i % 16))      # uninterrupted calls, from none to a series
        if i % 50 == 0:
            time.sleep(0.002)                              # the series ends; the next calls begin another


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64, torch.float32, torch.float64])
def test_operators_and_types(rt, dtype):
    word = rt.zeros((1,), dtype)
    for _ in range(20):
        rt.atomic_set(word, 5, 0)
        assert rt.atomic_fetch_add(word, 3, 0) == 5 and rt.atomic_swap(word, 2, 0) == 8 and rt.g(word, 0) == 2
        if not dtype.is_floating_point:
            assert rt.atomic_compare_swap(word, 2, 9, 0) == 2 and rt.atomic_fetch(word, 0) == 9
            assert rt.atomic_fetch_or(word, 6, 0) == 9 and rt.g(word, 0) == 15
        rt.wait_until(word, "gt", 1)


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.bfloat16])
def test_small_elements(rt, dtype):
    x = rt.empty((5,), dtype)
    x.copy_(torch.arange(5, device="cuda"))
    for _ in range(10):
        assert [rt.g(x[i:i + 1], 0) for i in range(5)] == [0, 1, 2, 3, 4]


def test_a_busy_stream_keeps_its_order(rt):
    word = rt.zeros((1,), torch.int64)
    for i in range(20):
        for _ in range(10):
            rt.g(word, 0)                                  # a series is running
        torch.cuda._sleep(400_000)
        word.fill_(i + 100)
        assert rt.atomic_fetch_add(word, 1, 0) == i + 100


def test_a_wait_for_another_stream(rt):
    flag = rt.zeros((1,), torch.int64)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for i in range(1, 10):
        for _ in range(10):
            assert rt.g(flag, 0) == i - 1
        with torch.cuda.stream(side):
            torch.cuda._sleep(2_000_000)
            flag.fill_(i)
        rt.wait_until(flag, "eq", i)
        assert rt.g(flag, 0) == i


def test_another_stream_of_the_runtime(rt):
    word, stream = rt.zeros((1,), torch.int64), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        for i in range(30):
            rt.set_stream(stream if i % 2 else torch.cuda.current_stream())
            with torch.cuda.stream(stream if i % 2 else torch.cuda.current_stream()):
                torch.cuda._sleep(100_000)
                word.fill_(i)
                assert all(rt.g(word, 0) == i for _ in range(10)) and rt.atomic_fetch_add(word, 1, 0) == i
    finally:
        rt.set_stream(torch.cuda.current_stream())


def test_threads(rt):
    counter, words = rt.zeros((1,), torch.int64), rt.zeros((4,), torch.int64)
    torch.cuda.synchronize()
    errors = []

    def work(k):
        try:
            for i in range(200):
                rt.atomic_fetch_add(counter, 1, 0)
                assert rt.atomic_fetch_add(words[k:k + 1], 1, 0) == i
        except BaseException as e:                         # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and rt.g(counter, 0) == 800


def test_while_another_stream_is_captured(rt):
    word, out, side = rt.zeros((1,), torch.int64), torch.zeros(8, device="cuda"), torch.cuda.Stream()
    rt.set_stream(None)                                    # the runtime's own stream: nothing of the caller's is in it
    try:
        torch.cuda.synchronize()
        for _ in range(10):
            rt.g(word, 0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out.add_(1)
            for i in range(25):
                assert rt.atomic_fetch_add(word, 1, 0) == i
        graph.replay()
        torch.cuda.synchronize()
        assert bool((out == 1).all())
    finally:
        rt.set_stream(torch.cuda.current_stream())


@pytest.mark.parametrize("n", [32768, 32769, 65536, 100_001, 262143, 262144, 262145])
@pytest.mark.parametrize("skew", [0, 1, 4])
def test_payloads_of_a_series(rt, n, skew):
    """Both sides of what the block takes as a put with signal, on and off the two sides' common alignment."""
    box, flag = rt.empty((n + 64,), torch.uint8), rt.zeros((1,), torch.int64)
    src = torch.empty(n + 64, dtype=torch.uint8, device="cuda")
    for i in range(1, 13):
        src.copy_(torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda"))
        box.fill_(7)
        torch.cuda.synchronize()
        for _ in range(6):
            rt.g(flag, 0)                                  # a series is running
        rt.put_signal(box[16 + skew:16 + skew + n], src[16:16 + n], flag, i, 0)
        rt.wait_until(flag, "ge", i)
        assert torch.equal(box[16 + skew:16 + skew + n], src[16:16 + n])
        assert bool((box[:16 + skew] == 7).all()) and bool((box[16 + skew + n:] == 7).all())
    rt.free(box, collective=False)
    rt.free(flag, collective=False)


@pytest.fixture()
def blocking_stream():
    """A stream that the legacy default stream and it wait for one another (torch's own streams do not)."""
    import ctypes as C
    handle = C.c_void_p()
    assert int(torch.cuda.cudart().cudaStreamCreate(C.addressof(handle))) == 0
    yield torch.cuda.ExternalStream(handle.value)
    torch.cuda.synchronize()
    assert int(torch.cuda.cudart().cudaStreamDestroy(handle.value)) == 0


@pytest.mark.parametrize("runtime_on", ["legacy", "blocking"])
def test_work_that_the_stream_waits_for(rt, blocking_stream, runtime_on):
    """The runtime on one of the legacy default stream and a blocking stream, work on the other one: a call follows it, as a launch would."""
    word = rt.zeros((1,), torch.int64)
    legacy = torch.cuda.default_stream()
    mine, other = (legacy, blocking_stream) if runtime_on == "legacy" else (blocking_stream, legacy)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        torch.cuda._sleep(400_000)
        word.add_(100)
    torch.cuda.synchronize()
    try:
        rt.set_stream(mine)
        with torch.cuda.stream(other):
            for i in range(50):
                rt.atomic_set(word, 0, 0)
                torch.cuda.synchronize()
                for _ in range(10):
                    rt.g(word, 0)                          # a series is running
                graph.replay()                             # some 200 us, launched in less time than ends a series
                assert rt.atomic_fetch_add(word, 1, 0) == 100
                assert rt.g(word, 0) == 101
    finally:
        rt.set_stream(torch.cuda.current_stream())
