"""Non-blocking messages of a context through its ring (csrc/cuda/gpu_backend.cu, k_ring): sizes around its limit and its 16-byte
pieces, windows beyond its slots, pauses in which the serving block ends, messages that depend on earlier ones, other operations of the
same context in between, and several threads."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def rt():
    import roc_shmem_b200 as shmem
    r = shmem.init("device", rank=0, world_size=1, heap_bytes=256 << 20)
    yield r
    shmem.finalize()


@pytest.mark.parametrize("n", [1, 15, 16, 64, 100, 4096, 16383, 16384, 16385])
@pytest.mark.parametrize("window", [1, 17, 600])
def test_windows(rt, n, window):
    import roc_shmem_b200 as shmem
    ctx = rt.ctx_create(shmem.CTX_SERIALIZED)
    sym, src, back = rt.empty((window, n), torch.uint8), torch.randint(0, 256, (window, n), dtype=torch.uint8, device="cuda"), torch.zeros(window, n, dtype=torch.uint8, device="cuda")
    sym.zero_()
    torch.cuda.synchronize()
    for pause in (0, 3e-5):                          # longer than the block waits for a message
        for i in range(window):
            ctx.put(sym[i], src[i], 0, nbi=True)
            if pause and i % 37 == 0:
                time.sleep(pause)
        ctx.quiet()
        assert torch.equal(sym, src)
        for i in range(window):
            ctx.get(back[i], sym[i], 0, nbi=True)
        ctx.quiet()
        assert torch.equal(back, src)
        src.add_(1)
        torch.cuda.synchronize()
    ctx.destroy()


def test_dependent_messages_keep_their_order(rt):
    """Each message reads what the one before wrote, or overwrites it; a fence orders messages that share nothing."""
    import roc_shmem_b200 as shmem
    ctx = rt.ctx_create(shmem.CTX_SERIALIZED)
    n, steps = 4096, 300
    sym, a, b = rt.empty((n,), torch.uint8), torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda")
    rows = torch.arange(steps, device="cuda").to(torch.uint8).view(-1, 1).repeat(1, n).contiguous()
    got = torch.zeros_like(rows)
    torch.cuda.synchronize()
    for i in range(steps):
        ctx.put(sym, rows[i], 0, nbi=True)
        ctx.get(got[i], sym, 0, nbi=True)
        if i % 50 == 0:
            ctx.fence()
    ctx.put(sym, a, 0, nbi=True)
    ctx.put(sym[8:72], rows[9][8:72], 0, nbi=True)      # into the middle of the one before
    ctx.get(b, sym, 0, nbi=True)
    ctx.quiet()
    assert torch.equal(got, rows)
    assert bool((b[8:72] == 9).all()) and int(b.sum()) == 9 * 64
    ctx.destroy()


def test_other_operations_follow_the_messages(rt):
    import roc_shmem_b200 as shmem
    ctx = rt.ctx_create(shmem.CTX_SERIALIZED)
    word, big, flag = rt.zeros((4,), torch.int64), rt.zeros((1 << 20,), torch.uint8), rt.zeros((1,), torch.int64)
    vals = torch.arange(1, 65, dtype=torch.int64, device="cuda")
    src = torch.full((1 << 20,), 5, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for i in range(64):
        ctx.put(word[:1], vals[i:i + 1], 0, nbi=True)
        assert rt.atomic_fetch_add(word[:1], 1000, 0, ctx=ctx) == i + 1      # sees the message, and the next message overwrites it
        ctx.put(word[1:2], vals[i:i + 1], 0, nbi=True)
        if i % 4 == 0:
            ctx.put(big, src, 0, nbi=True)                                  # too large for the ring
        if i % 5 == 0:
            ctx.put(word[2:3], vals[i:i + 1], 0)                            # blocking
            assert int(word[2]) == i + 1 and int(word[1]) == i + 1
        rt.put_signal(word[3:4], vals[i:i + 1], flag, i + 1, 0, ctx=ctx)
        assert int(flag) == i + 1 and int(word[3]) == i + 1 and int(word[1]) == i + 1
    ctx.quiet()
    assert torch.equal(big, src)
    ctx.destroy()


@pytest.mark.parametrize("kind", ["large", "copy engine", "host buffer", "put_signal", "p"])
@pytest.mark.parametrize("before,behind", [(1, 1), (1, 40), (64, 300), (0, 700)])
def test_messages_behind_an_operation_that_nobody_waits_for(rt, kind, before, behind):
    """Messages, an operation of the stream, a fence, a message into the operation's range and more behind it: after quiet all of it
    is done, in that order, and nothing is done again once the sources hold something else."""
    import roc_shmem_b200 as shmem
    ctx = rt.ctx_create(shmem.CTX_SERIALIZED)
    n = {"large": 1 << 20, "copy engine": 8 << 20, "host buffer": 1 << 18, "put_signal": 1 << 17, "p": 8}[kind]
    sym, small, flag = rt.zeros((n,), torch.uint8), rt.zeros((before + behind, 64), torch.uint8), rt.zeros((1,), torch.int64)
    src = torch.zeros(n, dtype=torch.uint8, device="cpu" if kind == "host buffer" else "cuda")
    if kind == "host buffer":
        src = src.pin_memory()
    msgs, patch = torch.zeros(before + behind, 64, dtype=torch.uint8, device="cuda"), torch.zeros(2, dtype=torch.uint8, device="cuda")
    for r in range(12):
        src.fill_(r + 1)
        msgs.fill_(r + 1)
        patch.fill_(r + 101)
        torch.cuda.synchronize()
        for i in range(before):
            ctx.put(small[i], msgs[i], 0, nbi=True)
        if kind == "put_signal":
            ctx.put_signal(sym, src, flag, r + 1, 0, nbi=True)
        elif kind == "p":
            rt.p(sym.view(torch.int64), (r + 1) * 0x0101010101010101, 0, ctx=ctx)
        else:
            ctx.put(sym, src, 0, nbi=True)
        ctx.fence()
        ctx.put(sym[3:5], patch, 0, nbi=True)
        for i in range(before, before + behind):
            ctx.put(small[i], msgs[i], 0, nbi=True)
        ctx.quiet()
        for t in (src, msgs, patch):
            t.fill_(200)
        torch.cuda.synchronize()
        if kind == "put_signal":
            assert int(flag) == r + 1
        assert int((sym == r + 1).sum()) == n - 2 and bool((sym[3:5] == r + 101).all()) and bool((small == r + 1).all()), r
    ctx.destroy()


def test_threads(rt):
    """Three threads, two of them on one context, each with rows of its own."""
    import roc_shmem_b200 as shmem
    shared, own = rt.ctx_create(0), rt.ctx_create(0)
    rows, n, rounds = 40, 256, 25
    sym = rt.zeros((3, rows, n), torch.uint8)
    src = torch.randint(0, 256, (3, rounds, rows, n), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    bad, done = [], []

    def work(t, ctx):
        try:
            torch.cuda.set_device(0)
            for r in range(rounds):
                for i in range(rows):
                    ctx.put(sym[t, i], src[t, r, i], 0, nbi=True)
                ctx.quiet()
                if not torch.equal(sym[t], src[t, r]):
                    bad.append((t, r))
                done.append((t, r))
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=work, args=(t, c)) for t, c in enumerate((shared, shared, own))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not bad and not any(t.is_alive() for t in threads) and len(done) == 3 * rounds, bad
    shared.destroy()
    own.destroy()


def test_quiet_of_one_thread_beside_messages_of_another(rt):
    """One context: a thread's large puts are done when its quiet returns, whatever blocks another thread's messages launch meanwhile."""
    ctx = rt.ctx_create(0)
    n, rounds = 1 << 20, 150
    big, small = rt.zeros((n,), torch.uint8), rt.zeros((32, 64), torch.uint8)
    src, msgs = torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.randint(0, 256, (32, 64), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    bad, end = [], threading.Event()

    def puts():
        try:
            torch.cuda.set_device(0)
            for r in range(rounds):
                src.fill_(r % 250 + 1)
                torch.cuda.current_stream().synchronize()
                ctx.put(big, src, 0, nbi=True)
                ctx.quiet()
                if not bool((big == r % 250 + 1).all()):
                    bad.append(r)
        except Exception as e:  # noqa: BLE001
            bad.append(e)
        finally:
            end.set()

    def messages():
        try:
            torch.cuda.set_device(0)
            while not end.is_set():
                for i in range(32):
                    ctx.put(small[i], msgs[i], 0, nbi=True)
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=f) for f in (puts, messages)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not bad and not any(t.is_alive() for t in threads), bad
    ctx.quiet()
    assert torch.equal(small, msgs)
    ctx.destroy()


def test_more_messages_than_slots_while_a_stream_is_captured(rt):
    """Non-blocking puts behind long copies, more of them than the ring has slots, while another stream is captured."""
    ctx = rt.ctx_create(0)
    big, small = rt.zeros((64 << 20,), torch.uint8), rt.zeros((600, 64), torch.uint8)
    src, msgs = torch.full((64 << 20,), 3, dtype=torch.uint8, device="cuda"), torch.randint(0, 256, (600, 64), dtype=torch.uint8, device="cuda")
    x, g = torch.zeros(16, device="cuda"), torch.cuda.CUDAGraph()
    rows = list(zip(small.unbind(0), msgs.unbind(0)))
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        x.add_(1)
        for _ in range(64):
            ctx.put(big, src, 0, nbi=True)
        for d, s in rows:
            ctx.put(d, s, 0, nbi=True)
        x.add_(1)
    ctx.quiet()
    assert torch.equal(small, msgs) and bool((big == 3).all())
    g.replay()
    torch.cuda.synchronize()
    assert bool((x == 2).all())
    ctx.destroy()
