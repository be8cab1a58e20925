"""Long non-blocking messages of a context (the ring's form of several blocks): sizes around its pieces and its limits, mixed with short ones, off
16-byte boundaries, in both directions, behind one another where they touch, and around operations of the context."""
import pytest
import torch

pytestmark = pytest.mark.gpu
KIB = 1024


@pytest.fixture(scope="module")
def rt():
    import roc_shmem_b200 as shmem
    r = shmem.init("device", rank=0, world_size=1, heap_bytes=512 << 20)
    yield r
    r.finalize()


@pytest.fixture()
def ctx(rt):
    with rt.ctx_create() as c:
        yield c


def _random(n):
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("n", [4096, 12345, 16384, 16385, 20481, 64 * KIB, 100_001, 128 * KIB + 1, 512 * KIB, 512 * KIB + 1, 1 << 20])
@pytest.mark.parametrize("skew", [0, 1, 4])
def test_sizes(rt, ctx, n, skew):
    count = 20
    sym, local = rt.empty((count, n + 64), torch.uint8), torch.empty((count, n + 64), dtype=torch.uint8, device="cuda")
    for move, dst, src, there, here in ((ctx.put, sym, local, 16 + skew, 16), (ctx.get, local, sym, 16, 16 + skew)):
        src.copy_(_random(src.numel()).view_as(src))
        dst.fill_(7)
        torch.cuda.synchronize()
        for i in range(count):
            move(dst[i, there:there + n], src[i, here:here + n], 0, nbi=True)
        ctx.quiet()
        assert torch.equal(dst[:, there:there + n], src[:, here:here + n])
        assert bool((dst[:, :there] == 7).all()) and bool((dst[:, there + n:] == 7).all())
    rt.free(sym, collective=False)


@pytest.mark.parametrize("seed", range(4))
def test_mixed_with_short_ones(rt, ctx, seed):
    import random
    rng = random.Random(seed)
    sizes = [rng.choice([1, 64, 4096, 16_000, 16_400, 20_000, 300_000]) for _ in range(300)]
    at = [0]
    for n in sizes:
        at.append(at[-1] + (n + 15) // 16 * 16)
    sym, local = rt.zeros((at[-1],), torch.uint8), _random(at[-1])
    flag = rt.zeros((1,), torch.int64)
    torch.cuda.synchronize()
    for i, n in enumerate(sizes):
        ctx.put(sym[at[i]:at[i] + n], local[at[i]:at[i] + n], 0, nbi=True)
        if i % 37 == 36:
            ctx.atomic_fetch_add(flag, 1, 0)               # an operation of the context between messages
        if i % 53 == 52:
            ctx.fence()
    ctx.quiet()
    for i, n in enumerate(sizes):
        assert torch.equal(sym[at[i]:at[i] + n], local[at[i]:at[i] + n]), i
    assert rt.g(flag, 0) == 300 // 37
    rt.free(sym, collective=False)


def test_messages_that_touch_follow_one_another(rt, ctx):
    n, steps = 70_000, 40
    sym = rt.zeros((steps + 1, n), torch.uint8)
    first = _random(n)
    torch.cuda.synchronize()
    for _ in range(5):
        sym[1:].zero_()
        torch.cuda.synchronize()
        ctx.put(sym[0], first, 0, nbi=True)
        for i in range(steps):                             # each reads what the one before it writes
            size = n if i % 3 else 13000
            ctx.put(sym[i + 1, :size], sym[i, :size], 0, nbi=True)
            if size < n:
                ctx.get(sym[i + 1, size:], sym[i, size:], 0, nbi=True)
        ctx.quiet()
        assert torch.equal(sym[steps], first)
    rt.free(sym, collective=False)


def test_more_than_the_ring_holds(rt, ctx):
    n = 17000
    sym, local = rt.zeros((1000, n), torch.uint8), _random(1000 * n).view(1000, n)
    torch.cuda.synchronize()
    for i in range(1000):
        ctx.put(sym[i], local[i], 0, nbi=True)
    ctx.quiet()
    assert torch.equal(sym, local)
    rt.free(sym, collective=False)


def test_what_the_stream_wrote_before(rt, ctx):
    """The messages of a window behind a synchronised kernel move what it wrote."""
    n = 50_000
    sym, local = rt.zeros((8, n), torch.int32), torch.zeros((8, n), dtype=torch.int32, device="cuda")
    for i in range(1, 60):
        local.fill_(i)
        torch.cuda.current_stream().synchronize()
        for k in range(8):
            ctx.put(sym[k], local[k], 0, nbi=True)
        ctx.quiet()
        assert bool((sym == i).all())
    rt.free(sym, collective=False)


def test_what_the_messages_wrote_before(rt, ctx):
    """Within one window, through the same blocks: a buffer is read by messages, written by another one, and read again, over and over."""
    n, rounds = 300_000, 30
    sym, values = rt.zeros((2 * rounds + 1, n), torch.uint8), _random(rounds * n).view(rounds, n)
    torch.cuda.synchronize()
    for _ in range(5):
        sym.zero_()
        torch.cuda.synchronize()
        for i in range(rounds):
            ctx.put(sym[0], values[i], 0, nbi=True)
            ctx.put(sym[2 * i + 1], sym[0], 0, nbi=True)
            ctx.get(sym[2 * i + 2], sym[0], 0, nbi=True)
        ctx.quiet()
        assert torch.equal(sym[1::2], values) and torch.equal(sym[2::2], values)
    rt.free(sym, collective=False)


def test_beside_products(rt, ctx):
    """Blocks that find a place late, or not before the messages are done."""
    a = torch.randn(4096, 4096, device="cuda", dtype=torch.bfloat16)
    side, n = torch.cuda.Stream(), 200_000
    sym, local = rt.zeros((16, n), torch.uint8), _random(16 * n).view(16, n)
    torch.cuda.synchronize()
    for count in (1, 2, 5, 16) * 10:
        sym.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            for _ in range(4):
                a @ a
        for k in range(count):
            ctx.put(sym[k], local[k], 0, nbi=True)
        ctx.quiet()
        assert torch.equal(sym[:count], local[:count])
    torch.cuda.synchronize()
    rt.free(sym, collective=False)


def test_a_context_made_while_the_default_stream_is_busy(rt):
    n = 200_000
    sym, local = rt.zeros((8, n), torch.uint8), _random(8 * n).view(8, n)
    torch.cuda.synchronize()
    for _ in range(5):
        sym.zero_()
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)
        with rt.ctx_create() as c:
            for k in range(8):
                c.put(sym[k], local[k], 0, nbi=True)
            c.quiet()
        assert torch.equal(sym, local)
    rt.free(sym, collective=False)
