"""Collectives of a local group at the sizes where the staged reduction can go wrong: every unrolled number of sources and the
general one, a stage short of, at and past its limits, ranges that do not divide by the blocks, and repeated calls that find
the group's tables already on the device."""
import pytest
import torch

pytestmark = pytest.mark.gpu

KIB = 1024


@pytest.mark.parametrize("pes", [2, 3, 4, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int32])
def test_group_reductions(pes, dtype):
    from roc_shmem_b200.gpu import COLL_REDUCE, COLL_REDUCE_SCATTER, LocalGroup
    from roc_shmem_b200.utils import dtypes as D
    g = LocalGroup(pes, heap_bytes=64 << 20)
    try:
        torch.manual_seed(pes)
        es = torch.empty(0, dtype=dtype).element_size()
        top = (4 << 20) // es
        src, dst = g.empty((top,), dtype), g.empty((top,), dtype)
        for t in src:
            t.copy_(torch.randint(-8, 9, (top,), device="cuda"))         # whole numbers: exact in every type and order
        total = sum(t.double() for t in src)
        for nbytes in (16 * pes, 1040 * pes, 64 * KIB + 16 * pes, 160 * KIB * pes, 4 * 128 * KIB * pes - 16 * pes, 400 * KIB * pes + 48 * pes):
            n = min(nbytes // es, top) // (pes * 16 // es) * (pes * 16 // es)
            for ctas in (1, 3):
                for t in dst:
                    t.fill_(99)
                torch.cuda.synchronize()
                g.collective(COLL_REDUCE, dst, src, n, dtype=dtype, op=D.SUM, ctas=ctas)
                for t in dst:
                    assert torch.equal(t[:n].double(), total[:n]) and bool((t[n:] == 99).all())
                share = n // pes
                for t in dst:
                    t.fill_(99)
                torch.cuda.synchronize()
                g.collective(COLL_REDUCE_SCATTER, dst, src, share, dtype=dtype, op=D.SUM, ctas=ctas)
                for pe, t in enumerate(dst):
                    assert torch.equal(t[:share].double(), total[pe * share:(pe + 1) * share]) and bool((t[share:] == 99).all())
    finally:
        g.close()


@pytest.mark.parametrize("pes,ctas", [(2, 1), (3, 5), (8, 16), (8, 18)])
@pytest.mark.parametrize("nbytes", [16, 32 * KIB - 16, 32 * KIB, 96 * KIB + 16, 160 * KIB + 8, 700 * KIB + 48])
def test_group_moves(pes, ctas, nbytes):
    """fcollect and alltoall on both sides of the size and the alignment from which blocks move their share with bulk copies,
    and shares that do not fill the last chunk."""
    from roc_shmem_b200.gpu import COLL_ALLTOALL, COLL_FCOLLECT, LocalGroup
    g = LocalGroup(pes, heap_bytes=64 << 20)
    try:
        torch.manual_seed(nbytes)
        src, dst = g.empty((pes * nbytes,), torch.uint8), g.empty((pes * nbytes + 64,), torch.uint8)
        for kind in (COLL_FCOLLECT, COLL_ALLTOALL):
            for s, d in zip(src, dst):
                s.copy_(torch.randint(0, 256, s.shape, device="cuda", dtype=torch.uint8))
                d.fill_(7)
            torch.cuda.synchronize()
            g.collective(kind, dst, src, nbytes, ctas=ctas)
            for me, d in enumerate(dst):
                part = slice(0, nbytes) if kind == COLL_FCOLLECT else slice(me * nbytes, (me + 1) * nbytes)
                assert torch.equal(d[:pes * nbytes], torch.cat([s[part] for s in src])) and bool((d[pes * nbytes:] == 7).all())
    finally:
        g.close()


def test_first_collective_on_a_stream_of_its_own():
    """A group made and used on a stream that does not wait for the default one, whose first call finds that stream busy: the
    count of finished blocks starts at zero on the launch's stream (a call that returned early would find the old values)."""
    import torch

    from roc_shmem_b200 import gpu
    from roc_shmem_b200.utils import dtypes as D
    stream = torch.cuda.Stream()
    for _ in range(3):
        torch.cuda.synchronize()
        junk = torch.full((1 << 20,), -1, dtype=torch.int32, device="cuda")          # what a fresh allocation may hold
        del junk
        torch.cuda.empty_cache()
        with torch.cuda.stream(stream):
            g = gpu.LocalGroup(4, heap_bytes=128 << 20)
            src, dst = g.empty((4096,), torch.int32), g.empty((4096,), torch.int32)
            for i, (s, d) in enumerate(zip(src, dst)):
                s.fill_(i + 1)
                d.zero_()
            torch.cuda._sleep(20_000_000)
            for _ in range(3):
                g.collective(gpu.COLL_REDUCE, dst, src, 4096, dtype=torch.int32, op=D.SUM, ctas=4)
                host = [d.cpu() for d in dst]
                assert all(bool((h == 10).all()) for h in host)
        for rt in g.pes:
            rt.finalize()
