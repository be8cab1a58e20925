"""Group collectives by few blocks, of which each tells the host itself that it is done, and by more, which are counted, against sums and copies by
torch: at odd sizes, for every kind, with results in place of the sources, in a team that leaves PEs out, and between calls of more blocks than
there are multiprocessors, which are turned away."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(gpu, kind, op, src, n, root):
    """What each member's dest holds afterwards (None: it is left alone); reductions in team order, as the collective makes them."""
    pes = len(src)

    def reduced(parts):
        acc = parts[0].clone()
        for p in parts[1:]:
            acc = acc + p if op == "sum" else acc * p if op == "prod" else torch.maximum(acc, p)
        return acc
    if kind == gpu.COLL_REDUCE:
        return [reduced(src)] * pes
    if kind == gpu.COLL_REDUCE_ROOT:
        return [reduced(src) if k == root else None for k in range(pes)]
    if kind == gpu.COLL_REDUCE_SCATTER:
        return [reduced([s[k * n:(k + 1) * n] for s in src]) for k in range(pes)]
    if kind == gpu.COLL_FCOLLECT:
        return [torch.cat(src)] * pes
    if kind == gpu.COLL_ALLTOALL:
        return [torch.cat([s[k * n:(k + 1) * n] for s in src]) for k in range(pes)]
    return [None if k == root else src[root] for k in range(pes)]


@pytest.mark.parametrize("pes,ctas", [(2, 1), (2, 4), (3, 2), (5, 1), (8, 1)])
@pytest.mark.parametrize("n", [1, 7, 1024, 1031, 4096, 40001])
def test_few_blocks_and_many(pes, ctas, n):
    from roc_shmem_b200 import gpu
    from roc_shmem_b200.utils import dtypes as D
    g = gpu.LocalGroup(pes, heap_bytes=64 << 20)
    try:
        torch.manual_seed(n + pes)
        many = 8 // pes + 1                               # more than tell the host themselves
        kinds = [(gpu.COLL_REDUCE, n, n, n), (gpu.COLL_REDUCE_SCATTER, n * pes, n, n), (gpu.COLL_FCOLLECT, n, n * pes, n * 4),
                 (gpu.COLL_ALLTOALL, n * pes, n * pes, n * 4), (gpu.COLL_BROADCAST, n, n, n * 4), (gpu.COLL_REDUCE_ROOT, n, n, n)]
        for dtype, op in ((torch.float32, "sum"), (torch.int32, "max"), (torch.float32, "prod")):
            for kind, n_src, n_dst, count in kinds:
                call = dict(dtype=dtype, op={"sum": D.SUM, "max": D.MAX, "prod": D.PROD}[op], root=pes - 1)
                src, one, two = g.empty((n_src,), dtype), g.empty((n_dst + 1,), dtype), g.empty((n_dst + 1,), dtype)
                for s in src:
                    s.copy_((torch.randn(n_src, device="cuda") * 100).to(dtype))
                for t in one + two:
                    t.fill_(7)
                want = _expected(gpu, kind, op, [s.clone() for s in src], n, pes - 1)
                torch.cuda.synchronize()
                g.collective(kind, one, src, count, ctas=ctas, **call)
                g.collective(kind, two, src, count, ctas=many, **call)
                for a, b, w in zip(one, two, want):
                    for t in (a, b):
                        assert torch.equal(t[:n_dst], torch.full_like(t[:n_dst], 7) if w is None else w) and bool((t[n_dst:] == 7).all())
                if kind == gpu.COLL_REDUCE:               # in place, several calls in a row
                    for _ in range(2):
                        for s, d in zip(src, two):
                            d[:n].copy_(s)
                        torch.cuda.synchronize()
                        g.collective(kind, two, two, count, dtype=dtype, op=call["op"], ctas=ctas)
                        for a, b in zip(one, two):
                            assert torch.equal(a, b)
                for pe, rt in enumerate(g.pes):
                    for t in (src[pe], one[pe], two[pe]):
                        rt.free(t, collective=False)
    finally:
        g.close()


def test_more_blocks_than_multiprocessors():
    """The exchanging form's launch, which wants them all at once, turns such calls away, and takes barriers; the passes in between share its device
    table and counter."""
    import roc_shmem_b200 as shmem
    from roc_shmem_b200 import gpu
    pes, n = 8, 4099
    blocks = torch.cuda.get_device_properties(0).multi_processor_count // pes
    g = gpu.LocalGroup(pes, heap_bytes=64 << 20)
    try:
        src, dst = g.empty((n * pes,), torch.int32), g.empty((n * pes,), torch.int32)
        for i, ctas in enumerate((2, blocks, blocks + 6, 4, 1, 2 * blocks + 8, blocks, 1) * 2):
            kind = (gpu.COLL_FCOLLECT, gpu.COLL_ALLTOALL, gpu.COLL_BROADCAST)[i % 3]
            for s, d in zip(src, dst):
                s.copy_(torch.randint(-1000, 1000, s.shape, device="cuda"))
                d.fill_(7)
            part = n * pes if kind == gpu.COLL_ALLTOALL else n
            want = _expected(gpu, kind, None, [s[:part].clone() for s in src], n, 3)
            torch.cuda.synchronize()
            if ctas > blocks:
                with pytest.raises(shmem.ShmemError, match="cooperative launch"):
                    g.collective(kind, dst, src, n * 4, root=3, ctas=ctas)
                want = [None] * pes
            else:
                g.collective(kind, dst, src, n * 4, root=3, ctas=ctas)
            g.collective(gpu.COLL_BARRIER, None, None, 0, ctas=1 + i % 3)
            for d, w in zip(dst, want):
                m = 0 if w is None else w.numel()
                assert (w is None or torch.equal(d[:m], w)) and bool((d[m:] == 7).all()), (i, ctas, kind)
    finally:
        g.close()


def test_a_team_that_leaves_pes_out():
    from roc_shmem_b200 import gpu
    from roc_shmem_b200.utils import dtypes as D
    g = gpu.LocalGroup(4, heap_bytes=64 << 20)
    try:
        slots = g.team_split(0, 0, 2, 2)                  # PEs 0 and 2
        src, dst = g.empty((100,), torch.float32), g.empty((100,), torch.float32)
        for pe, (s, d) in enumerate(zip(src, dst)):
            s.fill_(pe + 1)
            d.fill_(9)
        torch.cuda.synchronize()
        g.collective(gpu.COLL_REDUCE, dst, src, 100, dtype=torch.float32, op=D.SUM, team_slot=slots[0], ctas=1)
        assert [float(d[0]) for d in dst] == [4, 9, 4, 9]
    finally:
        g.close()
