"""Group collectives of at most eight blocks of all PEs together against the same call with more blocks, at odd sizes, for every kind, with results in place of the sources, and in a team that leaves PEs out."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pes,ctas", [(2, 1), (2, 4), (3, 2), (5, 1), (8, 1)])
@pytest.mark.parametrize("n", [1, 7, 1024, 1031, 4096, 40001])
def test_cluster_and_cooperative_launch_agree(pes, ctas, n):
    from roc_shmem_b200 import gpu
    from roc_shmem_b200.utils import dtypes as D
    g = gpu.LocalGroup(pes, heap_bytes=64 << 20)
    try:
        torch.manual_seed(n + pes)
        many = 8 // pes + 1                               # blocks per PE that no longer fit
        kinds = [(gpu.COLL_REDUCE, n, n, n), (gpu.COLL_REDUCE_SCATTER, n * pes, n, n), (gpu.COLL_FCOLLECT, n, n * pes, n * 4),
                 (gpu.COLL_ALLTOALL, n * pes, n * pes, n * 4), (gpu.COLL_BROADCAST, n, n, n * 4), (gpu.COLL_REDUCE_ROOT, n, n, n)]
        for dtype, op in ((torch.float32, D.SUM), (torch.int32, D.MAX), (torch.float32, D.PROD)):
            for kind, n_src, n_dst, count in kinds:
                src, one, two = g.empty((n_src,), dtype), g.empty((n_dst + 1,), dtype), g.empty((n_dst + 1,), dtype)
                for s in src:
                    s.copy_((torch.randn(n_src, device="cuda") * 100).to(dtype))
                for t in one + two:
                    t.fill_(7)
                torch.cuda.synchronize()
                g.collective(kind, one, src, count, dtype=dtype, op=op, root=pes - 1, ctas=ctas)
                g.collective(kind, two, src, count, dtype=dtype, op=op, root=pes - 1, ctas=many)
                for a, b in zip(one, two):
                    assert torch.equal(a, b) and bool((a[n_dst:] == 7).all())
                if kind == gpu.COLL_REDUCE:               # in place, several calls in a row
                    for _ in range(2):
                        for s, d in zip(src, two):
                            d[:n].copy_(s)
                        torch.cuda.synchronize()
                        g.collective(kind, two, two, count, dtype=dtype, op=op, ctas=ctas)
                        for a, b in zip(one, two):
                            assert torch.equal(a, b)
                for pe, rt in enumerate(g.pes):
                    for t in (src[pe], one[pe], two[pe]):
                        rt.free(t, collective=False)
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
