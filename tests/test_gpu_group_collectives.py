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
