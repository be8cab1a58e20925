"""Collectives of a local group as one pass over all members' memory, against the same call through the entry whose PEs exchange flags
(the multi-PE algorithms): every kind, type and operator, at sizes around vectors, blocks and unrolled rounds, off 16-byte boundaries, in
place, for several numbers of members and blocks, and in a team that leaves PEs out.  Same order of the sums: the same bits."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

FLOATS, INTS = [torch.float32, torch.float64, torch.float16, torch.bfloat16], [torch.int8, torch.uint8, torch.int16, torch.int32, torch.int64]


class Both:
    def __init__(self, pes):
        from roc_shmem_b200 import gpu
        from roc_shmem_b200.utils import dtypes as D
        self.gpu, self.D, self.pes = gpu, D, pes
        self.g = gpu.LocalGroup(pes, heap_bytes=192 << 20)
        self.handles = (C.c_void_p * pes)(*[rt.h.value for rt in self.g.pes])
        self.exchanging = self.g.lib.bshmem_gpu_group_collective_noalloc
        vp, i, u = C.c_void_p, C.c_int, C.c_uint64
        self.exchanging.restype, self.exchanging.argtypes = i, [C.POINTER(vp), i, i, i, i, i, i, u, u, u, i]
        self.src, self.one, self.two = (self.g.empty((24 << 20,), torch.uint8) for _ in range(3))
        torch.manual_seed(pes)

    def views(self, bufs, dtype, start, n):
        es = torch.empty(0, dtype=dtype).element_size()
        return [b[start:start + max(n, 1) * es].view(dtype) for b in bufs]

    def check(self, kind, dtype, op, n, ctas, start=0, root=0, slot=0, members=None):
        """The call both ways from the same sources; all of both destinations is compared."""
        g, m = self.g, len(members) if members else self.pes
        es = torch.empty(0, dtype=dtype).element_size()
        top = n * m * es + start + 256
        assert top <= self.src[0].numel()
        for s, a, b in zip(self.src, self.one, self.two):
            v = self.views([s], dtype, start, n * m)[0]
            if dtype.is_floating_point:
                v.copy_(torch.randn(v.shape, device="cuda"))
            else:
                v.copy_(torch.randint(-100, 100, v.shape, device="cuda").to(dtype))
            a[:top].fill_(77)
            b[:top].fill_(77)
        reduces = kind in (self.gpu.COLL_REDUCE, self.gpu.COLL_REDUCE_SCATTER, self.gpu.COLL_REDUCE_ROOT)
        count = n if reduces else n * es
        off = [self.g.pes[0].offset_of(t[0]) + start for t in (self.src, self.one, self.two)]
        torch.cuda.synchronize()
        code = self.D.code_of(dtype)
        src, one, two = (self.views(t, dtype, start, n * m) for t in (self.src, self.one, self.two))
        rest = dict(dtype=dtype, op=op, root=root, team_slot=slot)
        rooted = kind == self.gpu.COLL_REDUCE_ROOT         # which that entry does not know: an allreduce, seen at the root only
        told = self.gpu.COLL_REDUCE if rooted else kind
        assert self.exchanging(self.handles, self.pes, slot, told, code, op, root, off[2], off[0], count, ctas) == 0
        for pe, b in enumerate(self.two):
            if rooted and pe != (members or range(self.pes))[root]:
                b[:top].fill_(77)
        g.collective(kind, one, src, count, ctas=ctas, **rest)
        for pe, (a, b) in enumerate(zip(self.one, self.two)):
            assert torch.equal(a[:top], b[:top]), (kind, dtype, op, n, ctas, start, root, pe)

    def close(self):
        self.g.close()


@pytest.fixture(scope="module", params=[1, 2, 3, 4, 5, 7, 8, 9])
def both(request):
    b = Both(request.param)
    yield b
    b.close()


def test_reductions(both):
    gpu, D = both.gpu, both.D
    for dtype in FLOATS + INTS:
        ops = [D.SUM, D.MIN, D.MAX, D.PROD] + ([] if dtype.is_floating_point else [D.AND, D.OR, D.XOR])
        for i, op in enumerate(ops):
            for kind in (gpu.COLL_REDUCE, gpu.COLL_REDUCE_SCATTER):
                for n, ctas in ((1, 1), (8 * 512 * (1 + i % 3) + 13, 2)):
                    both.check(kind, dtype, op, n, ctas)
            both.check(gpu.COLL_REDUCE_ROOT, dtype, op, 5000 + i, 3, root=both.pes - 1)


@pytest.mark.parametrize("n", [0, 15, 16 * 511, 16 * 513 + 1, 300_001])
def test_sizes_and_alignments(both, n):
    gpu, D = both.gpu, both.D
    for start in (0, 4):                                   # the second is off every 16-byte boundary
        for ctas in (1, 3, 148 // both.pes):
            for dtype in (torch.float32, torch.bfloat16):
                for kind in (gpu.COLL_REDUCE, gpu.COLL_REDUCE_SCATTER, gpu.COLL_REDUCE_ROOT):
                    both.check(kind, dtype, D.SUM, n, ctas, start)
            for kind in (gpu.COLL_FCOLLECT, gpu.COLL_ALLTOALL, gpu.COLL_BROADCAST):
                both.check(kind, torch.uint8, 0, n, ctas, start, root=both.pes // 2)


def test_results_in_place_of_the_sources(both):
    gpu, D = both.gpu, both.D
    n = 100_003
    for ctas in (1, 5):
        for s in both.views(both.src, torch.float32, 0, n):
            s.copy_(torch.randn(n, device="cuda"))
        want = both.views(both.src, torch.float32, 0, n)
        total = want[0].clone()
        for w in want[1:]:
            total += w                                     # in team order, as the collective adds
        torch.cuda.synchronize()
        both.g.collective(gpu.COLL_REDUCE, want, want, n, dtype=torch.float32, op=D.SUM, ctas=ctas)
        assert all(torch.equal(w, total) for w in want)


def test_a_team_that_leaves_pes_out(both):
    gpu, D = both.gpu, both.D
    if both.pes < 4:
        pytest.skip("needs PEs to leave out")
    slots = both.g.team_split(0, 1, 2, both.pes // 2)      # the odd PEs
    for kind in (gpu.COLL_REDUCE, gpu.COLL_REDUCE_SCATTER, gpu.COLL_FCOLLECT, gpu.COLL_ALLTOALL, gpu.COLL_BROADCAST, gpu.COLL_REDUCE_ROOT):
        both.check(kind, torch.float32, D.SUM, 3001, 2, root=both.pes // 2 - 1, slot=slots[1], members=list(range(1, both.pes, 2)))


@pytest.mark.parametrize("n", [16, 16 * 7, 16 * 512, 16 * 4095, 16 * 4097, 16 * 100_003])
def test_alltoall_of_whole_vectors(both, n):
    """Blocks of whole vectors are moved as one range per block of the launch: from fewer vectors than threads to several rounds of it."""
    for start in (0, 4, 16):
        for ctas in (1, 3, 148 // both.pes):
            both.check(both.gpu.COLL_ALLTOALL, torch.uint8, 0, n, ctas, start)
