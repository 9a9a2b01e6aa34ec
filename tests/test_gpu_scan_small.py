"""Scans on both sides of the small-table rule (one cluster up to 2^19
values), with every number of CTAs in the cluster and of terms, on aligned
and unaligned columns; the count is stored whatever was there before."""
import numpy as np
import pytest

from oracle import oracle as O
from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 1023, 1025, 7 * 1024, 8 * 1024 + 1, 70_001, (1 << 19), (1 << 19) + 1])
def test_small_scans(ctx, n, offset):
    cols = [D.uniform(n + offset, c + n, [1 << 32, 256, 1 << 20, 64, 1 << 32][c]) for c in range(5)]
    dev = [torch.from_numpy(c.view(np.int32)).cuda() for c in cols]
    ctx.attach_columns([d.data_ptr() + 4 * offset for d in dev], n)
    views = [c[offset:] for c in cols]
    words = O.words(n)
    for terms in ([(0, 1 << 30, 3 << 30)], [(1, 10, 200), (2, 0, 1 << 19)], [(0, 5, 1 << 31), (1, 0, 99), (3, 7, 60)],
                  [(0, 0, 3 << 30), (1, 0, 99), (2, 9, 1 << 19), (3, 1, 60), (4, 0, 1 << 31)], [(1, 300, 400)]):
        want, wcnt = O.range_scan([views[c] for c, _, _ in terms], [t[1] for t in terms], [t[2] for t in terms])
        bm = torch.full((words + 3,), -1, dtype=torch.int32, device="cuda")
        cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
        for _ in range(2):
            ctx.scan_async(terms, bm.data_ptr(), cnt.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        got = bm.cpu().numpy().view(np.uint32)
        assert int(cnt.item()) == wcnt and np.array_equal(got[:words], want), terms
        assert (got[words:] == 0xFFFFFFFF).all()
    ctx.load_columns([np.zeros(4, np.uint32)])  # the borrowed columns go
