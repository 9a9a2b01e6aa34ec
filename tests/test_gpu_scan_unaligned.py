"""Scans around the rules that look at the tiles: a cluster's warps have one
tile each up to 2^17 rows; columns that are not 16-byte aligned run in
rounds of a fixed grid."""
import numpy as np
import pytest

from oracle import oracle as O
from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("n", [(1 << 17) - 1, 1 << 17, (1 << 17) + 1, 148 * 8 * 8 * 1024 + 517])
def test_scan_tile_rules(ctx, n, offset):
    cols = [D.uniform(n + offset, c + n, 1 << (20 + 4 * c)) for c in range(3)]
    dev = [torch.from_numpy(c.view(np.int32)).cuda() for c in cols]
    ctx.attach_columns([d.data_ptr() + 4 * offset for d in dev], n)
    views = [c[offset:] for c in cols]
    words = O.words(n)
    for terms in ([(0, 1 << 17, 1 << 19)], [(1, 5, 1 << 23), (2, 1 << 20, 1 << 28)], [(c, 9, 3 << (18 + 4 * c)) for c in range(3)]):
        want, wcnt = O.range_scan([views[c] for c, _, _ in terms], [t[1] for t in terms], [t[2] for t in terms])
        bm = torch.full((words + 3,), -1, dtype=torch.int32, device="cuda")
        cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
        ctx.scan_async(terms, bm.data_ptr(), cnt.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        got = bm.cpu().numpy().view(np.uint32)
        assert int(cnt.item()) == wcnt and np.array_equal(got[:words], want), terms
        assert (got[words:] == 0xFFFFFFFF).all()
    ctx.load_columns([np.zeros(4, np.uint32)])  # the borrowed columns go
