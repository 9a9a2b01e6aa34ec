"""BinDex builds whose sort scratch lies with the index, in the filter vectors'
place, or apart: few areas on both sides of the size up to which it is kept,
built, rebuilt over each other, and queried."""
import numpy as np
import pytest

from oracle import oracle as O
from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [3_000, 100_000, 160_000, 190_000, 500_001])
def test_bindex_builds_with_few_areas(n):
    import rtscan_b200 as R
    col = D.zipf(n, n, 1.2)
    words = O.words(n)
    with R.Context(0) as ctx:
        ctx.load_columns([col])
        for K in (2, 16, 3, 128, 64, 16):
            ctx.build_bindex(0, K)
            starts, ranks = ctx.bindex_areas(0, K)
            s = np.sort(col)
            assert np.array_equal(np.asarray(starts, np.uint32), s[np.arange(K) * (n // K)])
            for lo, hi in ((0, int(s[n // 3])), (int(s[n // 5]), int(s[n - 1 - n // 7])), (7, 7)):
                bm = torch.full((words,), -1, dtype=torch.int32, device="cuda")
                cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
                ctx.bindex_scan_async([(0, lo, hi)], bm.data_ptr(), cnt.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream)
                torch.cuda.synchronize()
                want, wcnt = O.range_scan([col], [lo], [hi])
                assert int(cnt.item()) == wcnt and np.array_equal(bm.cpu().numpy().view(np.uint32), want), (K, lo, hi)
