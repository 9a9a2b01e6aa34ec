"""Separate-pass scans of one context on several streams at once: the bitmap
that their later terms go through is one."""
import numpy as np
import pytest

from oracle import oracle as O
from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_separate_scans_on_many_streams():
    import rtscan_b200 as R
    n = 20_000_003
    cols = [D.uniform(n, c, 1 << (10 + 3 * c)) for c in range(4)]
    words = O.words(n)
    rng = np.random.default_rng(5)
    jobs = []
    for i in range(6):
        terms = []
        for c in rng.permutation(4)[:2 + i % 3]:
            a, b = sorted(int(x) for x in rng.integers(0, 1 << (10 + 3 * int(c)), 2))
            terms.append((int(c), a, b))
        jobs.append((terms, O.range_scan([cols[c] for c, _, _ in terms], [t[1] for t in terms], [t[2] for t in terms]),
                     torch.empty(words, dtype=torch.int32, device="cuda"),
                     torch.empty(1, dtype=torch.int64, device="cuda"), torch.cuda.Stream()))
    with R.Context(0) as ctx:
        ctx.load_columns(cols)
        for _ in range(3):
            for _, _, bm, cnt, _ in jobs:
                bm.fill_(-1)
                cnt.fill_(-1)
            torch.cuda.synchronize()
            for terms, _, bm, cnt, s in jobs:
                ctx.scan_separate_async(terms, bm.data_ptr(), cnt.data_ptr(), s.cuda_stream)
            torch.cuda.synchronize()
            for terms, (want, wcnt), bm, cnt, _ in jobs:
                assert int(cnt.item()) == wcnt and np.array_equal(bm.cpu().numpy().view(np.uint32), want), terms
