"""Host-buffer batches whose chunks are packed by clusters: word counts that
are no multiple of the cluster's shares, one and several chunks, queries from
empty to dense, bitmaps at a stride of their own."""
import numpy as np
import pytest

from oracle import oracle as O
from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096 * 32, 4097 * 32 + 1, 300_001, (1 << 21) + 4097 * 32 + 5])
def test_host_batch_packs_what_the_scan_found(ctx, n):
    rng = np.random.default_rng(n)
    # runs of equal values: bitmaps with long runs of zero words beside dense ones
    cols = [np.repeat(D.uniform(n // 500 + 1, n, 1000), 500)[:n].copy(), D.uniform(n, n + 1)]
    queries = [[(0, int(a), int(a + w))] for a, w in zip(rng.integers(0, 900, 25), rng.integers(0, 60, 25))]
    queries += [[(0, 0, 400), (1, 0, int(h))] for h in rng.integers(0, 1 << 32, 12, dtype=np.uint64)]
    queries += [[(0, 2000, 3000)], [(1, 0, 3)], []]
    words = O.words(n)
    out = np.full((len(queries), words + 3), 0xFFFFFFFF, np.uint32)
    got, counts = ctx.scan_batch_host(cols, queries, out, words + 3)
    for i, q in enumerate(queries):
        if not q:
            want, wcnt = O.mask_tail(np.full(words, 0xFFFFFFFF, np.uint32), n), n
        else:
            want, wcnt = O.range_scan([cols[c] for c, _, _ in q], [t[1] for t in q], [t[2] for t in q])
        assert counts[i] == wcnt and np.array_equal(got[i, :words], want), (i, q)
    assert (got[:, words:] == 0xFFFFFFFF).all()
