"""Host-buffer batches whose dense queries lie between packed ones: their
words wait for later chunks, leave when the query turns sparse, at the end
of a group of chunks and at the end; queries answered outside the passes
and runs of dense ones among them."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [70, 141])
@pytest.mark.parametrize("n", [(1 << 20) + 5, 3 * (1 << 20) + 77, 6 * (1 << 20) + 31, 8 * (1 << 20) + 9])
def test_host_batch_alternating_densities(ctx, n, nq):
    rng = np.random.default_rng(n + nq)
    # column 0: noise; column 1: eight plateaus, so a query on it is dense in some chunks only
    cols = [rng.integers(0, 1000, n).astype(np.uint32), (np.arange(n) * 8 // n * 1000 + rng.integers(0, 1000, n)).astype(np.uint32)]
    queries = []
    for i in range(nq):
        if i % 23 == 11:
            queries.append([])
        elif i % 2 == 0:
            a = int(rng.integers(0, 6))
            queries.append([(1, 1000 * a, 1000 * a + 1500)] if i % 4 else [(0, 0, 500 + i)])
        else:
            queries.append([(0, i, i), (1, 0, 10)] if i % 3 else [(0, 400, 900 if i % 9 else 401)])
    words = O.words(n)
    out = np.full((nq, words + 2), 0xFFFFFFFF, np.uint32)
    got, counts = ctx.scan_batch_host(cols, queries, out, words + 2)
    for i, q in enumerate(queries):
        if not q:
            want, wcnt = O.mask_tail(np.full(words, 0xFFFFFFFF, np.uint32), n), n
        else:
            want, wcnt = O.range_scan([cols[c] for c, _, _ in q], [t[1] for t in q], [t[2] for t in q])
        assert counts[i] == wcnt and np.array_equal(got[i, :words], want), (i, q)
    assert (got[:, words:] == 0xFFFFFFFF).all()
