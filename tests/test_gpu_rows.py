"""The thread-per-row pass kernel (batch_rows_kernel) against the oracle at
the sizes where it can go wrong: rows around its 1024- and 2048-row blocks
and past one block per CTA, query counts around its quads of 128 slots and
its shapes, every column count, table positions past the lines, bitmaps that
TMA can and cannot write."""
import numpy as np
import pytest

from oracle import oracle as O
from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KINDS = [lambda n, s: D.normal(n, s), lambda n, s: D.zipf(n, s, 1.2), lambda n, s: D.uniform(n, s),
         lambda n, s: D.uniform(n, s, 256), lambda n, s: D.uniform(n, s, 1 << 20), lambda n, s: D.zipf(n, s, 1.5),
         lambda n, s: D.normal(n, s), lambda n, s: D.uniform(n, s, 64)]


def check(ctx, cols, queries, pad_words):
    """Every bitmap and count; pad_words extra words per bitmap stay as they were."""
    n = len(cols[0])
    words = O.words(n)
    stride = (words + 3) // 4 * 4 + pad_words
    out = torch.full((len(queries), stride), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((len(queries),), -1, dtype=torch.int64, device="cuda")
    ctx.scan_batch_async(queries, out.data_ptr(), stride, cnt.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got, cnt = out.cpu().numpy().view(np.uint32), cnt.cpu().numpy()
    for i, q in enumerate(queries):
        if not q:
            want, wcnt = O.mask_tail(np.full(words, 0xFFFFFFFF, np.uint32), n), n
        else:
            want, wcnt = O.range_scan([cols[c] for c, _, _ in q], [t[1] for t in q], [t[2] for t in q])
        assert cnt[i] == wcnt and np.array_equal(got[i, :words], want), (i, q)
    assert (got[:, words:] == 0xFFFFFFFF).all(), "wrote past a bitmap"


@pytest.mark.parametrize("ncols", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("nq,n", [(21, 2047), (128, 2049), (129, 1023), (256, 1025), (300, 4128), (385, 1024),
                                  (512, 2080)])
def test_rows_pass_at_block_edges(ctx, ncols, nq, n):
    cols = [KINDS[c](n, 31 * n + c) for c in range(ncols)]
    ctx.load_columns(cols)
    queries = D.batch_queries(cols, nq, seed=nq + ncols, max_cols=min(ncols, 6))
    check(ctx, cols, queries, 0)


@pytest.mark.parametrize("pad_words", [0, 1])
@pytest.mark.parametrize("nq,ncols", [(100, 3), (200, 3), (384, 3), (500, 3), (300, 6)])
def test_rows_pass_many_blocks(ctx, nq, ncols, pad_words):
    """More than one block per CTA, a last block that is not full, a query in
    the middle that the pass does not hold (bitmaps out of order)."""
    n = 2 * 296 * 2048 + 545
    cols = [KINDS[c](n, 77 + c) for c in range(ncols)]
    ctx.load_columns(cols)
    queries = D.batch_queries(cols, nq, seed=nq)
    if pad_words:
        queries[nq // 2] = []
    check(ctx, cols, queries[:nq], 4 * pad_words)
    check(ctx, cols, queries[:40], pad_words)


def test_rows_pass_positions_past_the_lines(ctx):
    """512 two-sided queries on one column: 1024 boundaries, more than the
    table lines of two CTAs per SM hold."""
    n = 50_003
    cols = [D.normal(n, 5), D.uniform(n, 6, 64)]
    ctx.load_columns(cols)
    s = np.unique(cols[0])
    at = np.linspace(1, len(s) - 2, 1024).astype(int)
    lo, hi = s[at[:512]].astype(int), s[at[512:]].astype(int) - 1
    queries = [[(0, int(a), int(b))] + ([(1, i % 40, 50)] if i % 3 == 0 else []) for i, (a, b) in
               enumerate(zip(lo, hi))]
    check(ctx, cols, queries, 0)


def test_passes_over_different_columns_share_in_groups(ctx):
    """Passes over two sets of columns (the second of more than four), then
    more passes than one group holds."""
    n = 9_001
    cols = [KINDS[c](n, 5 + c) for c in range(8)]
    ctx.load_columns(cols)
    first = D.batch_queries(cols[:2], 512, seed=1, max_cols=2)
    second = [[(2 + c, lo, hi) for c, lo, hi in q] for q in D.batch_queries(cols[2:], 600, seed=2, max_cols=3)]
    check(ctx, cols, first + second, 0)
    check(ctx, cols, D.batch_queries(cols[:3], 512 * 5 + 40, seed=3, max_cols=3), 0)
