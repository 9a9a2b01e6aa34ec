"""Passes of up to 31 queries (batch_few_kernel) against the oracle: rows
around its 1024-row tiles, the query counts of its range, every column count,
aligned and unaligned columns, bounds crowded into one bucket and at the ends
of the domain with rows on and beside them."""
import numpy as np
import pytest

from rtscan_b200 import datagen as D
from test_gpu_rows import KINDS, check

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ncols", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("nq,n", [(2, 1023), (4, 1025), (16, 4096), (31, 2080), (20, 33)])
def test_few_pass_sizes(ctx, ncols, nq, n):
    cols = [KINDS[c](n, 13 * n + c) for c in range(ncols)]
    ctx.load_columns(cols)
    check(ctx, cols, D.batch_queries(cols, nq, seed=nq + ncols, min_cols=min(ncols, 3), max_cols=ncols), nq % 4)


@pytest.mark.parametrize("offset", [0, 1, 2])
def test_few_pass_many_tiles(ctx, offset):
    """More than one tile per warp, columns at every 4-byte offset."""
    n = 148 * 2 * 16 * 1024 + 12_345
    cols = [KINDS[c](n + offset, 7 + c) for c in range(3)]
    dev = [torch.from_numpy(c.view(np.int32)).cuda() for c in cols]
    views = [c[offset:] for c in cols]
    ctx.attach_columns([d.data_ptr() + 4 * offset for d in dev], n)
    check(ctx, views, D.batch_queries(views, 9, seed=offset, min_cols=2, max_cols=3), 0)
    ctx.load_columns([np.zeros(4, np.uint32)])  # the borrowed columns go


def test_few_pass_bounds_in_one_bucket_and_at_the_ends(ctx):
    rng = np.random.default_rng(3)
    top = 0xFFFFFFFF
    edges = np.array([0, 1, 2, 3, 1 << 20, (1 << 20) + 1, (1 << 20) + 2, (1 << 31) - 1, 1 << 31, top - 2, top - 1, top],
                     dtype=np.uint64)
    col = rng.choice(np.concatenate([edges, edges + 1, edges - (edges > 0)]) & top, size=20_000).astype(np.uint32)
    cols = [col, rng.permutation(col)]
    ctx.load_columns(cols)
    queries = []
    for i in range(30):
        a, b = sorted(int(x) for x in rng.choice(edges, 2))
        q = [(i % 2, a, b)]
        if i % 3 == 0:
            q.append((1 - i % 2, int(edges[i % 6]), int(edges[6 + i % 6])))
        queries.append(q)
    check(ctx, cols, queries, 0)
    check(ctx, cols, [[(0, int(v), int(v))] for v in edges] + [[(0, 5, top)], [(0, 0, 7)]], 0)
