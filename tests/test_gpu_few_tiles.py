"""Passes of up to 31 queries around the rules of batch_few_kernel: tile
sizes of 128 to 1024 rows on both sides of every line, queries tested by
their terms or through buckets, and columns whose bounds and rows crowd into
one bucket."""
import numpy as np
import pytest

from rtscan_b200 import datagen as D
from test_gpu_rows import KINDS, check

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LINE = 148 * 16 * 128  # rows of one 128-row tile per warp


@pytest.mark.parametrize("ncols", [1, 4, 5, 8])
@pytest.mark.parametrize("n,nq", [(129, 4), (1000, 2), (LINE - 1, 31), (LINE + 1, 5), (2 * LINE + 130, 3),
                                  (2 * LINE - 129, 4), (4 * LINE, 2), (4 * LINE + 1, 4), (4 * LINE + 1025, 12)])
def test_few_pass_tiles(ctx, ncols, n, nq):
    cols = [KINDS[c](n, 3 * n + c) for c in range(ncols)]
    ctx.load_columns(cols)
    check(ctx, cols, D.batch_queries(cols, nq, seed=nq + ncols, min_cols=min(ncols, 4), max_cols=ncols), nq % 4)


@pytest.mark.parametrize("nq", [3, 4, 5, 17, 31])
@pytest.mark.parametrize("n", [5_000, LINE + 77, 4 * LINE + 77])
def test_few_pass_crowded_bounds(ctx, nq, n):
    """Nearly every row and bound within 100 values of 3e9, a few near 0."""
    rng = np.random.default_rng(n + nq)
    cols = [np.where(rng.random(n) < 0.95, 3_000_000_000 + rng.integers(0, 100, n), rng.integers(0, 100, n))
            .astype(np.uint32) for _ in range(4)]
    ctx.load_columns(cols)
    queries = []
    for i in range(nq):
        base = 0 if i % 8 == 7 else 3_000_000_000
        q = []
        for c in range(4):
            a, b = sorted(int(x) for x in rng.integers(0, 100, 2))
            if (i + c) % 3:
                q.append((c, base + a, base + b))
        queries.append(q)
    check(ctx, cols, queries, 0)
