"""Bitmap to row ids on both sides of the compaction's rules: blocks of one and
of four tiles, the block count up to which the write pass sums the counts
itself, and words taken a lane at a time or a bit at a time."""
import numpy as np
import pytest

from test_gpu_compact import run

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("tiles", [4735, 4736, 4739, 32768, 32769])
def test_rows_blocks_of_tiles(ctx, tiles):
    n = tiles * 32768 - 5
    rng = np.random.default_rng(tiles)
    some = rng.integers(0, n, 100_000)
    runs = (rng.integers(0, n - 9000, 20)[:, None] + np.arange(9000)).ravel()  # dense stretches over tile edges
    rows = np.unique(np.concatenate([some, runs, [0, n - 1, 32767, 32768]]))
    for capacity in (len(rows), len(rows) - 12_345):
        run(ctx, rows, n, capacity)


@pytest.mark.parametrize("share", [0.02, 0.5, 0.72, 0.75, 0.98])
def test_rows_on_both_sides_of_the_dense_rule(ctx, share):
    n = 5 * 32768 + 100
    rng = np.random.default_rng(int(share * 100))
    rows = np.nonzero(rng.random(n) < share)[0]
    for capacity in (len(rows), len(rows) - 1, len(rows) // 3):
        run(ctx, rows, n, capacity)
