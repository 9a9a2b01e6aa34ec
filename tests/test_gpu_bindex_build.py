"""BinDex builds at the edges of the filter-vector kernel's area table (64
areas) and of the sort's bit range, on columns at every 4-byte offset and
row counts around a word and a warp's 1024 rows."""
import numpy as np
import pytest

from oracle import oracle as O
from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def check_index(ctx, col, K):
    ob = O.BinDex(col, K=K)
    starts, ranks = ctx.bindex_areas(0, K)
    assert np.array_equal(starts, ob.area_start_values())
    assert np.array_equal(ranks, np.searchsorted(np.sort(col), starts, side="left").astype(np.uint64))
    for k in sorted({0, K // 3, min(62, K - 2), min(63, K - 2), min(64, K - 2), K - 2}):
        assert np.array_equal(ctx.bindex_filter_vector(0, k), ob.filter_vector(k)), k


@pytest.mark.parametrize("K", [2, 3, 64, 65, 66, 128, 129, 130, 257, 4096])
def test_filter_vectors_at_table_edges(ctx, K):
    col = np.concatenate([D.zipf(9_000, K, 1.1), D.uniform(1_003, K)])
    ctx.load_columns([col])
    ctx.build_bindex(0, K)
    check_index(ctx, col, K)


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [31, 32, 1023, 1025, 70_001])
def test_builds_of_unaligned_columns(ctx, offset, n):
    col = D.uniform(n + offset, n)
    dev = torch.from_numpy(col.view(np.int32)).cuda()
    ctx.attach_columns([dev.data_ptr() + 4 * offset], n)
    ctx.build_bindex(0, 16)
    check_index(ctx, col[offset:], 16)
    ctx.load_columns([np.zeros(4, np.uint32)])  # the borrowed column goes


@pytest.mark.parametrize("top", [0, 1, 255, 256, (1 << 24) - 1, 1 << 24, 0xFFFFFFFF])
def test_sorts_of_every_width(ctx, top):
    rng = np.random.default_rng(7)
    col = rng.integers(0, top + 1, 40_000, dtype=np.uint64).astype(np.uint32)
    col[123] = top
    ctx.load_columns([col])
    ctx.build_bindex(0, 32)
    check_index(ctx, col, 32)
    ctx.build_bindex(0, 32)  # again, over the index that is there
    check_index(ctx, col, 32)
    ctx.build_bindex(0, 100)
    check_index(ctx, col, 100)
