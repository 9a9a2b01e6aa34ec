"""Bitmap to row ids around the tiles of the compaction (32768 rows) and past
the tile count up to which the write pass sums the counts itself (2^28 rows),
with buffers that end inside a tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def run(ctx, rows, n, capacity):
    words = np.zeros((n + 31) // 32, np.uint32)
    np.bitwise_or.at(words, rows >> 5, np.uint32(0x80000000) >> (rows & 31).astype(np.uint32))
    bm = torch.from_numpy(words.view(np.int32)).cuda()
    out = torch.full((capacity + 3,), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    ctx.bitmap_rows_async(bm.data_ptr(), n, out.data_ptr(), capacity, cnt.data_ptr(),
                          torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = out.cpu().numpy().view(np.uint32)
    assert int(cnt.item()) == len(rows)
    k = min(capacity, len(rows))
    assert np.array_equal(got[:k], rows[:k].astype(np.uint32))
    assert (got[k:] == 0xFFFFFFFF).all(), "wrote past capacity"


@pytest.mark.parametrize("n", [32767, 32768, 32769, 3 * 32768 + 1023])
@pytest.mark.parametrize("share", [0.002, 0.3, 1.0])
def test_rows_at_tile_edges(ctx, n, share):
    rng = np.random.default_rng(n)
    rows = np.nonzero(rng.random(n) < share)[0]
    for capacity in (len(rows), len(rows) // 2, 0):
        run(ctx, rows, n, capacity)


@pytest.mark.parametrize("tiles", [8192, 8193])
def test_rows_past_the_self_summed_tiles(ctx, tiles):
    n = tiles * 32768 - 7
    rng = np.random.default_rng(tiles)
    rows = np.unique(np.concatenate([rng.integers(0, n, 200_000), [0, n - 1, 32767, 32768]]))
    run(ctx, rows, n, len(rows))
