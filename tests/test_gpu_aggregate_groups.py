"""Fused scan-and-aggregate around the row groups that a thread takes at a
time (four, two or one of four rows, by the number of columns) and past one
round of the grid."""
import numpy as np
import pytest

from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ncols", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("n", [1, 1023, 1025, 2047, 2049, 4095, 4097, 148 * 32 * 256 * 4 + 1027])
def test_aggregate_row_groups(ctx, n, ncols):
    cols = [D.uniform(n, c + n, 1 << (10 + 2 * c)) for c in range(ncols)]
    ctx.load_columns(cols)
    terms = [(c, 1 << (7 + 2 * c), 7 << (7 + 2 * c)) for c in range(ncols)]
    hit = np.ones(n, bool)
    for c, lo, hi in terms:
        hit &= (cols[c] >= lo) & (cols[c] <= hi)
    a, b = 0, ncols - 1
    cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    out = torch.full((2,), -1, dtype=torch.int64, device="cuda")
    ctx.scan_aggregate_async(terms, a, b, cnt.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    lo, hi64 = (int(x) & (2 ** 64 - 1) for x in out.cpu().tolist())
    want = sum(int(x) * int(y) for x, y in zip(cols[a][hit], cols[b][hit])) if n < 10_000 else \
        int((cols[a][hit].astype(np.uint64) * cols[b][hit].astype(np.uint64)).sum())  # (below 2^64)
    assert int(cnt.item()) == int(hit.sum()) and (lo | hi64 << 64) == want
