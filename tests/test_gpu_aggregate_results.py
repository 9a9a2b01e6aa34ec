"""Fused scan-and-aggregate with only one of its results asked for: the count
alone, the sum alone, both; 16-byte and 4-byte loads; one block, blocks that
do not fill the grid, and several rounds of it."""
import numpy as np
import pytest

from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("want_count,want_sum", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("n", [5, 100_003, 148 * 16 * 256 * 8 + 4099])
def test_aggregate_one_result(ctx, n, want_count, want_sum, offset):
    cols = [D.uniform(n + offset, c + n, 1 << (12 + c)) for c in range(3)]
    dev = [torch.from_numpy(c.view(np.int32)).cuda() for c in cols]
    cols = [c[offset:] for c in cols]
    ctx.attach_columns([d.data_ptr() + 4 * offset for d in dev], n)
    terms = [(c, 1 << (9 + c), 7 << (9 + c)) for c in range(3)]
    hit = np.ones(n, bool)
    for c, lo, hi in terms:
        hit &= (cols[c] >= lo) & (cols[c] <= hi)
    cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    out = torch.full((2,), -1, dtype=torch.int64, device="cuda")
    ctx.scan_aggregate_async(terms, 0 if want_sum else -1, -1, cnt.data_ptr() if want_count else 0,
                             out.data_ptr() if want_sum else 0)
    torch.cuda.synchronize()
    assert int(cnt.item()) == (int(hit.sum()) if want_count else -1)
    want = [int(cols[0][hit].astype(np.uint64).sum()), 0] if want_sum else [-1, -1]
    assert out.cpu().tolist() == want
    ctx.load_columns([np.zeros(4, np.uint32)])  # the borrowed columns go
