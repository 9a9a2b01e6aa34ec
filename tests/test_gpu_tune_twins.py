"""The autotuner times no launch shape twice: where every table pass reads
shared positions, warps per CTA changes nothing of variant 4."""
import pytest

from rtscan_b200 import datagen as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncols", [3, 6])
def test_autotune_times_each_launch_once(ncols):
    import rtscan_b200 as R
    cols = [D.uniform(60_000, 3 + c) for c in range(ncols)]
    with R.Context(0) as ctx:
        ctx.load_columns(cols)
        ctx.autotune_batch(D.batch_queries(cols, 300, seed=1, max_cols=3))
        rep = ctx.autotune_report()
    shapes = [(c["max_queries_per_pass"], c["table_budget_bytes"]) for c in rep["candidates"] if c["variant"] == 4]
    assert len(shapes) == len(set(shapes)) and len(shapes) >= 17
