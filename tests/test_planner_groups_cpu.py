"""Batch plans on the CPU: groups of passes that share positions over up to
eight columns, few-query passes as their kernel reads them, consecutive
bitmaps and dropped queries (tests/planner_groups_check.cu)."""
import re
import subprocess

import pytest

from test_planner_cpu import compile_check


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    return compile_check(tmp_path_factory, "planner_groups_check.cu", "batch.cu")


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_plan_groups_few_passes_and_bitmaps(harness, seed):
    r = subprocess.run([harness, str(seed), "80"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    counts = [int(x) for x in re.findall(r"(\d+) (?:groups|over|lookups|direct|table|passes|given)", r.stdout)]
    assert len(counts) == 7 and all(c > 0 for c in counts), r.stdout
