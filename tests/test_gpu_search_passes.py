"""Table passes that search their own positions (no memory for shared ones)
against the terms row by row: every slot shape, 8- and 16-warp blocks, up to
four and up to eight columns (tests/search_passes_check.cu)."""
import subprocess

import pytest

from test_planner_cpu import compile_check

pytestmark = pytest.mark.gpu


def test_passes_that_search_their_positions(tmp_path_factory):
    check = compile_check(tmp_path_factory, "search_passes_check.cu", "batch.cu")
    r = subprocess.run([check, "1"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "search passes ok: 150 cases" in r.stdout, (r.returncode, r.stderr[-3000:])
