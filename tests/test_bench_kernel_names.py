"""The bench takes profiled figures only for a kernel that was profiled: not for
the CTAs that the automatic choice takes on small grids (no GPU needed)."""
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("kind,asked,n,name", [
    ("tile", "auto", 64, "k_stage_pf/small"), ("tile", "auto", 256, "k_stage_pf/small"),
    ("tile", "auto", 264, "k_stage_pf/32x8"), ("tile", "tile", 64, "k_stage_pf/32x8"),
    ("tile32", "auto", 320, "k_stage_pf/32x32"), ("strip", "strip", 64, "k_stage_strip")])
def test_small_grids_have_no_profiled_figures(kind, asked, n, name):
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    assert bench.kernel_name(kind, asked, n, 148) == name
    assert (bench.profiled_traffic(name) is None) == (name == "k_stage_pf/small")
