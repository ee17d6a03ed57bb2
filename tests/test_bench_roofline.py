"""The 2D roofline entry of bench.py counts what a stage computes, not launches."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


@pytest.mark.parametrize("kind,key,skip", [("rec", "rec_per_cell", 4), ("flux", "flux_per_face", 5)])
@pytest.mark.parametrize("launches", [1, 2])
def test_2d_roofline_counts_both_directions(kind, key, skip, launches):
    import bench
    n, steps, ms = 512, 20, 30.0
    opc = bench.load_opcounts()["lhlld_wcns4_2d"]
    timing = {kind: (3 * steps * launches, ms), "prim": (3 * steps, 1.0)}
    r = bench.roofline_2d(timing, n, 3 * steps, 1.25e12, opc)
    flops = 3 * steps * 2 * opc[key] * (n + 8 - skip) * (n + 8)
    assert r["kernel"] == kind
    assert r["achieved"] == pytest.approx(flops / (ms * 1e-3) / 1e12)
    assert r["frac"] == pytest.approx(r["achieved"] / 1.25)
