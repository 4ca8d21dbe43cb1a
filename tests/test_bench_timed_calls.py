"""The bench's bandwidth of the shortlist sums does not depend on how many calls were timed: the
proposal's statistics count one call, the kernel's time all of them."""
import os
import sys
from types import SimpleNamespace

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


@pytest.mark.parametrize("steps", [1, 3, 20])
def test_bandwidth_of_the_shortlist_sums(steps):
    import bench
    W = bench.workload("cfg3")
    st = {"cols_shortlist": 100.0, "mean_shortlist": 8000.0}
    per_call = 40.0  # ms
    r = bench.proposal_roofline("lp.pick", {"lp.pick": (per_call * steps, 10 * steps, 0.0)}, {}, W,
                                {"hbm_gbs": 6000.0}, "measured", st, SimpleNamespace(steps=steps))
    offsets = 32 * 32 * 16 - 24 * 24 * 12  # interior mask of a 32 x 32 x 16 tile, overlap 1/4
    assert r["achieved"] == pytest.approx(100 * 8000 * offsets * 0.25 / (per_call / 1e3) / 1e9)
