"""bench.full_count_roofline on a graph whose degrees 1..32 are one launch: its
bytes are those of all three small tiers."""
import os
import sys
from types import SimpleNamespace

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def _roof(times):
    plan = {f"{c}_{k}": 0 for c in "ve" for k in ("tiny", "group16", "group32", "mid", "big", "hub")}
    plan.update(v_tiny=100, e_tiny=400, v_group16=50, e_group16=600, v_group32=10, e_group32=250)
    st = np.zeros((2, 8), dtype=np.float32)
    st[1, :3] = times
    run = SimpleNamespace(changed=np.array([1000, 1000]), step_tier_ms=st)
    return bench.full_count_roofline(plan, [run], 1000, 6000.0)


def test_one_launch_counts_the_bytes_of_every_small_tier():
    assert _roof([0, 0, 1.0])["bytes_per_launch"] == 8 * 1250 + 12 * 160


def test_three_launches_count_their_own():
    groups = _roof([0.25, 0.5, 1.0])["groups"]
    assert [groups[k]["bytes_per_launch"] for k in ("tiny", "group16", "group32")] == [4400, 5400, 2120]
