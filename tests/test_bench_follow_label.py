"""The benchmark line names how parent-following steps are taken: with batches
always on it names no build, which the launch plan does not tell then."""
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))


@pytest.mark.parametrize("setting,plan,text", [(1, 0, "off"), (2, 1, "always"), (0, 1, "by colony, one-wave build"),
                                               (0, 2, "by colony, full-panel build")])
def test_follow_batches(setting, plan, text):
    import bench
    assert bench.follow_batches(setting, plan) == text
