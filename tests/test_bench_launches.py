"""The benchmark counts the launches of the step that the handle uses, tuned or not.  CPU only."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


@pytest.mark.parametrize("block,want", [(256, 1), (32, 96), (64, 96), (128, 96)])
def test_launches_follow_the_configuration(block, want):
    import bench

    class Batch:
        def step_config(self):
            return {"min_blocks": 1, "block": block, "persistent": False, "warps_per_sm": 0}

    assert bench.step_launches(Batch(), 8) == want
