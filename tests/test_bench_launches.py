"""The benchmark counts the launches of the step that the handle uses, tuned or not, and its reference arm
answers without the reference.  CPU only."""
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


def test_reference_arm_without_the_reference(monkeypatch, tmp_path, capsys):
    """Where the oracle is not built the reference arm says so in its one line and ends normally."""
    import json

    import bench

    monkeypatch.setattr(bench, "ORACLE_LIB", str(tmp_path / "none.so"))
    monkeypatch.setattr(bench, "GAE_LIB_REF", str(tmp_path / "none.so"))
    for config in ("c3", "gae"):
        monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--config", config])
        bench.main()
        line = json.loads(capsys.readouterr().out)
        assert line["impl"] == "reference" and "not at hand" in line["unavailable"]
