"""The launch configuration that a handle uses can be read, kept and pinned again: the one-kernel step of
small batches too, which is the default there."""
import numpy as np
import pytest

from gpu_util import random_controls
from test_gpu_step_paths import GETTERS, pair
from test_step_phases import host  # noqa: F401  (host: the fixture)

pytestmark = pytest.mark.gpu
ONE = {"min_blocks": 1, "block": 256, "persistent": False, "warps_per_sm": 0}


@pytest.mark.parametrize("n", [65, 2048, 2049])
def test_configurations_are_named(pkg, host, n):  # noqa: F811
    rsb, x, y = pair(pkg, host, n, "walls", 5)
    default = y.step_config()
    assert (default == ONE) == (n <= 2048)
    y.set_step_config(3, 32, True, 0)
    assert y.step_config() == {"min_blocks": 3, "block": 32, "persistent": True, "warps_per_sm": 0}
    if n > 2048:
        with pytest.raises(rsb.RsbError):
            y.set_step_config(**ONE)
        assert y.step_config()["block"] == 32
    y.set_step_config(**default)
    assert y.step_config() == default
    rows = y.autotune(8)
    assert len(rows) == 28
    kept = y.step_config()
    assert kept == default or kept in [{k: type(ONE[k])(r[k]) for k in ONE} for r in rows]
    y.set_step_config(**kept)
    assert y.step_config() == kept
    x.set_controls(ctl := random_controls(rsb, x.num_cars, np.random.default_rng(n)))
    y.set_controls(ctl)
    for b in (x, y):
        b.step(8)
    for g in GETTERS:
        assert getattr(x, g)().tobytes() == getattr(y, g)().tobytes(), g
