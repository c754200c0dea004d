"""rsb_autotune behind steps that are still queued on another stream leaves their results alone."""
import numpy as np
import pytest

from gpu_util import random_controls
from test_gpu_step_paths import GETTERS
from test_step_phases import host, start  # noqa: F401  (host: the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [500, 4096])
def test_autotune_behind_queued_steps(pkg, host, n):  # noqa: F811
    torch = pytest.importorskip("torch")
    rsb = pkg.rsb
    x, y = (rsb.Batch(pkg.engine_library(), n, team_size=3, meshes_path=host[1], seed=3) for _ in range(2))
    cars, balls = start(rsb, x, "heap", 7)
    ctl = random_controls(rsb, x.num_cars, np.random.default_rng(1))
    for b in (x, y):
        b.set_balls(balls)
        b.set_cars(cars)
        b.set_controls(ctl)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    x.step(80, stream=stream.cuda_stream)
    x.autotune(2)
    torch.cuda.synchronize()
    y.step(80)
    for g in GETTERS:
        assert getattr(x, g)().tobytes() == getattr(y, g)().tobytes(), g
