"""The engine's step and ball prediction against the host build of the same physics, byte for byte,
on a generated arena: batches stepped by one kernel and by a kernel per phase, at the edges of the
blocks' shares and of the rule between the two, and predictions at the edges of a warp's share.

The physics is compiled once for both (no contraction, restated float functions), so nothing may
differ."""
import numpy as np
import pytest

from gpu_util import random_controls
from test_step_phases import host, start  # noqa: F401  (host: the fixture)

pytestmark = pytest.mark.gpu
GETTERS = ("get_cars", "get_balls", "get_pads", "get_arena_info")


def pair(pkg, host, n, kind, seed):  # noqa: F811
    rsb, (lib, arena) = pkg.rsb, host
    teams = np.array([3, 1, 2, 0, 3], np.int32)[np.arange(n) % 5]
    x, y = (rsb.Batch(w, n, team_sizes=teams, meshes_path=arena, seed=seed) for w in (lib, pkg.engine_library()))
    cars, balls = start(rsb, x, kind, seed)
    for b in (x, y):
        b.set_balls(balls)
        b.set_cars(cars)
    return rsb, x, y


@pytest.mark.parametrize("n,pinned", [(1, False), (32, False), (63, False), (65, False), (1023, False), (2048, False),
                                      (2049, False), (65, True)])
@pytest.mark.parametrize("kind", ["walls", "heap"])
def test_step_paths(pkg, host, n, pinned, kind):  # noqa: F811
    rsb, x, y = pair(pkg, host, n, kind, 17 + n)
    if pinned:
        y.set_step_config(3, 64)
    rng = np.random.default_rng(n)
    for k, ticks in enumerate((1, 8, 3, 8)):
        ctl = random_controls(rsb, x.num_cars, rng)
        for b in (x, y):
            b.set_controls(ctl)
            b.step(ticks)
        for g in GETTERS:
            assert getattr(x, g)().tobytes() == getattr(y, g)().tobytes(), f"{g} after step {k}"


@pytest.mark.parametrize("n", [1, 33, 297, 1185])
def test_predictions_are_the_ball_alone(pkg, host, n):  # noqa: F811
    rsb, x, y = pair(pkg, host, n, "walls", 3 + n)
    got = y.predict_ball((1, 60, 200))
    # the same balls in arenas without cars; balls of arenas whose goals reset them stay out of the compare
    lib, arena = host
    z = rsb.Batch(lib, n, team_sizes=np.zeros(n, np.int32), meshes_path=arena)
    z.set_balls(x.get_balls())
    at = 0
    for k, t in enumerate((1, 60, 200)):
        z.step(t - at)
        at = t
        want = z.get_balls()
        assert got[:, k].tobytes() == want.tobytes(), f"after {t} ticks"
