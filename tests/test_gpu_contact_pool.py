"""The engine against the host build of the same physics, byte for byte, in arenas with more manifolds
than a tick keeps: batches stepped by one kernel (at the edges of its blocks' shares) and by a kernel
per phase."""
import numpy as np
import pytest

from test_contact_pool import WS_OVERFLOW, crammed
from test_step_phases import host  # noqa: F401  (host: the fixture)

pytestmark = pytest.mark.gpu
GETTERS = ("get_cars", "get_balls", "get_pads", "get_arena_info")


def same_steps(x, y, steps):
    for k, ticks in enumerate(steps):
        for b in (x, y):
            b.step(ticks)
        for g in GETTERS:
            assert getattr(x, g)().tobytes() == getattr(y, g)().tobytes(), f"{g} after step {k}"


@pytest.mark.parametrize("n,pinned", [(1, False), (2, False), (64, False), (65, False), (130, False), (65, True)])
@pytest.mark.parametrize("place", ["corner", "post"])
def test_more_manifolds_than_a_tick_keeps(pkg, host, n, pinned, place):  # noqa: F811
    rsb, (lib, arena) = pkg.rsb, host
    x, y = (rsb.Batch(w, n, team_size=3, meshes_path=arena, seed=5) for w in (lib, pkg.engine_library()))
    cars, balls = crammed(rsb, x, place, n, np.arange(1, n, 4))
    for b in (x, y):
        b.set_balls(balls)
        b.set_cars(cars)
    if pinned:
        y.set_step_config(3, 64)
    same_steps(x, y, (1, 1, 8))
    assert (x.get_arena_info()["status"] & WS_OVERFLOW).any()


def test_every_arena_of_a_large_batch(pkg, host):  # noqa: F811
    """A kernel per phase: 64 starts with more manifolds than a tick keeps, repeated."""
    rsb, (lib, arena) = pkg.rsb, host
    n = 64 * 64
    x, y = (rsb.Batch(w, n, team_size=3, meshes_path=arena, seed=5) for w in (lib, pkg.engine_library()))
    one = rsb.Batch(lib, 64, team_size=3, meshes_path=arena, seed=5)
    cars, balls = crammed(rsb, one, "corner", 3)
    for b in (x, y):
        b.set_balls(np.tile(balls, n // 64))
        b.set_cars(np.tile(cars, n // 64))
    same_steps(x, y, (1, 1, 2))
    assert (x.get_arena_info()["status"] & WS_OVERFLOW).all()
