"""Ball prediction where a ball's triangle list is full (96 triangles) and where a
warp holds 32 balls: the host form of its tick against the ball-only arena, and the kernel against the
host build, byte for byte."""
from __future__ import annotations

import os
import struct

import numpy as np
import pytest

from gpu_util import random_balls
from test_step_phases import host  # noqa: F401  (the fixture)

FULL_WARPS = 2  # warps per SM: with that many full ones and more balls, every warp takes 32


@pytest.fixture(scope="module")
def patch(tmp_path_factory):
    """An arena whose one mesh is a bumpy patch of 968 triangles of 24 uu: in the box of a ball over its
    middle more than a list holds, over its edge fewer."""
    rng = np.random.default_rng(3)
    n, step = 23, 24.0
    xy = (np.arange(n) - (n - 1) / 2) * step
    v = np.array([(x, y, 150 + rng.uniform(0, 30)) for x in xy for y in xy], np.float32) / np.float32(50)
    t = np.array([k for i in range(n - 1) for j in range(n - 1) for a in (i * n + j,)
                  for k in ((a, a + n, a + 1), (a + 1, a + n, a + n + 1))], np.int32)
    d = tmp_path_factory.mktemp("patch")
    os.mkdir(d / "soccar")
    (d / "soccar" / "mesh_0.cmf").write_bytes(struct.pack("<ii", len(t), len(v)) + t.tobytes() + v.tobytes())
    return str(d)


def over_the_patch(rsb, n):
    rng = np.random.default_rng(n)
    balls = random_balls(rsb, n, n)
    for c in "xy":
        balls["pos"][c] = rng.uniform(-300, 300, n)
        balls["vel"][c] *= 0.1
    balls["pos"]["z"] = rng.uniform(290, 700, n)
    return balls


def test_full_lists_on_the_host(pkg, host, patch):  # noqa: F811
    rsb, (lib, _) = pkg.rsb, host
    b = rsb.Batch(lib, 64, team_size=0, meshes_path=patch)
    b.set_balls(over_the_patch(rsb, 64))
    seen = np.zeros(4, np.int64)
    assert lib.rsb_host_ball_ticks_differ(b._h, 240, seen.ctypes.data) == 0
    assert seen[3] and seen[1]


def predictions(pkg, lib, arena, balls, ticks):
    rsb = pkg.rsb
    x, y = (rsb.Batch(w, len(balls), team_size=0, meshes_path=arena) for w in (lib, pkg.engine_library()))
    y.set_balls(balls)
    x.set_balls(y.get_balls())  # a prediction starts from the public state
    got = y.predict_ball(ticks)
    for k, t in enumerate(ticks):
        x.step(t - (ticks[k - 1] if k else 0))
        assert got[:, k].tobytes() == x.get_balls().tobytes(), f"after {t} ticks"


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 300, 1185])
def test_full_lists(pkg, host, patch, n):  # noqa: F811
    predictions(pkg, host[0], patch, over_the_patch(pkg.rsb, n), (1, 40, 240))


@pytest.mark.gpu
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_full_warps(pkg, host, more):  # noqa: F811
    torch = pytest.importorskip("torch")
    n = 32 * FULL_WARPS * torch.cuda.get_device_properties(0).multi_processor_count + more
    balls = random_balls(pkg.rsb, n, 5)
    balls["pos"]["z"][::2] = 100
    predictions(pkg, host[0], host[1], balls, (1, 60))
