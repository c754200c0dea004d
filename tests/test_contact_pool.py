"""Arenas with more manifolds than a tick keeps (16): cars and ball crammed where ramps, corner, wall
and floor meet, 20 to 38 pairs with contacts each.  Which of them an arena keeps is decided by its own
dispatch order, whatever shares its storage and however its contacts come in: the phases (queues taken
from the back) against the one-thread tick, byte for byte."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, ROOT
from gpu_util import random_balls, random_cars
from host_util import ARENA_BUILD
from test_step_phases import QUEUES, host  # noqa: F401  (host: the fixture)

WS_OVERFLOW = 2
# centre, half width and height of the region: beside a corner wall, a back wall's ramp, a goal post
PLACES = {"corner": (3980, 3900, 40, 70), "ramp": (2900, 5000, 60, 130), "post": (850, 5100, 60, 130)}


def crammed(rsb, b, place, seed, spread=()):
    """Every car and the ball of an arena in one of the four mirrored places; `spread`: arenas whose
    cars stand apart."""
    x0, y0, w, z1 = PLACES[place]
    rng = np.random.default_rng(seed)
    n, m = b.num_arenas, b.num_cars
    arena = np.repeat(np.arange(n), np.diff(b.car_offset))
    balls, cars = random_balls(rsb, n, seed), random_cars(rsb, b.get_cars(), seed + 1)
    sx, sy = rng.choice([-1, 1], n), rng.choice([-1, 1], n)
    for rows, k, a in ((balls, n, np.arange(n)), (cars, m, arena)):
        apart = np.isin(a, spread)
        at = {"x": sx[a] * (x0 + rng.uniform(-w, w, k)), "y": sy[a] * (y0 + rng.uniform(-w, w, k)),
              "z": rng.uniform(20, z1, k)}
        for c in "xyz":
            rows["pos"][c] = np.where(apart, rows["pos"][c], at[c])
            rows["vel"][c] *= 0.1
    return cars, balls


@pytest.fixture(scope="module")
def pool(pkg, host, tmp_path_factory):  # noqa: F811
    """The phases with the engine's pool of contact points."""
    out = str(tmp_path_factory.mktemp("pool") / "librsbpool.so")
    r = subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-pthread",
                        "-ffp-contract=off", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG_DIR, "csrc"),
                        "-I", os.path.join(ROOT, "tests", "cpp"), os.path.join(ROOT, "tests", "cpp", "contact_pool_host.cpp"),
                        ARENA_BUILD, "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    lib = pkg.rsb.load_library(out)
    lib.rsb_host_records_differ.restype = C.c_int64
    lib.rsb_host_records_differ.argtypes = [C.c_void_p, C.c_void_p]
    lib.rsb_host_step_phases.argtypes = [C.c_void_p, C.c_int32, C.c_void_p, C.c_int32, C.c_int32, C.c_void_p, C.c_void_p]
    return lib, host[1]


@pytest.mark.parametrize("place", list(PLACES))
@pytest.mark.parametrize("n", [1, 2, 64, 65])
def test_kept_manifolds_are_the_arena_s_own(pkg, pool, n, place):
    rsb, (lib, arena) = pkg.rsb, pool
    spread = np.arange(1, n, 4)
    full = np.zeros(n, bool)
    for seed in range(max(1, 12 // n)):
        x, y = (rsb.Batch(lib, n, team_size=3, meshes_path=arena, seed=seed) for _ in range(2))
        cars, balls = crammed(rsb, x, place, 7 * seed + n, spread)
        for b in (x, y):
            b.set_balls(balls)
            b.set_cars(cars)
        counts, stats = np.zeros(len(QUEUES), np.int64), np.zeros(4, np.uint64)
        for tick in range(6):
            x.step(1)
            assert lib.rsb_host_step_phases(y._h, 1, None, -1, 1, counts.ctypes.data, stats.ctypes.data) == 0
            d = lib.rsb_host_records_differ(x._h, y._h)
            assert d == -1, f"tick {tick}: plane {d >> 40}, arena {(d & ((1 << 40) - 1)) % n}"
        full |= (x.get_arena_info()["status"] & WS_OVERFLOW) != 0
    assert full.sum() >= (n + 1) // 2 and not full[spread].any()
