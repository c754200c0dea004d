"""The step's phases (csrc/phys/step_phases.h, what the kernels run) against the one-thread tick
(stepArena), both compiled for the host: every persistent record byte for byte, tick after tick,
over starts that reach each queue (rays and boxes against meshes, cars on cars, cars on the ball,
demolitions and respawns, balls in goals, a non-finite car, empty arenas)."""
from __future__ import annotations

import ctypes as C
import importlib.util
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, ROOT
from gpu_util import random_balls, random_cars, random_controls
from host_util import ARENA_BUILD

SRC = os.path.join(ROOT, "tests", "cpp", "step_phases_host.cpp")
QUEUES = ("mesh rays", "body rays", "car-mesh", "ball-mesh", "car-ball", "car-car", "planes", "blocks", "islands",
          "bodies", "triangles", "deep", "combine")


@pytest.fixture(scope="module")
def host(pkg, tmp_path_factory):
    """The host library with both forms of the step, and a generated arena."""
    out = str(tmp_path_factory.mktemp("phases") / "librsbphases.so")
    cmd = [shutil.which("g++") or "g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-pthread", "-ffp-contract=off",
           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG_DIR, "csrc"), "-I", os.path.join(ROOT, "tests", "cpp"),
           SRC, ARENA_BUILD, "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    spec = importlib.util.spec_from_file_location("perf_cases_arena", os.path.join(ROOT, "perf", "cases.py"))
    cases = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(cases)
    lib = pkg.rsb.load_library(out)
    lib.rsb_host_records_differ.restype = C.c_int64
    lib.rsb_host_records_differ.argtypes = [C.c_void_p, C.c_void_p]
    lib.rsb_host_ball_ticks_differ.restype = C.c_int64
    lib.rsb_host_ball_ticks_differ.argtypes = [C.c_void_p, C.c_int32, C.c_void_p]
    lib.rsb_host_step_phases.argtypes = [C.c_void_p, C.c_int32, C.c_void_p, C.c_int32, C.c_int32, C.c_void_p, C.c_void_p]
    return lib, cases._arena()


def start(rsb, b, kind, seed):
    """Cars and balls of one kind of start."""
    rng = np.random.default_rng(seed)
    n, m = b.num_arenas, b.num_cars
    balls = random_balls(rsb, n, seed)
    cars = random_cars(rsb, b.get_cars(), seed + 1)
    arena = np.repeat(np.arange(n), np.diff(b.car_offset))
    if kind == "walls":      # near the ramps, the corners and the goals
        for a, k in ((balls, n), (cars, m)):
            a["pos"]["x"] = rng.choice([-1, 1], k) * rng.uniform(800, 3900, k)
            a["pos"]["y"] = rng.choice([-1, 1], k) * rng.uniform(3600, 5300, k)
            a["pos"]["x"][np.abs(a["pos"]["y"]) > 4900] *= 0.2
            a["pos"]["z"] = rng.uniform(40, 700, k)
    elif kind == "heap":     # every car of an arena beside its ball, fast
        for c in "xy":
            cars["pos"][c] = balls["pos"][c][arena] + rng.uniform(-220, 220, m)
        balls["pos"]["z"] = rng.uniform(95, 200, n)
        cars["pos"]["z"] = rng.uniform(17, 260, m)
        for c in "xyz":
            cars["vel"][c] = rng.uniform(-2300, 2300, m)
        cars["is_supersonic"] = 1
    elif kind == "stack":    # cars on the roofs of others, driving
        order = np.concatenate([np.arange(k) for k in np.diff(b.car_offset)])
        cars["pos"]["x"] = balls["pos"]["x"][arena] + rng.uniform(-30, 30, m)
        cars["pos"]["y"] = 0.8 * balls["pos"]["y"][arena] + rng.uniform(-30, 30, m)
        cars["pos"]["z"] = 17 + 55.0 * order
        cars["vel"]["x"] *= 0.05
        cars["vel"]["y"] *= 0.05
        balls["pos"]["z"] = 1500
    if kind in ("walls", "heap"):
        for c in "xyz":
            cars["ang_vel"][c] = rng.uniform(-5, 5, m)
    cars["is_demoed"][rng.random(m) < 0.15] = 1
    cars["demo_respawn_timer"] = rng.uniform(0, 0.4, m).astype(np.float32)
    return cars, balls


def compare(pkg, host, n, teams, kind, seed, ticks, steps, cull=False, mutate=None, cand_cap=-1, by_bodies=1):
    rsb, (lib, arena) = pkg.rsb, host
    x, y = (rsb.Batch(lib, n, team_sizes=teams, meshes_path=arena, seed=seed) for _ in range(2))
    cars, balls = start(rsb, x, kind, seed)
    if mutate:
        mutate(cars, balls)
    rng = np.random.default_rng(seed + 5)
    counts, stats = np.zeros(len(QUEUES), np.int64), np.zeros(4, np.uint64)
    for b in (x, y):
        b.set_balls(balls)
        if b.num_cars:
            b.set_cars(cars)
    mask = np.zeros(n, np.uint32)
    for k in range(steps):
        ctl = random_controls(rsb, max(1, x.num_cars), rng)[:x.num_cars]
        for b in (x, y):
            if b.num_cars:
                b.set_controls(ctl)
        x.step(ticks)
        st = lib.rsb_host_step_phases(y._h, ticks, mask.ctypes.data if cull else None, cand_cap, by_bodies,
                                      counts.ctypes.data, stats.ctypes.data)
        assert st == 0
        d = lib.rsb_host_records_differ(x._h, y._h)
        assert d == -1, f"step {k}: plane {('ball', 'car', 'pad', 'arena')[d >> 40]}, word {(d & ((1 << 40) - 1)) // n}"
    return dict(zip(QUEUES, counts.tolist()), rows=int(stats[3]))


@pytest.mark.parametrize("kind,ticks", [("field", 8), ("walls", 8), ("heap", 3), ("heap", 8), ("stack", 1), ("stack", 8)])
def test_phases_match_the_one_thread_tick(pkg, host, kind, ticks):
    teams = np.array([3, 1, 2, 3, 0] * 21 + [3], np.int32)  # 106 arenas: blocks of 32 and a remainder
    seen = {q: 0 for q in QUEUES}
    for seed in (11, 12):
        got = compare(pkg, host, len(teams), teams, kind, seed, ticks, 160 // ticks)
        seen = {q: seen[q] + got[q] for q in QUEUES}
    assert seen["mesh rays"] and seen["body rays"] and seen["planes"] and seen["islands"] and seen["bodies"]
    if kind == "walls":
        assert seen["car-mesh"] and seen["ball-mesh"] and seen["triangles"] and seen["deep"] and seen["combine"]
    if kind in ("heap", "stack"):
        assert seen["car-car"]
    if kind == "heap":
        assert seen["car-ball"]


@pytest.mark.parametrize("n", [1, 31, 32, 33])
def test_batch_sizes_around_a_block(pkg, host, n):
    compare(pkg, host, n, np.array([3, 2, 1] * 11, np.int32)[:n], "heap", 31, 8, 12)


@pytest.mark.parametrize("cand_cap", [0, 3, 40])
def test_more_triangles_than_there_is_room_for(pkg, host, cand_cap):
    """Pairs that find the candidate list full are taken on one thread, with the same results."""
    for kind in ("walls", "heap"):
        got = compare(pkg, host, 64, np.full(64, 3, np.int32), kind, 71, 8, 12, cand_cap=cand_cap)
        assert got["triangles"] > cand_cap


def test_islands_of_one_body_against_the_whole_solver(pkg, host):
    """Solver rows counted and records equal whether bodies that touch static objects only are
    solved by themselves or with their arena."""
    for kind in ("walls", "field"):
        got = [compare(pkg, host, 64, np.full(64, 3, np.int32), kind, 81, 8, 12, by_bodies=k) for k in (0, 1)]
        assert got[0]["bodies"] == 0 and got[1]["bodies"] > 0
        assert got[0]["rows"] == got[1]["rows"] > 0


def test_empty_arenas(pkg, host):
    compare(pkg, host, 33, np.zeros(33, np.int32), "field", 41, 8, 20)


def test_no_culled_body_is_the_exact_step(pkg, host):
    compare(pkg, host, 33, np.full(33, 2, np.int32), "walls", 51, 8, 12, cull=True)


@pytest.mark.parametrize("value", [np.nan, np.inf, 3e7])
def test_states_that_are_not_finite(pkg, host, value):
    """A car or a ball that is not finite (or moves so far that its box is refused) leaves the same
    records in both forms, its arena's other bodies included."""
    def mutate(cars, balls):
        cars["vel"]["x"][0] = value
        cars["pos"]["y"][9] = value
        balls["vel"]["z"][2] = value

    compare(pkg, host, 7, np.full(7, 2, np.int32), "heap", 61, 2, 3, mutate=mutate)


@pytest.mark.parametrize("kind", ["field", "walls", "still", "notfinite"])
def test_ball_alone_matches_the_ball_only_arena(pkg, host, kind):
    """The ball prediction's own tick against the ball-only arena, every tick of 360, byte by byte:
    flight, floor and ceiling, ramps, corners, goals, resting balls and balls that are not finite."""
    rsb, (lib, arena) = pkg.rsb, host
    b = rsb.Batch(lib, 256, team_size=1, meshes_path=arena)
    _, balls = start(rsb, b, "walls" if kind == "walls" else "field", 91)
    if kind == "still":
        for f in ("vel", "ang_vel"):
            for c in "xyz":
                balls[f][c][::2] = 0
        balls["pos"]["z"] = 93.15
    if kind == "notfinite":
        for i, v in enumerate((np.nan, np.inf, 3e7, 1e30)):
            balls["vel"]["xyz"[i % 3]][i] = v
            balls["pos"]["xyz"[i % 3]][8 + i] = v
    b.set_balls(balls)
    seen = np.zeros(4, np.int64)
    assert lib.rsb_host_ball_ticks_differ(b._h, 360, seen.ctypes.data) == 0
    assert seen[0] and seen[1]
    if kind == "walls":
        assert seen[2]
