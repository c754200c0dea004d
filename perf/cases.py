"""Performance cases of the batched soccar simulator.

Each case is work that a training program has the library do through its public entry
points: whole env steps (actions in, physics ticks, observations, masks, rewards, terminals,
resets of the finished arenas), and the stages that such a program also calls by themselves:
observations, ball prediction, VantaObs rows and GAE over a rollout buffer.

The arena is generated here, so that the cases need no files: a soccar field of the usual
dimensions (side planes, ceiling and floor are the library's own planes), with quarter-pipe
ramps along every wall, cut corners, back walls with goal mouths, and the two goals, about
8,700 triangles in 14 meshes, written once per process in the .cmf layout that the library
loads.
"""
from __future__ import annotations

import atexit
import importlib.util
import math
import os
import shutil
import struct
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_DIR = os.path.join(os.getcwd(), "emy-s-framework_b200")
if not os.path.isdir(PKG_DIR):
    PKG_DIR = os.path.join(ROOT, "emy-s-framework_b200")

EPISODE_TICKS = 1800   # episode length of the repository's benchmark
ACTION_SETS = 8        # different action arrays that the passes cycle through


def _pkg():
    """The package (its folder's name is not an identifier, so it is loaded by path)."""
    name = "emy_s_framework_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(PKG_DIR, "__init__.py"),
                                                      submodule_search_locations=[PKG_DIR])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ------------------------------------------------------------------ the arena

HALF_X, HALF_Y, HEIGHT, RAMP = 4096.0, 5120.0, 2048.0, 256.0
DIAG = 8064.0                                     # |x| + |y| of the corner walls
GOAL_X, GOAL_Z, GOAL_BACK = 892.755, 642.775, 6000.0
UU_PER_UNIT = 50.0                                # mesh files hold Bullet units
ARC = 12                                          # segments of a quarter pipe


def _profile():
    """(distance from the wall, height) from the floor up to the ceiling."""
    rows = []
    for k in range(ARC + 1):
        t = 0.5 * math.pi * k / ARC
        rows.append((RAMP * (1 - math.sin(t)), RAMP * (1 - math.cos(t))))
    rows += [(0.0, GOAL_Z), (0.0, 1026.0), (0.0, 1409.0)]
    for k in range(ARC + 1):
        t = 0.5 * math.pi * k / ARC
        rows.append((RAMP * (1 - math.cos(t)), HEIGHT - RAMP + RAMP * math.sin(t)))
    return rows


class _Mesh:
    def __init__(self):
        self.verts, self.tris, self.index = [], [], {}

    def vertex(self, p):
        key = tuple(round(c, 3) for c in p)
        if key not in self.index:
            self.index[key] = len(self.verts)
            self.verts.append(p)
        return self.index[key]

    def triangle(self, a, b, c, inside):
        """One triangle, wound so that its normal points to `inside`."""
        a, b, c = (np.asarray(v, float) for v in (a, b, c))
        n = np.cross(b - a, c - a)
        if np.dot(n, n) < 1e-6:
            return
        if np.dot(n, np.asarray(inside, float) - a) < 0:
            b, c = c, b
        self.tris.append([self.vertex(tuple(v)) for v in (a, b, c)])

    def quad(self, a, b, c, d, inside):
        self.triangle(a, b, c, inside)
        self.triangle(a, c, d, inside)

    def write(self, path):
        v = np.asarray(self.verts, np.float32) / np.float32(UU_PER_UNIT)
        t = np.asarray(self.tris, np.int32)
        with open(path, "wb") as f:
            f.write(struct.pack("<ii", len(t), len(v)))
            f.write(t.tobytes())
            f.write(v.astype(np.float32).tobytes())


def _sweep(mesh, columns, rows, skip, inside):
    """Quads between neighbouring columns (functions of the profile point) and rows."""
    for c in range(len(columns) - 1):
        for r in range(len(rows) - 1):
            if skip(c, r):
                continue
            (d0, z0), (d1, z1) = rows[r], rows[r + 1]
            q = [columns[c](d0) + (z0,), columns[c + 1](d0) + (z0,), columns[c + 1](d1) + (z1,), columns[c](d1) + (z1,)]
            mesh.quad(*q, inside)


def _arena_meshes():
    rows = _profile()
    wall = range(ARC, len(rows) - 1 - ARC)  # the rows of the upright part of a wall
    k = math.sqrt(2.0) - 1.0
    inside = (0.0, 0.0, HEIGHT / 2)
    meshes = []
    # side walls: the upright part is the library's own plane, the meshes hold the ramps
    for sx in (-1, 1):
        for sy in (-1, 1):
            m = _Mesh()
            cols = [(lambda d, t=i / 20: (sx * (HALF_X - d), sy * t * (DIAG - HALF_X - k * d))) for i in range(21)]
            _sweep(m, cols, rows, lambda c, r: r in wall, inside)
            meshes.append(m)
    # corner walls
    for sx in (-1, 1):
        for sy in (-1, 1):
            m = _Mesh()

            def corner(d, t):
                x0, y0 = HALF_X - d, DIAG - HALF_X - k * d
                x1, y1 = DIAG - HALF_Y - k * d, HALF_Y - d
                return sx * (x0 + t * (x1 - x0)), sy * (y0 + t * (y1 - y0))

            cols = [(lambda d, t=i / 10: corner(d, t)) for i in range(11)]
            _sweep(m, cols, rows, lambda c, r: False, inside)
            meshes.append(m)
    # back walls, half by half, open at the goal mouth
    for sy in (-1, 1):
        for sx in (-1, 1):
            m = _Mesh()
            cols = [(lambda d, x=GOAL_X * i / 4: (sx * x, sy * (HALF_Y - d))) for i in range(5)]
            cols += [(lambda d, t=i / 8: (sx * (GOAL_X + t * (DIAG - HALF_Y - k * d - GOAL_X)), sy * (HALF_Y - d)))
                     for i in range(1, 9)]
            _sweep(m, cols, rows, lambda c, r: c < 4 and rows[r + 1][1] <= GOAL_Z, inside)
            meshes.append(m)
    # goals: side walls, roof, back, and the caps that close the ramps beside the mouth
    for sy in (-1, 1):
        m = _Mesh()
        centre = (0.0, sy * (HALF_Y + 440.0), GOAL_Z / 2)
        ys = [HALF_Y + (GOAL_BACK - HALF_Y) * i / 4 for i in range(5)]
        zs = [GOAL_Z * i / 3 for i in range(4)]
        xs = [GOAL_X * i / 4 for i in range(-4, 5)]
        for sx in (-1, 1):
            for i in range(4):
                for j in range(3):
                    m.quad((sx * GOAL_X, sy * ys[i], zs[j]), (sx * GOAL_X, sy * ys[i + 1], zs[j]),
                           (sx * GOAL_X, sy * ys[i + 1], zs[j + 1]), (sx * GOAL_X, sy * ys[i], zs[j + 1]), centre)
            for i in range(ARC):
                (d0, z0), (d1, z1) = rows[i], rows[i + 1]
                m.triangle((sx * GOAL_X, sy * HALF_Y, 0.0), (sx * GOAL_X, sy * (HALF_Y - d0), z0),
                           (sx * GOAL_X, sy * (HALF_Y - d1), z1), centre)
        for i in range(8):
            for j in range(4):
                m.quad((xs[i], sy * ys[j], GOAL_Z), (xs[i + 1], sy * ys[j], GOAL_Z), (xs[i + 1], sy * ys[j + 1], GOAL_Z),
                       (xs[i], sy * ys[j + 1], GOAL_Z), centre)
            for j in range(3):
                m.quad((xs[i], sy * GOAL_BACK, zs[j]), (xs[i + 1], sy * GOAL_BACK, zs[j]),
                       (xs[i + 1], sy * GOAL_BACK, zs[j + 1]), (xs[i], sy * GOAL_BACK, zs[j + 1]), centre)
        meshes.append(m)
    return meshes


_arena_dir = None


def _arena():
    """Folder with soccar/mesh_<i>.cmf, written once per process."""
    global _arena_dir
    if _arena_dir is None:
        _arena_dir = tempfile.mkdtemp(prefix="soccar_arena_")
        atexit.register(shutil.rmtree, _arena_dir, True)
        os.mkdir(os.path.join(_arena_dir, "soccar"))
        for i, m in enumerate(_arena_meshes()):
            m.write(os.path.join(_arena_dir, "soccar", "mesh_%d.cmf" % i))
    return _arena_dir


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one collector thread's handful of arenas stepped from the host, every result read back
        # (the tests' and the smoke run's size): launches and latency
        {"name": "env_1v1_16_host", "kind": "env", "teams": 1, "arenas": 16, "ticks": 8, "start": "kickoff",
         "call": "host", "cull": "exact", "settle": 20},
        # a small training run, 250 arenas of 2v2, the policy on the device
        {"name": "env_2v2_250", "kind": "env", "teams": 2, "arenas": 250, "ticks": 8, "start": "random",
         "call": "device", "cull": "exact", "settle": 30},
        # a mid-size run that replays its env step as a CUDA graph, odd arena count, shorter steps
        {"name": "env_3v3_1023_graph", "kind": "env", "teams": 3, "arenas": 1023, "ticks": 4, "start": "random",
         "call": "graph", "cull": "exact", "settle": 40},
        # the benchmark's second configuration: 2v2 x 8,192
        {"name": "env_2v2_8192", "kind": "env", "teams": 2, "arenas": 8192, "ticks": 8, "start": "random",
         "call": "device", "cull": "exact", "settle": 30},
        # its mixed batch of 1v1, 2v2 and 3v3 arenas, stepped as a CUDA graph
        {"name": "env_mixed_32768_graph", "kind": "env", "teams": 0, "arenas": 32768, "ticks": 8, "start": "random",
         "call": "graph", "cull": "exact", "settle": 16},
        # its headline: 3v3 x 65,536
        {"name": "env_3v3_65536", "kind": "env", "teams": 3, "arenas": 65536, "ticks": 8, "start": "random",
         "call": "device", "cull": "exact", "settle": 12},
        # high-contact 1v1 starts with boost and jump pressed often, distance-bound culling, odd count
        {"name": "env_1v1_50001_contact", "kind": "env", "teams": 1, "arenas": 50001, "ticks": 8, "start": "contact",
         "call": "device", "cull": "voxel", "settle": 12},
        # the observations of the headline batch by themselves (rebuilt after states were set)
        {"name": "obs_3v3_65536", "kind": "obs", "teams": 3, "arenas": 65536},
        # ball prediction for every arena, kept on the device: 1, 2 and 3 s ahead
        {"name": "predict_16384", "kind": "predict", "teams": 1, "arenas": 16384, "horizon": 360},
        # VantaObs rows, with the ball prediction that they read
        {"name": "vanta_2v2_4096", "kind": "vanta", "teams": 2, "arenas": 4096},
        # GAE over the rollout buffer of the headline batch: 393,216 players x 32 steps
        {"name": "gae_393216x32", "kind": "gae", "players": 393216, "steps": 32, "ragged": False, "scaled": False},
        # a small collector's buffer: episodes of uneven length, truncations, reward scaling and clipping
        {"name": "gae_ragged_257x400", "kind": "gae", "players": 257, "steps": 400, "ragged": True, "scaled": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("env", "env", "env", "env", "obs", "predict", "vanta", "gae"))
    teams = rng.choice((1, 2, 3, 0))
    if kind == "env":
        call = rng.choice(("host", "device", "device", "graph"))
        arenas = _log_int(rng, 8, 65536 if call != "host" else 16384)
        return {"kind": "env", "teams": teams, "arenas": arenas, "ticks": rng.choice((1, 4, 8, 8, 8)),
                "start": rng.choice(("kickoff", "random", "random", "contact")), "call": call,
                "cull": rng.choice(("exact", "exact", "voxel")), "settle": 30 if arenas <= 8192 else 12}
    if kind == "obs":
        return {"kind": "obs", "teams": teams, "arenas": _log_int(rng, 8, 65536)}
    if kind == "predict":
        return {"kind": "predict", "teams": 1, "arenas": _log_int(rng, 8, 32768), "horizon": rng.choice((120, 240, 360))}
    if kind == "vanta":
        return {"kind": "vanta", "teams": teams, "arenas": _log_int(rng, 8, 16384)}
    steps = _log_int(rng, 8, 1024)
    return {"kind": "gae", "players": _log_int(rng, 16, max(32, min(393216, 12_000_000 // steps))), "steps": steps,
            "ragged": rng.random() < 0.5, "scaled": rng.random() < 0.5}


def _team_sizes(case):
    """Team size of every arena (0: 1v1, 2v2 and 3v3 in turn)."""
    if case["teams"]:
        return np.full(case["arenas"], case["teams"], np.int32)
    return np.array([1 + a % 3 for a in range(case["arenas"])], np.int32)


class _DeviceArray:
    """A device buffer of a batch, for torch.as_tensor: the tensor keeps this object, and with it
    the batch that owns the buffer."""

    def __init__(self, batch, ptr, shape, typestr):
        self.batch = batch
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _view(batch, which, shape, typestr="<f4"):
    return torch.as_tensor(_DeviceArray(batch, batch.device_ptr(which), shape, typestr), device="cuda")


def _action_weights(lut, start):
    """Uniform over the table, or (contact starts) boost and jump each pressed with 0.6."""
    w = np.ones(len(lut))
    if start == "contact":
        for b in (0, 1):
            for j in (0, 1):
                sel = ((lut["boost"] != 0) == bool(b)) & ((lut["jump"] != 0) == bool(j))
                w[sel] = (0.6 if b else 0.4) * (0.6 if j else 0.4) / max(1, sel.sum())
    return w / w.sum()


def _batch(case, seed, start, cull="exact"):
    rsb = _pkg().rsb
    lib = _pkg().engine_library()
    mode = {"exact": rsb.RSB_CULL_EXACT, "voxel": rsb.RSB_CULL_VOXEL}[cull]
    batch = rsb.Batch(lib, case["arenas"], team_size=None, team_sizes=_team_sizes(case), meshes_path=_arena(),
                      tick_skip=case.get("ticks", 8), rewards=rsb.default_rewards(lib, episode_max_ticks=EPISODE_TICKS),
                      cull_mode=mode, seed=seed)
    lut = rsb.default_action_lut(lib)
    batch.set_action_lut(lut)
    reset = {"kickoff": rsb.RSB_RESET_KICKOFF, "random": rsb.RSB_RESET_RANDOM_STATE,
             "contact": rsb.RSB_RESET_HIGH_CONTACT}[start]
    rng = np.random.default_rng(seed)
    acts = rng.choice(len(lut), size=(ACTION_SETS, batch.num_cars), p=_action_weights(lut, start)).astype(np.int32)
    batch.reset_all(seed, reset)
    return batch, acts, reset


def _device_step(s, k):
    """One env step on the device, as a collector with its policy on the GPU runs it."""
    b, st = s["batch"], s["stream"].cuda_stream
    b.snapshot(stream=st)
    b.set_actions_device(s["actions"][k % ACTION_SETS].data_ptr(), b.num_cars, stream=st)
    b.step(s["ticks"], stream=st)
    b.build_obs(stream=st)
    b.build_rewards_terminals(s["ticks"], stream=st)
    b.reset_done(s["seed"] + k, s["reset"], stream=st)


def prepare(case, seed):
    if case["kind"] == "gae":
        return _prepare_gae(case, seed)
    rsb = _pkg().rsb
    start = case.get("start", "random")
    batch, acts, reset = _batch(case, seed, start, case.get("cull", "exact"))
    s = {"kind": case["kind"], "call": case.get("call"), "batch": batch, "reset": reset, "seed": seed + 1, "pass": 0,
         "ticks": case.get("ticks", 8), "stream": torch.cuda.Stream(), "actions": torch.from_numpy(acts).cuda()}
    torch.cuda.synchronize()
    # play on from the start, so that the cars have landed and spread as they do in a long run
    for k in range(case.get("settle", 8)):
        _device_step(s, k)
    s["pass"] = case.get("settle", 8)
    torch.cuda.synchronize()
    n, m = batch.num_arenas, batch.num_cars
    if case["kind"] in ("env", "obs"):
        s["out"] = {"obs": _view(batch, rsb.RSB_BUF_OBS, (m, batch.obs_stride)),
                    "masks": _view(batch, rsb.RSB_BUF_MASKS, (m, rsb.RSB_NUM_ACTIONS), "|u1"),
                    "rewards": _view(batch, rsb.RSB_BUF_REWARDS, (m,)),
                    "terminals": _view(batch, rsb.RSB_BUF_TERMINALS, (n,), "|u1")}
    if case.get("call") == "graph":
        s["current"] = s["actions"][0].clone()  # the policy writes its actions into one fixed buffer
        torch.cuda.synchronize()
        batch.env_graph_capture(s["current"].data_ptr(), s["ticks"], reset, seed + 2)
    elif case.get("call") == "host":
        s["host_actions"], s["out"] = acts, batch.pinned_outputs()
    if case["kind"] == "predict":
        h = case["horizon"]
        s["slices"] = (h // 3, 2 * h // 3, h)
        batch.predict_ball(s["slices"][:1], to_host=False, stream=s["stream"].cuda_stream)  # sizes the buffer
        s["out"] = _view(batch, rsb.RSB_BUF_BALL_PRED, (n, 3, 18))
    if case["kind"] == "vanta":
        batch.vanta_configure()
        s["out"] = _view(batch, rsb.RSB_BUF_VANTA_OBS, (m, rsb.RSB_VANTA_OBS_SIZE))
    return s


def run(s):
    if s["kind"] == "gae":
        return _run_gae(s)
    b, st, k = s["batch"], s["stream"].cuda_stream, s["pass"]
    s["pass"] = k + 1
    if s["kind"] == "obs":
        b.build_obs(stream=st)
        return {"obs": s["out"]["obs"], "masks": s["out"]["masks"]}
    if s["kind"] == "predict":
        b.predict_ball(s["slices"], to_host=False, stream=st)
        return s["out"]
    if s["kind"] == "vanta":
        b.build_vanta_obs(stream=st)
        return s["out"]
    if s["call"] == "graph":
        with torch.cuda.stream(s["stream"]):
            s["current"].copy_(s["actions"][k % ACTION_SETS])
        b.env_graph_launch(stream=st)
    elif s["call"] == "host":
        b.snapshot()
        b.set_actions(s["host_actions"][k % ACTION_SETS])
        b.step(s["ticks"])
        b.build_obs()
        b.build_rewards_terminals(s["ticks"])
        b.copy_outputs(s["out"])
        b.reset_done(s["seed"] + k, s["reset"])
    else:
        _device_step(s, k)
    return s["out"]


# ------------------------------------------------------------------ GAE

GAMMA, LAM, RETURN_STD, CLIP = 0.99, 0.95, 2.5, 1.0


def _gae_inputs(case, seed):
    """A rollout buffer, player after player: rewards of a shaped task, a critic's values, and
    terminals (1 done, 2 cut off); every player's last step ends its trajectory."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)
    P, L = case["players"], case["steps"]
    rews = torch.randn(P * L, generator=g, device="cuda") * 0.3
    rews += (torch.rand(P * L, generator=g, device="cuda") < 0.01) * 5.0
    vals = torch.randn(P * L + 1, generator=g, device="cuda") * 2.0
    term = torch.zeros(P, L, dtype=torch.int8, device="cuda")
    if case["ragged"]:
        u = torch.rand(P, L, generator=g, device="cuda")
        term[u < 0.01] = 1
        term[u > 0.996] = 2
    term[:, -1] = 2
    term = term.reshape(-1).contiguous()
    truncs = torch.randn(int((term == 2).sum()), generator=g, device="cuda") * 2.0
    return rews, term, vals, truncs


def _prepare_gae(case, seed):
    rsb, lib = _pkg().rsb, _pkg().engine_library()
    rews, term, vals, truncs = _gae_inputs(case, seed)
    T = rews.numel()
    params = rsb.gae_params(lib, gamma=GAMMA, lam=LAM, return_std=RETURN_STD if case["scaled"] else 0.0,
                            clip_range=CLIP if case["scaled"] else 0.0)
    out = {k: torch.zeros(T, device="cuda") for k in ("advantages", "targets", "returns")}
    out["clip_portion"] = torch.zeros(1, device="cuda")
    return {"kind": "gae", "in": (rews, term, vals, truncs), "out": out, "params": params, "stream": torch.cuda.Stream()}


def _run_gae(s):
    rews, term, vals, truncs = s["in"]
    o = s["out"]
    _pkg().rsb.compute_gae_device(_pkg().engine_library(), rews.data_ptr(), term.data_ptr(), vals.data_ptr(),
                                  truncs.data_ptr(), truncs.numel(), o["advantages"].data_ptr(),
                                  o["targets"].data_ptr(), o["returns"].data_ptr(), o["clip_portion"].data_ptr(),
                                  rews.numel(), s["params"], s["stream"].cuda_stream)
    return o


def exact(case, seed):
    """GAE in 64 bits.  The other cases start from a state that the physics has played on to, which
    only the library can make from the seed, so they have no value of their own."""
    if case["kind"] != "gae":
        return None
    rews, term, vals, truncs = _gae_inputs(case, seed)
    P, L = case["players"], case["steps"]
    f32 = lambda v: float(np.float32(v))  # noqa: E731  (the parameters are passed as 32-bit values)
    gamma, lam = f32(GAMMA), f32(LAM)
    r, v, t = rews.double().reshape(P, L), vals.double(), term.reshape(P, L)
    scaled = r / f32(RETURN_STD) if case["scaled"] else r
    used = scaled.clamp(-CLIP, CLIP) if case["scaled"] else scaled
    # the bootstrap value of the n-th cut-off step is the n-th from the end of the list
    cut = (term == 2).reshape(-1)
    order = torch.cumsum(cut.long(), 0) - 1
    boot = torch.zeros(P * L, dtype=torch.float64, device=v.device)
    boot[cut] = truncs.double().flip(0)[order[cut]]
    nxt = torch.where(cut, boot, torch.where((term == 1).reshape(-1), torch.zeros_like(boot), v[1:])).reshape(P, L)
    run_on = (t == 0).double()
    delta = used + gamma * nxt - v[:-1].reshape(P, L)
    adv, ret = torch.zeros_like(r), torch.zeros_like(r)
    a = torch.zeros(P, dtype=torch.float64, device=v.device)
    g = torch.zeros_like(a)
    for k in range(L - 1, -1, -1):
        a = delta[:, k] + gamma * lam * run_on[:, k] * a
        g = r[:, k] + gamma * run_on[:, k] * g
        adv[:, k], ret[:, k] = a, g
    total, kept = scaled.abs().sum(), used.abs().sum()
    return {"advantages": adv.reshape(-1), "targets": (v[:-1].reshape(P, L) + adv).reshape(-1),
            "returns": ret.reshape(-1), "clip_portion": ((total - kept) / max(float(total), 1e-7)).reshape(1)}


# ------------------------------------------------------------------ what a pass cannot do without

BALL, CAR, PAD, ARENA = 92, 344, 34 * 8, 32   # bytes of the persistent records
CTL, MASK = 24, 90
# arithmetic of one tick, counted from the model's equations: a car's four wheel rays against the
# planes, its suspension, friction, drive and air terms, and its integration; the ball's contact
# with the nearest surface and its integration
CAR_TICK, BALL_TICK = 2500, 600


def work(case):
    if case["kind"] == "gae":
        n = case["players"] * case["steps"]
        return {"bytes": n * (4 + 1 + 4 + 12) + 4 * case["players"], "flops": 12 * n}
    n = case["arenas"]
    cars = int(2 * _team_sizes(case).sum())
    row = 51 + 29 * 2 * int(_team_sizes(case).max())
    obs = cars * (4 * row + MASK)
    if case["kind"] == "obs":
        # read: the kinematics, flags and action of every car, the ball, the pads
        return {"bytes": obs + cars * (22 * 4 + CTL) + n * (10 * 4 + PAD), "flops": 40 * obs // 4}
    if case["kind"] == "predict":
        return {"bytes": n * (BALL + 3 * 72), "flops": n * case["horizon"] * BALL_TICK}
    if case["kind"] == "vanta":
        return {"bytes": n * (BALL + PAD + ARENA) + cars * (CAR + 366 * 4), "flops": n * 360 * BALL_TICK}
    t = case["ticks"]
    state = n * (BALL + PAD + ARENA) + cars * CAR
    return {"bytes": 2 * state + cars * (CTL + 4 + 4) + obs + n, "flops": t * (cars * CAR_TICK + n * BALL_TICK)}
