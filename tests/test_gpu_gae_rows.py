"""Device GAE against the recurrence in 32-bit numpy, step by step: rows at the edges of the blocks'
chunks and of the windows that a segment goes on through, rows that allow no wide loads, buffers
with and without truncations, and calls side by side on several streams.

The recurrences round as the kernel does (32-bit products and sums, in the same order), so
advantages, returns and targets are equal bit for bit.  The clip portion is a quotient of sums of n
magnitudes, each summed in at most 16 + 5 + 8 + n / 2^20 + 13 steps: 64 roundings of 2^-24, twice,
bound its error by 8e-6 of the sum.
"""
import numpy as np
import pytest

from gae_util import make_case

pytestmark = pytest.mark.gpu
CLIP_TOL = 8e-6


def recurrence(c):
    f = np.float32
    T, gamma, gl = len(c["rews"]), f(c["gamma"]), f(c["gamma"]) * f(c["lam"])
    r = c["rews"] / f(c["std"]) if c["std"] > 0 else c["rews"]
    used = np.clip(r, -f(c["clip"]), f(c["clip"])) if c["std"] > 0 and c["clip"] > 0 else r
    term = c["term"]
    nxt = np.append(c["vals"], f(0))[1:T + 1].copy()
    nxt[term == 1] = 0
    nxt[term == 2] = c["trunc"][::-1][:int((term == 2).sum())]
    delta = (used + gamma * nxt) - c["vals"][:T]
    adv, ret = np.empty(T, f), np.empty(T, f)
    a = b = f(0)
    for t in range(T - 1, -1, -1):
        if term[t] != 0:
            a = b = f(0)
        b = c["rews"][t] + b * gamma
        a = delta[t] + gl * a
        adv[t], ret[t] = a, b
    tot = np.abs(r.astype(np.float64)).sum()
    clipped = np.abs(used.astype(np.float64)).sum() if c["std"] > 0 else 0.0
    return adv, c["vals"][:T] + adv, ret, (tot - clipped) / max(tot, 1e-7)


def launch(pkg, torch, c, skew, stream):
    """Inputs and outputs `skew` elements into their allocations."""
    def row(x, dtype):
        t = torch.zeros(len(x) + 8, dtype=dtype, device="cuda")
        t[skew:skew + len(x)] = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        return t

    T, lib = len(c["rews"]), pkg.engine_library()
    d = {"in": [row(c["rews"], torch.float32), row(c["term"], torch.int8), row(c["vals"], torch.float32),
                row(c["trunc"], torch.float32)],
         "out": [row(np.full(T, np.nan, np.float32), torch.float32) for _ in range(3)], "clip": torch.zeros(1, device="cuda")}
    torch.cuda.synchronize()
    at = lambda t: t.data_ptr() + skew * t.element_size()  # noqa: E731
    p = pkg.rsb.gae_params(lib, gamma=c["gamma"], lam=c["lam"], return_std=c["std"], clip_range=c["clip"])
    run = lambda: pkg.rsb.compute_gae_device(  # noqa: E731
        lib, at(d["in"][0]), at(d["in"][1]), at(d["in"][2]), at(d["in"][3]), len(c["trunc"]), *map(at, d["out"]),
        d["clip"].data_ptr(), T, p, stream.cuda_stream)
    read = lambda: [t[skew:skew + T].cpu().numpy() for t in d["out"]] + [float(d["clip"].item())]  # noqa: E731
    return run, read


def check(got, want):
    for g, w, what in zip(got[:3], want[:3], ("advantages", "targets", "returns")):
        assert (g.view(np.uint32) == w.view(np.uint32)).all(), what
    assert abs(got[3] - want[3]) <= CLIP_TOL


# T, probability of a terminal, whether the last step is one, elements into the allocation
@pytest.mark.parametrize("T,p,end,skew", [
    (1, 0.0, True, 0), (3, 0.3, False, 1), (4095, 0.01, False, 0), (4096, 0.0, True, 0), (4097, 0.5, True, 3),
    (4100, 0.001, False, 0), (9215, 0.0, False, 0), (12289, 0.0003, True, 2), (65537, 1 / 300, False, 0),
    (262144, 1 / 33, True, 0), (50001, 0.0, False, 1)])
@pytest.mark.parametrize("share,std,clip", [(0.4, 2.5, 1.0), (0.0, 0.0, 0.0)])
def test_rows(pkg, T, p, end, skew, share, std, clip):
    torch = pytest.importorskip("torch")
    c = make_case(T, p, std, clip, end, 7 * T + skew, trunc_share=share)
    if share == 0.0 and end:
        c["term"][T - 1], c["trunc"] = 1, c["trunc"][:0]
    run, read = launch(pkg, torch, c, skew, torch.cuda.Stream())
    run()
    torch.cuda.synchronize()
    check(read(), recurrence(c))


def test_streams_side_by_side(pkg):
    """Twenty streams, more than there are scratch slots, three calls each."""
    torch = pytest.importorskip("torch")
    cs = [make_case(30000 + 997 * i, 1 / 90, 1.5, 1.0, i % 2 == 0, i) for i in range(20)]
    calls = [launch(pkg, torch, c, 0, torch.cuda.Stream()) for c in cs]
    for _ in range(3):
        for run, _ in calls:
            run()
    torch.cuda.synchronize()
    for (_, read), c in zip(calls, cs):
        check(read(), recurrence(c))
