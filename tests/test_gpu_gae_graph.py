"""Device GAE under stream capture: each captured call works in scratch that its graph owns, so graphs
replayed side by side, calls on parallel branches of one graph, and larger calls between the replays
leave one another's results alone.  Bit for bit against the 32-bit recurrence, as in
test_gpu_gae_rows.py (the clip portion within its bound)."""
import pytest

from gae_util import make_case
from test_gpu_gae_rows import check, launch, recurrence

pytestmark = pytest.mark.gpu


def case(T, seed):
    return make_case(T, 1 / 90, 1.5, 1.0, seed % 2 == 0, seed, trunc_share=0.4)


def test_graphs_side_by_side(pkg):
    torch = pytest.importorskip("torch")
    cs = [case(300000 + 4099 * i, i) for i in range(4)]
    streams = [torch.cuda.Stream() for _ in cs]
    calls = [launch(pkg, torch, c, 0, s) for c, s in zip(cs, streams)]
    graphs = [torch.cuda.CUDAGraph() for _ in cs]
    for g, s, (run, _) in zip(graphs, streams, calls):
        with torch.cuda.graph(g, stream=s):
            run()
    larger = case(9 * 300000, 11)
    eager, read_eager = launch(pkg, torch, larger, 0, torch.cuda.Stream())
    want = [recurrence(c) for c in cs]
    for again in range(2):
        for _ in range(20):
            for g, s in zip(graphs, streams):
                with torch.cuda.stream(s):
                    g.replay()
        torch.cuda.synchronize()
        for (_, read), w in zip(calls, want):
            check(read(), w)
        eager()  # more chunks than any call before it
        torch.cuda.synchronize()
    check(read_eager(), recurrence(larger))


def test_parallel_branches_of_one_graph(pkg):
    torch = pytest.importorskip("torch")
    cs = [case(400000, 21), case(400000, 22)]
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    calls = [launch(pkg, torch, c, 0, s) for c, s in zip(cs, (s1, s2))]
    for _ in range(3):  # each graph replaces the one before, whose scratch it may take
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s1):
            s2.wait_stream(s1)
            calls[0][0]()
            calls[1][0]()
            s1.wait_stream(s2)
        for _ in range(10):
            g.replay()
        torch.cuda.synchronize()
        for (_, read), c in zip(calls, cs):
            check(read(), recurrence(c))
