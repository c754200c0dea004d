"""Device GAE on more streams than keep scratch of their own: no call waits on the host for work that
another stream still has to do, and the results stay each stream's own."""
import pytest

from gae_util import make_case
from test_gpu_gae_rows import check, launch, recurrence

pytestmark = pytest.mark.gpu


def test_no_call_waits_for_another_stream(pkg):
    torch = pytest.importorskip("torch")
    streams = [torch.cuda.Stream(priority=-(i % 2)) for i in range(40)]  # torch has 32 of each priority
    assert len({s.cuda_stream for s in streams}) == 40
    cs = [make_case(20000 + 997 * i, 1 / 90, 1.5, 1.0, i % 2 == 0, i) for i in range(40)]
    calls = [launch(pkg, torch, c, 0, s) for c, s in zip(cs, streams)]
    grown = make_case(400000, 1 / 90, 1.5, 1.0, True, 41)
    calls.append(launch(pkg, torch, grown, 0, torch.cuda.Stream()))
    for run, _ in calls[:40]:
        run()
    torch.cuda.synchronize()
    busy, done = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(2_000_000_000)  # about a second
        done.record()
    for run, _ in calls + calls[:5]:
        run()
    assert not done.query()
    torch.cuda.synchronize()
    for (_, read), c in zip(calls, cs + [grown]):
        check(read(), recurrence(c))
