"""The all-slices kernel as recorded: several groups to a call (kernel and counter clear replayed
per group), and two plans at the same time on two streams."""
import pytest
import torch

from namsa_gb300 import engine
from test_gpu_routes import BAND, KMAX
from test_gpu_stream import case, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('ny,nx,S,P', [(512, 512, 3, 150), (384, 384, 4, 301), (768, 768, 2, 70)])
def test_replays_of_many_groups(ny, nx, S, P):
    """Equal bits at every replay, and for other contents in the same buffers what those give."""
    torch.cuda.set_device(0)
    x, y = case(ny, nx, S, P, 1), case(ny, nx, S, P, 2)
    plan = engine.Plan(ny, nx)
    form, size, _, _ = plan.route(S, P, KMAX, BAND)
    assert form == 'all_slices' and P > 2 * size  # calls of up to two groups are issued directly
    plan.set_graph(False)
    want = [plan.multislice(*v, crop=64).clone() for v in (x, y)]
    plan.set_graph(True)
    out = torch.empty_like(want[0])
    for _ in range(3):
        assert torch.equal(plan.multislice(*x, crop=64, out=out), want[0])
    for a, b in zip(x[:4], y[:4]):
        a.copy_(b)
    assert torch.equal(plan.multislice(*x, crop=64, out=out), want[1])
    plan.check()
    plan.set_schedule(*plan.schedule[:2])
    assert rel(plan.multislice(*y, crop=64), want[1]) < 1e-6
    plan.close()


def test_two_plans_on_two_streams():
    torch.cuda.set_device(0)
    jobs = []
    for n, S, P, seed in ((512, 20, 24, 3), (384, 20, 90, 4)):
        plan = engine.Plan(n, n)
        x = case(n, n, S, P, seed)
        assert plan.route(S, P, KMAX, BAND)[0] == 'all_slices'
        jobs.append((plan, x, plan.multislice(*x, crop=32).clone(), torch.cuda.Stream()))
    torch.cuda.synchronize()
    for _ in range(4):
        got = []
        for _ in range(2):
            for plan, x, _, s in jobs:
                with torch.cuda.stream(s):
                    got.append(plan.multislice(*x, crop=32))
        torch.cuda.synchronize()
        for g, (_, _, want, _) in zip(got, jobs + jobs):
            assert torch.equal(g, want)
    for plan, *_ in jobs:
        plan.check()
        plan.close()
