"""Calls of one plan from several streams: the plan's waves, tables, partial sums and
counters are shared, so each call follows the others, whichever kind it is.

The same kernels run on the same inputs, so the results are equal, not close."""
import pytest
import torch

from namsa_gb300 import engine
from test_gpu_stream import DEV, case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,S,P', [(512, 12, 9), (128, 40, 4), (64, 30, 200)])
def test_detector_graph_free_and_recorded_calls_of_one_plan(n, S, P):
    """All slices in one kernel, clusters, and the two passes as a recorded graph."""
    torch.cuda.set_device(0)
    x, y = case(n, n, S, P, 1), case(n, n, S, P, 2)
    maps = torch.rand((3, n, n), generator=torch.Generator(DEV).manual_seed(3), device=DEV)
    plan = engine.Plan(n, n)
    want = plan.multislice(*x).clone()
    signals = plan.detect(*y, maps).clone()
    plan.set_graph(False)
    plain = plan.multislice(*y).clone()
    plan.set_graph(True)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for _ in range(4):
        with torch.cuda.stream(streams[0]):
            a = plan.multislice(*x)
        with torch.cuda.stream(streams[1]):
            b = plan.detect(*y, maps)
        plan.set_graph(False)
        with torch.cuda.stream(streams[2]):
            c = plan.multislice(*y)
        plan.set_graph(True)
        torch.cuda.synchronize()
        assert torch.equal(a, want) and torch.equal(b, signals) and torch.equal(c, plain)
    plan.check()
    plan.close()


def test_first_use_of_the_constant_table_from_two_streams():
    """The table of cbed_waves is there before the first call goes on, whatever its stream waits
    for; a first call under a capture has it too."""
    torch.cuda.set_device(0)
    n, P = 128, 2
    g = torch.Generator(DEV).manual_seed(9)
    waves = torch.view_as_complex(torch.randn((P, n, n, 2), generator=g, device=DEV))
    norm = torch.tensor([float(n * n)], dtype=torch.float64, device=DEV)
    want = torch.fft.fft2(waves.to(torch.complex128) / n).abs().square() * (1.0 / (n * n))
    plan = engine.Plan(n, n)
    a, b = waves.clone(), waves.clone()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        torch.cuda._sleep(100_000_000)
        first = plan.cbed_waves(a, norm)
    with torch.cuda.stream(s2):
        second = plan.cbed_waves(b, norm)
    torch.cuda.synchronize()
    assert torch.equal(first, second) and float((first - want).norm() / want.norm()) < 1e-6
    plan.close()
    plan = engine.Plan(n, n)
    c = waves.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = plan.cbed_waves(c, norm)
    c.copy_(waves)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, first)
    plan.close()
