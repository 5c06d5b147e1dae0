"""Tuning chooses among what was timed and narrows nothing else: calls of other sizes still take
the forms that an untuned plan would give them."""
import pytest
import torch

from namsa_gb300 import engine
from test_gpu_routes import BAND, KMAX
from test_gpu_stream import DEV, case, rel

pytestmark = pytest.mark.gpu


def test_all_slices_with_a_group_larger_than_the_tuned_one():
    """A tuned group of four waves (the passes' groups are capped by the workspace limit) leaves the
    one-kernel form its own groups; 1.3 times faster here, it wins the timing.  Detector sums are
    sized for its groups."""
    torch.cuda.set_device(0)
    x = case(512, 512, 12, 24, 3)
    maps = torch.rand((2, 512, 512), generator=torch.Generator(DEV).manual_seed(4), device=DEV)
    plan = engine.Plan(512, 512)
    want, signals = plan.multislice(*x).clone(), plan.detect(*x, maps).clone()
    (_, _, group), _ = plan.autotune(*x, iters=12, max_workspace_bytes=8 << 20)
    assert group <= 4
    assert plan.route(12, 24, KMAX, BAND)[:2] == ('all_slices', 24)
    assert plan.route(12, 24, KMAX, BAND, detector=True)[:2] == ('all_slices', 24)
    assert rel(plan.multislice(*x), want) < 2.4e-6 and rel(plan.detect(*x, maps), signals) < 2.4e-6
    plan.check()
    plan.close()


def test_clusters_with_a_tuned_group_of_one():
    torch.cuda.set_device(0)
    x = case(128, 128, 5, 4, 7)
    plan = engine.Plan(128, 128)
    want = plan.multislice(*x).clone()
    (_, _, group), _ = plan.autotune(*x, iters=2, max_workspace_bytes=1)
    assert group == 1 and plan.route(5, 4, KMAX, BAND)[0] == 'cluster'
    assert torch.equal(plan.multislice(*x), want)
    plan.close()


def test_schedules_of_few_lines_after_tuning():
    torch.cuda.set_device(0)
    many, one = case(64, 384, 3, 200, 5), case(64, 384, 3, 1, 6)
    plan = engine.Plan(64, 384)
    want = plan.multislice(*one).clone()
    plan.autotune(*many, iters=2)
    assert plan.route(3, 1, KMAX, BAND)[2] and not plan.route(3, 200, KMAX, BAND)[2]
    assert rel(plan.multislice(*one), want) < 1e-6
    plan.autotune(*one, iters=2)  # few lines timed: its winners run
    assert not plan.route(3, 1, KMAX, BAND)[2]
    assert rel(plan.multislice(*one), want) < 1e-6
    plan.close()


def test_tuned_batch():
    torch.cuda.set_device(0)
    jobs, want = [], []
    for ny, nx, P in ((512, 512, 24), (512, 512, 3), (64, 384, 70), (64, 384, 1), (128, 128, 2)):
        x = case(ny, nx, 6, P, ny + P)
        plan = engine.Plan(ny, nx)
        want.append(plan.multislice(*x).clone())
        plan.close()
        jobs.append(dict(zip(('trans', 'psik', 'norm', 'positions', 'kmax', 'lam', 'slice_t', 'k_band'), x),
                         out=torch.empty_like(want[-1])))
    batch = engine.Batch()
    batch.run(jobs)           # plans exist before the tuning
    batch.autotune(jobs, iters=4)
    for _ in range(2):
        for o, w in zip(batch.run(jobs), want):
            torch.cuda.synchronize()
            assert rel(o, w) < 1.2e-6
    batch.check()
    batch.close()


def test_clusters_beyond_the_tuned_group_take_one_launch():
    """Device and host calls: one kernel for all positions, one download."""
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.set_device(0)
    x = case(128, 128, 5, 6, 8)
    plan = engine.Plan(128, 128)
    want = plan.multislice(*x).clone()
    plan.autotune(*x, iters=2, max_workspace_bytes=1)
    host = [t.cpu().pin_memory() for t in (x[0], x[1], x[3])]
    h = plan.multislice_host(host[0], host[1], float(x[2].item()), host[2], *x[4:])
    torch.cuda.synchronize()
    assert torch.equal(h, want.cpu())
    for _ in range(2):  # the first trace of a process starts the tracer late
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            assert torch.equal(plan.multislice(*x), want)
            torch.cuda.synchronize()
    assert sum('resident_kernel' in e.name for e in prof.events()) == 1
    plan.close()
