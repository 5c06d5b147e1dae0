"""Waves held in clusters (small grids, few positions) against the separate passes.

Both run the same line schedules in the same order; the last pass scales by 1/N
and the norm in the same steps, so a pattern differs by float32 rounding of the
few operations that the compiler may fuse differently: 1e-6 relative."""
import numpy as np
import pytest
import torch

from namsa_gb300 import engine
from test_gpu_stream import both, case, rel

pytestmark = pytest.mark.gpu
DEV = 'cuda'

# every pair of lengths; one position, a cluster per position for the cluster sizes 16, 8 and 4, and two
# rounds of clusters of four; two slices (the smallest) and more
SHAPES = [(64, 64, 2, 1), (64, 64, 5, 15), (64, 64, 3, 37), (64, 64, 3, 70), (64, 128, 3, 3), (128, 64, 3, 20),
          (128, 128, 2, 1), (128, 128, 6, 9), (128, 128, 3, 33), (64, 256, 3, 2), (256, 64, 4, 17), (128, 256, 3, 1),
          (256, 128, 2, 8), (128, 256, 3, 30), (256, 128, 3, 15), (256, 256, 2, 1), (256, 256, 7, 6)]


@pytest.mark.parametrize('ny,nx,S,P', SHAPES)
def test_matches_separate_passes(ny, nx, S, P):
    torch.cuda.set_device(0)
    a, b = both(ny, nx, case(ny, nx, S, P, 3 * ny + nx + P),
                lambda plan, x: plan.multislice(*x, crop=(ny - 3, nx // 2 + 1)))
    assert rel(a, b) < 1e-6


@pytest.mark.parametrize('kb', [0.05, 1.3, 4.9, 9.0])
def test_band_widths(kb):
    """One band column, columns that do not divide by the cluster, and the whole grid; full patterns."""
    torch.cuda.set_device(0)
    for ny, nx in ((128, 128), (256, 256), (64, 256)):
        x = list(case(ny, nx, 3, 2, 11))
        x[7] = np.float32(kb)
        a, b = both(ny, nx, x, lambda plan, y: plan.multislice(*y))
        # relative 1e-6, written as a product: a band without a pixel gives empty patterns
        assert bool(torch.isfinite(a).all())
        assert torch.linalg.vector_norm(a.double() - b.double()) <= 1e-6 * torch.linalg.vector_norm(b.double())


def test_streams_host_buffers_and_capture():
    """Calls of one plan from two streams are ordered on the plan; host buffers and a captured call
    give the device call's patterns."""
    torch.cuda.set_device(0)
    x, y = case(128, 128, 9, 4, 1), case(128, 128, 9, 4, 2)
    plan = engine.Plan(128, 128)
    wx, wy = plan.multislice(*x).clone(), plan.multislice(*y).clone()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.cuda.stream(s1):
            a = plan.multislice(*x)
        with torch.cuda.stream(s2):
            b = plan.multislice(*y)
        torch.cuda.synchronize()
        assert torch.equal(a, wx) and torch.equal(b, wy)
    h = plan.multislice_host(x[0].cpu().pin_memory(), x[1].cpu().pin_memory(), float(x[2].item()),
                             x[3].cpu().pin_memory(), *x[4:])
    torch.cuda.synchronize()
    assert torch.equal(h, wx.cpu())
    out = torch.zeros_like(wx)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.multislice(*y, out=out)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, wy)
    plan.check()
    plan.close()


def test_autotuned_plan_keeps_the_clusters():
    """Tuning chooses among the passes; calls that the clusters take still go there, same bits.
    Schedules set by hand are the passes that run."""
    torch.cuda.set_device(0)
    x = case(128, 128, 5, 4, 7)
    plan = engine.Plan(128, 128)
    want = plan.multislice(*x).clone()
    plan.autotune(*x, iters=2)
    assert torch.equal(plan.multislice(*x), want)
    plan.set_schedule(*plan.schedule[:2])
    assert rel(plan.multislice(*x), want) < 1e-6
    plan.close()
