"""The all-slices kernel against the separate passes on the same inputs.

Both transform every line with the same float32 codelets or with radices of the
same error, so a pattern differs by rounding only: 2e-7 per slice (the growth the
oracle tests use) with a floor of 1e-6."""
import numpy as np
import pytest
import torch

from namsa_gb300 import engine

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def case(ny, nx, S, P, seed, semi=0.12):
    """Random phases, a wide smooth aperture (beyond the band) and random positions."""
    g = torch.Generator(DEV).manual_seed(seed)
    ph = 0.4 * torch.randn((S, ny, nx), generator=g, device=DEV)
    trans = torch.polar(torch.ones_like(ph), ph)
    kmax = np.float32(10.0)
    ky = torch.linspace(-5, 5, ny, device=DEV)[:, None]
    kx = torch.linspace(-5, 5, nx, device=DEV)[None]
    k = torch.sqrt(ky * ky + kx * kx)
    psik = torch.polar(torch.sigmoid(6 * (semi * 40 - k)), 0.3 * k * k)
    norm = (psik.abs().double().square().sum() * (ny * nx)).reshape(1)
    pos = (torch.rand((P, 2), generator=g, device=DEV) - 0.5) * 20
    return trans, psik, norm, pos.float(), kmax, 0.025, 1.7, np.float32(10.0 / 3)


def both(ny, nx, args, call):
    plan = engine.Plan(ny, nx)
    r, c, grp = plan.schedule
    a = call(plan, args)
    plan.check()
    plan.set_schedule(r, c, grp)  # schedules set by hand: the separate passes
    b = call(plan, args)
    plan.check()
    plan.close()
    return a, b


def rel(a, b):
    return float(torch.linalg.vector_norm(a.double() - b.double()) / torch.linalg.vector_norm(b.double()))


# every pair of line lengths; waves that fill a chunk, spill into the next or stay below one;
# two slices (the smallest) and more
SHAPES = [(256, 256, 3, 12), (256, 256, 2, 50), (384, 384, 3, 17), (512, 512, 3, 1), (512, 512, 2, 3), (512, 512, 4, 17),
          (768, 768, 2, 1), (768, 768, 3, 9), (256, 384, 3, 25), (384, 256, 3, 27), (256, 512, 3, 13), (512, 256, 2, 17),
          (256, 768, 2, 12), (768, 256, 2, 13), (384, 512, 3, 12), (512, 384, 2, 14), (384, 768, 2, 21),
          (768, 384, 2, 12), (512, 768, 2, 3), (768, 512, 3, 2)]


@pytest.mark.parametrize('ny,nx,S,P', SHAPES)
def test_matches_separate_passes(ny, nx, S, P):
    torch.cuda.set_device(0)
    a, b = both(ny, nx, case(ny, nx, S, P, ny + nx + P),
                lambda plan, x: plan.multislice(*x, crop=(ny - 3, nx // 2 + 1)))
    assert rel(a, b) < max(1e-6, 2e-7 * S)


def test_groups_of_one_call():
    """More positions than one L2-resident group: several groups, the last one smaller."""
    torch.cuda.set_device(0)
    a, b = both(384, 384, case(384, 384, 3, 150, 5), lambda plan, x: plan.multislice(*x, crop=64))
    assert rel(a, b) < 1e-6


def test_band_limits():
    """A band of a few columns, and one wider than the grid (every column)."""
    torch.cuda.set_device(0)
    for kb in (0.3, 9.0):
        x = list(case(512, 512, 3, 5, 11))
        x[7] = np.float32(kb)
        a, b = both(512, 512, x, lambda plan, y: plan.multislice(*y))
        assert rel(a, b) < 1e-6 and bool(torch.isfinite(a).all())


def test_detector_signals_and_plan_graph():
    torch.cuda.set_device(0)
    x = case(512, 512, 3, 9, 21)
    maps = torch.rand((2, 512, 512), generator=torch.Generator(DEV).manual_seed(2), device=DEV)
    a, b = both(512, 512, x, lambda plan, y: plan.detect(*y, maps))
    assert rel(a, b) < 1e-6
    plan = engine.Plan(512, 512)
    first = plan.multislice(*x).clone()
    out = torch.empty_like(first)
    for _ in range(3):  # replays of the recorded graph
        plan.multislice(*x, out=out)
        assert torch.equal(first, out)
    plan.set_graph(False)
    assert torch.equal(first, plan.multislice(*x))
    plan.close()


def test_host_buffers():
    """msx_multislice_host with uploads of eight slices: the first group runs upload by upload."""
    torch.cuda.set_device(0)
    x = case(512, 512, 19, 70, 31)
    plan = engine.Plan(512, 512)
    want = plan.multislice(*x, crop=32)
    got = plan.multislice_host(x[0].cpu().pin_memory(), x[1].cpu().pin_memory(), float(x[2].item()),
                               x[3].cpu().pin_memory(), *x[4:], crop=32)
    torch.cuda.synchronize()
    plan.check()
    plan.close()
    assert torch.equal(got, want.cpu())


def test_slices_at_an_odd_address_run_through_the_plain_passes():
    """Complex slices that start on an 8-byte boundary: bulk copies need 16."""
    torch.cuda.set_device(0)
    x = list(case(256, 256, 3, 14, 41))
    plan = engine.Plan(256, 256)
    want = plan.multislice(*x)
    buf = torch.empty(x[0].numel() + 1, dtype=torch.complex64, device=DEV)
    view = buf[1:].view(x[0].shape)
    view.copy_(x[0])
    assert view.data_ptr() % 16 == 8
    x[0] = view
    got = plan.multislice(*x)
    plan.check()
    plan.close()
    assert rel(got, want) < 1e-6


@pytest.mark.parametrize('ny,nx,P', [(64, 384, 1), (64, 384, 33), (128, 384, 17), (256, 384, 3), (64, 512, 32), (64, 768, 17),
                                     (128, 768, 9), (384, 768, 8), (384, 64, 5), (384, 128, 30), (768, 64, 25),
                                     (768, 128, 13), (768, 256, 7), (384, 384, 9)])
def test_schedules_of_few_lines(ny, nx, P):
    """Either side of the lines between the schedules of few and of many lines, and groups that
    fall on different sides of one."""
    torch.cuda.set_device(0)
    x = case(ny, nx, 4, P, ny + nx + P)
    a, b = both(ny, nx, x, lambda plan, y: plan.multislice(*y))
    assert rel(a, b) < 1e-6
    plan = engine.Plan(ny, nx, 4)
    assert rel(plan.multislice(*x), b) < 1e-6
    plan.close()
