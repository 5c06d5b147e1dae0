"""Complex slices that start on an 8-byte boundary (bulk copies need 16), and pointers that
are not even that, at every entry point that takes them."""
import ctypes

import pytest
import torch

from namsa_gb300 import engine
from test_gpu_stream import DEV, case, rel

pytestmark = pytest.mark.gpu


def at_eight(t):
    """The same values 8 bytes past a 16-byte boundary."""
    view = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)[1:].view(t.shape)
    view.copy_(t)
    assert view.data_ptr() % 16 == 8
    return view


@pytest.mark.parametrize('ny,nx,P', [(64, 64, 5), (256, 256, 14), (128, 512, 9)])
def test_timing_and_tuning_take_the_plain_passes(ny, nx, P):
    torch.cuda.set_device(0)
    x = list(case(ny, nx, 3, P, 41))
    plan = engine.Plan(ny, nx)
    want = plan.multislice(*x).clone()
    x[0] = at_eight(x[0])
    row, col, waves = plan.profile(*x, iters=2)
    assert row > 0 and col > 0 and waves == P
    plan.autotune(*x, iters=1)
    assert rel(plan.multislice(*x), want) < 1e-6
    plan.check()
    plan.close()


def test_pointers_off_an_8_byte_boundary_are_refused():
    """Refused before anything is launched."""
    torch.cuda.set_device(0)
    lib, p = engine.lib(), engine._ptr
    trans, psik, norm, pos, kmax, lam, t, kb = case(64, 64, 2, 2, 1)
    out = torch.empty((2, 64, 64), dtype=torch.float32, device=DEV)
    waves = torch.empty((2, 64, 64), dtype=torch.complex64, device=DEV)
    tab = torch.empty((64, 64), dtype=torch.complex64, device=DEV)
    plan = engine.Plan(64, 64)
    h, st = plan.handle, engine._stream()
    off = lambda q: ctypes.c_void_p(q.data_ptr() + 4)
    ins = [trans, psik, norm, pos]
    ms = (ctypes.c_float * 3)()
    for bad in range(4):
        a = [off(q) if i == bad else p(q) for i, q in enumerate(ins)]
        head = (h, a[0], 2, a[1], a[2], a[3], 2, float(kmax), lam, t, float(kb))
        assert lib.msx_multislice(*head, p(out), 64, 64, st) == -1
        assert lib.msx_multislice_detect(*head, p(out), 1, p(waves), st) == -1
        assert lib.msx_plan_profile(*head, 1, ms, st) == -1
        assert lib.msx_plan_autotune(*head, 1, 0, None, st) == -1
    assert lib.msx_plan_probe_waves(h, off(psik), p(pos), 2, float(kmax), p(waves), st) == -1
    assert lib.msx_plan_probe_waves(h, p(psik), p(pos), 2, float(kmax), off(waves), st) == -1
    assert lib.msx_plan_step_waves(h, p(waves), 2, off(trans), p(tab), st) == -1
    assert lib.msx_plan_step_waves(h, p(waves), 2, p(trans), off(tab), st) == -1
    assert lib.msx_plan_cbed_waves(h, off(waves), 2, p(norm), p(out), 64, 64, st) == -1
    assert lib.msx_plan_cbed_waves(h, p(waves), 2, off(norm), p(out), 64, 64, st) == -1
    batch = engine.Batch()
    jobs = batch._jobs([dict(trans=trans, psik=psik, norm=norm, positions=pos, kmax=kmax, lam=lam, slice_t=t, k_band=kb,
                             out=out)])
    jobs[0].psi_k_dev = psik.data_ptr() + 4
    assert lib.msx_batch_run(batch._h, ctypes.cast(jobs, ctypes.c_void_p), 1, st) == -1
    batch.close()
    plan.check()
    plan.close()
