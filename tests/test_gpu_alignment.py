"""Complex slices that start on an 8-byte boundary (bulk copies need 16), and pointers that
are not even that, at every entry point that takes them."""
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
