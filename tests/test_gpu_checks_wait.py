"""The check calls synchronise the device: work on non-blocking streams is over when they
return, so its error words are the ones that they read."""
import pytest
import torch

from namsa_gb300 import engine
from test_gpu_stream import DEV, case

pytestmark = pytest.mark.gpu


def late(work, check):
    """work() behind 50 ms of waiting on a stream of its own, then check()."""
    work()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(100_000_000)
        work()
    check()
    assert s.query()


def test_plan():
    torch.cuda.set_device(0)
    x = case(128, 128, 3, 4, 1)
    plan = engine.Plan(128, 128)
    out = torch.empty((4, 128, 128), dtype=torch.float32, device=DEV)
    late(lambda: plan.multislice(*x, out=out), plan.check)
    plan.close()


def test_gemm_and_tensor_core_dft():
    torch.cuda.set_device(0)
    a, c = torch.randn((256, 64), device=DEV), torch.empty((256, 256), device=DEV)
    late(lambda: engine.gemm_bf16(a, a, out=c), engine.gemm_check)
    x = torch.randn((128, 256), device=DEV, dtype=torch.complex64)
    late(lambda: engine.tc_dft(x, 1), engine.tc_check)
