"""Calls that share a host thread's scratch (operand images, split sums, partial losses),
issued from several streams without a wait in between: each gives what it gives alone."""
import pytest
import torch

from namsa_gb300 import engine

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def interleave(call, inputs, rounds=6):
    """call(x) for every input on a stream of its own, against the results one by one."""
    torch.cuda.set_device(0)
    want = [call(x).clone() for x in inputs]
    streams = [torch.cuda.Stream() for _ in inputs]
    torch.cuda.synchronize()
    for _ in range(rounds):
        got = []
        for s, x in zip(streams, inputs):
            with torch.cuda.stream(s):
                got.append(call(x))
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert torch.equal(g, w)


def randn(*shape, seed):
    return torch.randn(shape, generator=torch.Generator(DEV).manual_seed(seed), device=DEV)


# packed B; K split over the persistent kernel (n <= 32); K split with both operands packed
@pytest.mark.parametrize('m,n,k', [(40000, 64, 96), (48, 32, 40000), (64, 256, 20000)])
def test_gemm(m, n, k):
    interleave(lambda x: engine.gemm_bf16(*x), [(randn(m, k, seed=2 * i), randn(n, k, seed=2 * i + 1)) for i in range(3)])
    engine.gemm_check()


def test_tensor_core_dft():
    xs = [torch.view_as_complex(randn(2048, 256, 2, seed=i)) for i in range(3)]
    interleave(lambda x: engine.tc_dft(x, -1), xs)
    engine.tc_check()


def test_corrector_residual():
    def call(x):
        adj = torch.empty_like(x[0])
        loss = torch.empty(1, dtype=torch.float32, device=DEV)
        engine.residual(x[0], x[1], 0.5, adj, loss)
        return loss
    z = lambda i: torch.view_as_complex(randn(8, 256, 256, 2, seed=i))
    interleave(call, [(z(2 * i), z(2 * i + 1)) for i in range(3)])
