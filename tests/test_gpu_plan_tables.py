"""Tables that a plan keeps outlive the growth of its other buffers."""
import numpy as np
import pytest
import torch

from namsa_gb300 import engine

pytestmark = pytest.mark.gpu


def test_detector_buffer_growth_keeps_the_constant_table():
    """cbed_waves keeps a constant table in the plan; a detector call with more maps grows the
    partial sums only, and the table is used (and freed) once more afterwards."""
    n, P = 64, 3
    g = torch.Generator('cuda').manual_seed(5)
    z = lambda *s: torch.view_as_complex(torch.randn(s + (2,), generator=g, device='cuda'))
    trans, psik = z(2, n, n), z(n, n)
    norm = torch.tensor([float(n * n)], dtype=torch.float64, device='cuda')
    pos = torch.rand((P, 2), generator=g, device='cuda')
    args = (trans, psik, norm, pos, np.float32(3.0), 0.025, 1.0, np.float32(1.0))
    maps = torch.rand((8, n, n), generator=g, device='cuda')
    plan = engine.Plan(n, n)
    waves = z(P, n, n)
    first = plan.cbed_waves(waves.clone(), norm).clone()
    one = plan.detect(*args, maps[:1])
    eight = plan.detect(*args, maps)
    filler = [torch.full((n, n), 7.0, device='cuda') for _ in range(8)]  # other owners of freed memory
    assert torch.equal(plan.cbed_waves(waves.clone(), norm), first)
    assert torch.equal(eight[:, :1], one) and len(filler) == 8
    plan.close()
