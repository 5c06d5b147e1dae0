"""Operand and output forms of the persistent tensor-core GEMM that the corrector's sizes decide:
channel counts that make groups of rows bulk runs, 16-byte pieces or single values; odd grids
whose layers are not 16-byte aligned; narrow outputs; several K blocks with a remainder.
"""
import numpy as np
import pytest
import torch

from namsa_gb300 import engine
from oracle import corrector_oracle as CO

pytestmark = pytest.mark.gpu
DEV = 'cuda'


# the tolerances of the network test at its sizes: 3e-3 for the maps, 1e-2 for each gradient
@pytest.mark.parametrize('H,W,Cin,C,L,MX,MY,S', [
    (9, 9, 6, 1, 2, 3, 4, 1),       # 81 values a layer: nothing is aligned
    (10, 13, 5, 2, 2, 5, 6, 3),     # pairs of rows, odd width
    (16, 24, 6, 4, 2, 6, 8, 33),    # groups of 4 rows, samples past one group of row threads
    (24, 16, 3, 16, 1, 8, 12, 70),  # more samples than 64
    (12, 20, 6, 64, 1, 7, 10, 2),   # 64 channels, a K remainder in every transform
    (16, 16, 6, 8, 1, 4, 4, 130),   # more than one tile of samples in the mixing
])
def test_corrector_sizes_match_oracle(H, W, Cin, C, L, MX, MY, S):
    rng = np.random.default_rng(H * W + C)
    net = engine.Corrector(H, W, Cin, C, L, MX, MY, max_samples=S)
    ref = CO.Net(H, W, Cin, C, L, MX, MY, bf16_gemm=True)
    flat = CO.init_params(ref, seed=3, out_scale=0.5)
    flat = (flat + 0.02 * rng.standard_normal(flat.shape)).astype(np.float32)
    net.params.copy_(torch.from_numpy(flat))
    feats = rng.standard_normal((S, H, W, Cin)).astype(np.float32)
    maps = net.forward(torch.from_numpy(feats).to(DEV)).cpu().numpy()
    want, cache = CO.forward(ref, flat.astype(np.float64), feats.astype(np.float64))
    assert np.linalg.norm(maps - want) < 3e-3 * np.linalg.norm(want)
    dmaps = rng.standard_normal(maps.shape).astype(np.float32)
    net.backward(torch.from_numpy(dmaps).to(DEV))
    net.check()
    g = net.grads.cpu().numpy().astype(np.float64)
    gref = CO.backward(ref, cache, dmaps.astype(np.float64))
    o = 0
    for name, shape in ref.layout():
        n = int(np.prod(shape))
        assert np.linalg.norm(g[o:o + n] - gref[o:o + n]) < 1e-2 * max(np.linalg.norm(gref[o:o + n]), 1e-30), name
        o += n


# only the accumulation order differs: the bound of the GEMM tests on random operands
@pytest.mark.parametrize('m,n,k', [(1, 4, 1), (129, 8, 6), (31, 12, 48), (257, 16, 33), (640, 20, 129), (100, 36, 64),
                                   (300, 260, 70)])
@pytest.mark.parametrize('acc', [False, True])
def test_output_columns_in_16_byte_pieces(m, n, k, acc):
    """Aligned rows take whole pieces; the same product into rows one value off takes single values.
    Both are the same numbers."""
    g = torch.Generator().manual_seed(m * n + k)
    a, b, bias = (torch.randn(s, generator=g).to(DEV) for s in ((m, k), (n, k), (n,)))
    c0 = torch.randn(m, n, generator=g).to(DEV)
    ref = a.to(torch.bfloat16).float() @ b.to(torch.bfloat16).float().T + bias + (c0 if acc else 0)
    got = c0.clone()
    engine.gemm_bf16(a, b, bias, out=got, accumulate=acc)
    off = torch.full((m, n + 1), 7.0, device=DEV)
    off[:, 1:] = c0
    engine.gemm_bf16(a, b, bias, out=off[:, 1:], accumulate=acc)
    engine.gemm_check()
    assert torch.allclose(got, ref, rtol=1e-4, atol=1e-4 * k ** 0.5)
    assert torch.equal(off[:, 1:], got) and (off[:, 0] == 7).all()
