"""Atom windows of many bins: more blocks than a grid's second dimension holds.

Sampled bins against the formula in double; a float32 of the difference to the corner
differs by one rounding at most (2^-23 of the value), plus what the two double
evaluations differ by, 1e-12 of the subtracted corner value."""
import numpy as np
import pytest
import torch
from scipy.special import k0

from namsa_gb300 import engine, msa

pytestmark = pytest.mark.gpu


def window_bin(c, i, j, n, os, rng):
    a, b, cc, d = c
    g = np.linspace(-rng / 2, rng / 2, n)
    r = np.sqrt(g[i * os:(i + 1) * os, None] ** 2 + g[None, j * os:(j + 1) * os] ** 2)
    pre = 4 * np.pi ** 2 * 0.529 * 14.4
    v = sum(pre * a[k] * k0(2 * np.pi * r * np.sqrt(b[k]) + 0.1) + pre / 2 * cc[k] / d[k] * np.exp(-np.pi ** 2 * r * r / d[k])
            for k in range(3))
    return v.mean()


@pytest.mark.parametrize('bins,os,species', [(2000, 8, 1), (1001, 16, 2)])
def test_bins_beyond_65535_blocks(bins, os, species):
    torch.cuda.set_device(0)
    tab = msa.kirkland_table()[[13, 37][:species]]
    n, rng = bins * os, 8.0
    win = engine.atom_windows(torch.from_numpy(tab).cuda(), n, n, os, rng).cpu().numpy()
    assert win.shape == (species, bins, bins)
    for s in range(species):
        corner = window_bin(tab[s], 0, 0, n, os, rng)
        for i, j in ((0, 1), (3, bins // 2), (bins // 2, bins // 2), (bins - 1, 0), (bins - 7, 11), (bins // 2 - 1, bins - 2)):
            want = window_bin(tab[s], i, j, n, os, rng) - corner
            assert abs(win[s, i, j] - want) <= 2.0 ** -23 * abs(want) + 1e-12 * corner
        w = win[s]
        assert np.array_equal(w, w[::-1]) and np.array_equal(w, w[:, ::-1]) and w.min() == 0.0
