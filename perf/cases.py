"""The work that users of this package have it do, as cases that can be timed and checked.

Kinds of case:
  scan       Plan.multislice: CBED patterns of probe positions through a crystal's slices
  host       Plan.multislice_host: the same from and to page-locked host memory
  detect     Plan.detect: detector signals instead of patterns
  batch      Batch.run: many jobs of uneven grid, thickness, voltage and probe count
  build      MSAGPU set-up: atom windows, transmission slices and probe from an atom list
  corrector  Corrector: maps of coarse slices, and the parameter gradients of a training step

Inputs are made in plain torch from a seed: crystals of atoms with random thermal
displacements (a frozen-phonon configuration), binned into slices, each atom a screened
Coulomb potential, so that transmission slices, probes and positions have the values and
spectra of real ones.  Everything is float32 / complex64 as the entry points take it.
"""
import math

import numpy as np
import torch

from namsa_gb300 import MSAGPU, engine

DEV = 'cuda'
PROBE = {'smooth_apert': True, 'apert_smooth': 50, 'spherical_phase': True,
         'aberration_dict': {'C1': 0., 'C3': 1e4, 'C5': 0.}, 'scherzer': False}
GRIDS = (64, 128, 256, 384, 512, 768, 1024)
LARGEST = 1024 * 199 * 512 * 512  # probe-slice pixels of the largest listed case


def listed():
    return [
        # a few patterns of a small cell: the shortest call there is (128^2 Si, as in the smoke run)
        dict(name='cbed_128_p4', kind='scan', ny=128, nx=128, slices=23, probes=4, crop_y=128, crop_x=128, kv=200,
             semi=25e-3, slice_t=5.431 / 4, a=5.431, keep_out=False),
        # one CBED pattern of Si [001], 80 slices of a/4 at 100 keV: the interactive single-probe call
        dict(name='cbed_si256_p1', kind='scan', ny=256, nx=256, slices=80, probes=1, crop_y=256, crop_x=256, kv=100,
             semi=20e-3, slice_t=5.431 / 4, a=5.431, keep_out=False),
        # 64 positions through 1000 Angstrom of thick slices: evaluating a corrected (coarse-slice) crystal
        dict(name='scan_256_p64', kind='scan', ny=256, nx=256, slices=184, probes=64, crop_y=256, crop_x=256, kv=200,
             semi=20e-3, slice_t=5.431, a=5.431, keep_out=False),
        # a short line of positions on the production grid
        dict(name='scan_si512_p16', kind='scan', ny=512, nx=512, slices=199, probes=16, crop_y=256, crop_x=256,
             kv=200, semi=30e-3, slice_t=5.431 / 4, a=5.431, keep_out=False),
        # the full STEM scan: 1024 positions, central 256^2 of each pattern, into a kept stack
        dict(name='scan_si512_p1024', kind='scan', ny=512, nx=512, slices=199, probes=1024, crop_y=256, crop_x=256,
             kv=200, semi=30e-3, slice_t=5.431 / 4, a=5.431, keep_out=True),
        # a non-square cell, an odd number of positions and full patterns at 120 keV
        dict(name='scan_384x768_p77', kind='scan', ny=384, nx=768, slices=66, probes=77, crop_y=384, crop_x=768,
             kv=120, semi=25e-3, slice_t=1.5, a=5.56, keep_out=False),
        # 64 positions on the finest grid (the SrTiO3 precision study, 300 keV, 206 slices of a/2)
        dict(name='scan_sto1024_p64', kind='scan', ny=1024, nx=1024, slices=206, probes=64, crop_y=1024, crop_x=1024,
             kv=300, semi=25e-3, slice_t=3.905 / 2, a=3.905, keep_out=False),
        # a multi-crystal batch: 8 random jobs on 256^2 .. 768^2 grids as one submission
        dict(name='batch_uneven_8', kind='batch', jobs=8, max_grid=768, max_probes=96, max_slices=160, draw_seed=7),
        # bright-field, annular bright-field and annular dark-field signals of a scan, no patterns kept
        dict(name='detect_512_p128', kind='detect', ny=512, nx=512, slices=100, probes=128, kv=200, semi=30e-3,
             slice_t=5.431 / 4, a=5.431, detectors=3),
        # inputs and patterns in page-locked host memory: an application that keeps its data on the host
        dict(name='host_si512_p64', kind='host', ny=512, nx=512, slices=199, probes=64, crop_y=256, crop_x=256,
             kv=200, semi=30e-3, slice_t=5.431 / 4, a=5.431),
        # the set-up every new crystal pays: windows, 199 transmission slices and the probe at 512^2
        dict(name='build_si512', kind='build', n=512, cells=8, layers=50, a=5.431, species='14', slice_t=5.431 / 4,
             kv=200, semi=30e-3),
        # one training step of the coarse-slice corrector: 32 slices at 256^2, maps and all gradients
        dict(name='corrector_256_s32', kind='corrector', n=256, samples=32, channels=32, layers=4, modes_x=32,
             modes_y=64, train=True),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(['scan', 'scan', 'scan', 'scan', 'detect', 'host', 'batch', 'build', 'corrector'])
    if kind == 'batch':
        return dict(kind=kind, jobs=rng.randint(3, 12), max_grid=rng.choice([384, 512, 768]),
                    max_probes=logint(16, 128), max_slices=logint(30, 200), draw_seed=rng.randrange(1 << 20))
    if kind == 'build':
        n = rng.choice(GRIDS[1:])
        a = rng.uniform(3.5, 6.0)
        return dict(kind=kind, n=n, cells=max(1, round(n * 0.085 / a)), layers=rng.randint(4, 50 if n <= 512 else 20),
                    a=a, species=rng.choice(['14', '38 22 8', '79', '31 33']), slice_t=rng.uniform(1.0, 2.0),
                    kv=rng.choice([80, 120, 200, 300]), semi=rng.uniform(15e-3, 30e-3))
    if kind == 'corrector':
        n = rng.choice([128, 256, 512])
        return dict(kind=kind, n=n, samples=max(1, min(logint(1, 48), 32 * 256 * 256 // (n * n))), channels=32,
                    layers=rng.choice([2, 4]), modes_x=32, modes_y=64, train=rng.random() < 0.6)
    ny = rng.choice(GRIDS)
    nx = ny if rng.random() < 0.6 else rng.choice(GRIDS)
    slices = logint(8, 206)
    probes = logint(1, 1024)
    # at most a quarter of the largest listed work, and states that fit the card several times over
    most = max(1, LARGEST // (4 * slices * ny * nx))
    probes = min(probes, most, (4 << 30) // (ny * nx * 8))
    c = dict(kind=kind, ny=ny, nx=nx, slices=slices, probes=probes, kv=rng.choice([80, 100, 120, 200, 300]),
             semi=rng.uniform(15e-3, 30e-3), slice_t=rng.uniform(1.0, 3.0), a=rng.uniform(3.5, 6.0))
    if kind == 'detect':
        c['detectors'] = rng.randint(1, 4)
    else:
        c['crop_y'] = ny if rng.random() < 0.5 else rng.randint(ny // 4, ny)
        c['crop_x'] = nx if rng.random() < 0.5 else rng.randint(nx // 4, nx)
    if kind == 'scan':
        c['keep_out'] = rng.random() < 0.3
    return c


# ----------------------------------------------------------------------------- inputs
def wavelength(kv):
    v = kv * 1e3
    return 12.2643 / math.sqrt(v + 0.97845e-6 * v * v)


def phase_slices(ny, nx, slices, a, gen, pixel=0.085, peak=1.0):
    """Phases sigma V (slices, ny, nx) float32 of a crystal of cubic cells of about `a`
    Angstrom with thermal displacements: atoms on a pixel grid, each a screened Coulomb
    potential, made with one Fourier product per slice."""
    cy, cx = max(1, round(ny * pixel / a)), max(1, round(nx * pixel / a))
    per = 2 * cy * cx  # atoms of a slice: two per cell
    gy, gx = torch.meshgrid(torch.arange(cy), torch.arange(cx), indexing='ij')
    base = torch.stack([gy.reshape(-1), gx.reshape(-1)], 1).repeat(2, 1).double()
    base[per // 2:] += 0.5
    base = base.to(DEV)
    shift = torch.tensor([[0., 0.], [.25, .25], [.5, 0.], [.75, .25]], dtype=torch.float64, device=DEV)
    frac = base[None] + shift[torch.arange(slices, device=DEV) % 4][:, None]
    size = torch.tensor([ny / cy, nx / cx], dtype=torch.float64, device=DEV)
    u = torch.randn((slices, per, 2), generator=gen, device=DEV, dtype=torch.float64) * (0.08 / pixel)
    px = torch.floor(frac * size + u).long()
    py, px = px[..., 0] % ny, px[..., 1] % nx
    idx = (torch.arange(slices, device=DEV)[:, None] * ny + py) * nx + px
    grid = torch.zeros(slices * ny * nx, dtype=torch.float32, device=DEV)
    grid.index_add_(0, idx.reshape(-1), torch.ones(idx.numel(), device=DEV))  # whole numbers: exact in any order
    grid = grid.view(slices, ny, nx)
    ky = torch.fft.fftfreq(ny, pixel, device=DEV)[:, None]
    kx = torch.fft.rfftfreq(nx, pixel, device=DEV)[None]
    k2 = ky * ky + kx * kx
    form = torch.exp(-k2 / 16.0) / (k2 + 0.15 ** 2)
    one = torch.zeros((ny, nx), device=DEV)
    one[0, 0] = 1
    form = form * (0.4 * peak / torch.fft.irfft2(torch.fft.rfft2(one) * form, s=(ny, nx))[0, 0])
    for s in range(0, slices, 16):
        grid[s:s + 16] = torch.fft.irfft2(torch.fft.rfft2(grid[s:s + 16]) * form, s=(ny, nx))
    return grid


def centred(n, kmax):
    """The k axis j kmax / (n - 1) - kmax / 2 in double."""
    km = float(np.float32(kmax))
    return torch.arange(n, dtype=torch.float64, device=DEV) * km / (n - 1) - km / 2


def krad(ny, nx, kmax):
    return torch.sqrt(centred(ny, kmax)[:, None] ** 2 + centred(nx, kmax)[None] ** 2)


def scan_inputs(c, seed, pixel=0.085):
    """trans, psi_k, norm, positions and the optics of a multislice call."""
    gen = torch.Generator(DEV).manual_seed(seed)
    ny, nx = c['ny'], c['nx']
    ph = phase_slices(ny, nx, c['slices'], c['a'], gen, pixel)
    trans = torch.polar(torch.ones_like(ph), ph)
    kmax, lam = np.float32(1 / pixel), wavelength(c['kv'])
    k = krad(ny, nx, kmax)
    ks = c['semi'] / lam
    kl2 = (k * lam) ** 2
    chi = 2 * math.pi / lam * 0.25 * 1e4 * kl2 * kl2  # Cs = 1 um
    psik = torch.polar(torch.sigmoid(160.0 * (ks - k)), -chi).to(torch.complex64)
    norm = (psik.to(torch.complex128).abs().square().sum() * (ny * nx)).reshape(1)
    ext = torch.tensor([ny * pixel, nx * pixel], device=DEV)
    pos = ((torch.rand((c['probes'], 2), generator=gen, device=DEV) - 0.5) * 0.8 * ext).float()
    return dict(trans=trans, psik=psik, norm=norm, positions=pos, kmax=kmax, lam=lam, slice_t=float(c['slice_t']),
                k_band=np.float32(float(kmax) / 3))


def detector_maps(c, kmax):
    """Bright field, annular bright field and annular dark field rings over the k grid."""
    k = krad(c['ny'], c['nx'], kmax)
    ks = c['semi'] / wavelength(c['kv'])
    rings = [(0.0, 1.0), (0.5, 1.0), (1.2, 3.0), (2.0, 5.0)][:c['detectors']]
    return torch.stack([((k >= lo * ks) & (k < hi * ks)).float() for lo, hi in rings])


def batch_specs(c):
    """The jobs of an uneven batch: grids, thicknesses, voltages and probe counts from the case's own seed."""
    rng = np.random.default_rng(c['draw_seed'])
    grids = [g for g in (256, 384, 512, 768) if g <= c['max_grid']]
    out = []
    for _ in range(c['jobs']):
        n = int(rng.choice(grids))
        out.append(dict(ny=n, nx=n, slices=int(rng.integers(c['max_slices'] // 4, c['max_slices'] + 1)),
                        probes=int(rng.integers(min(16, c['max_probes']), c['max_probes'] + 1)), a=float(rng.uniform(3, 8)),
                        kv=int(rng.choice([80, 120, 200, 300])), semi=25e-3, slice_t=float(rng.uniform(1, 2))))
    return out


def atom_list(c, seed):
    """Structured atom array of a tiled cubic cell (diamond for one species, rock salt or
    perovskite sites for more) with thermal displacements of 0.08 Angstrom."""
    zs = [int(z) for z in c['species'].split()]
    if len(zs) == 1:
        basis = [(0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0), (.25, .25, .25), (.25, .75, .75), (.75, .25, .75),
                 (.75, .75, .25)]
        bz = zs * 8
    elif len(zs) == 2:
        basis, bz = [(0, 0, 0), (.25, .25, .25), (.5, .5, 0), (.75, .75, .25)], [zs[0], zs[1]] * 2
    else:
        basis, bz = [(0, 0, 0), (.5, .5, .5), (.5, .5, 0), (.5, 0, .5), (0, .5, .5)], [zs[0], zs[1]] + [zs[2]] * 3
    m = np.array([c['cells'], c['cells'], c['layers']])
    g = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing='ij'), -1).reshape(-1, 1, 3)
    xyz = ((g + np.array(basis)[None]) * c['a']).reshape(-1, 3)
    xyz += 0.08 * np.random.default_rng(seed).standard_normal(xyz.shape)
    xyz -= xyz.min(0)
    out = np.zeros(len(xyz), [('atomic_number', 'i'), ('x', 'f'), ('y', 'f'), ('z', 'f'), ('occ', 'f'), ('DW', 'f')])
    out['atomic_number'] = np.tile(bz, len(g))
    out['x'], out['y'], out['z'], out['occ'] = xyz[:, 0], xyz[:, 1], xyz[:, 2], 1
    return out


def corrector_inputs(c, seed):
    """Features (S, n, n, 6) of coarse slices, d loss / d maps and seeded parameters."""
    gen = torch.Generator(DEV).manual_seed(seed)
    n, S, C, L = c['n'], c['samples'], c['channels'], c['layers']
    ph = phase_slices(n, n, 4 * S, 5.431, gen).view(S, 4, n, n).permute(0, 2, 3, 1)
    feats = torch.cat([ph, ph.sum(3, keepdim=True), torch.full((S, n, n, 1), 0.68, device=DEV)], 3).contiguous()
    dmaps = torch.randn((S, n, n, 4), generator=gen, device=DEV) * 1e-4
    parts = []

    def add(shape, scale):
        parts.append((torch.randn(shape, generator=gen, device=DEV) * scale).reshape(-1))
    add((C, 6), 6 ** -0.5)
    add((C,), 0.05)
    for _ in range(L):
        add((c['modes_x'], c['modes_y'], C, C, 2), 0.5 / C)
        add((C, C), C ** -0.5)
        add((C,), 0.05)
    add((C, C), C ** -0.5)
    add((C,), 0.05)
    add((4, C), 0.3 * C ** -0.5)
    add((4,), 0.01)
    return feats, dmaps, torch.cat(parts)


# ----------------------------------------------------------------------------- the cases
def prepare(case, seed):
    kind = case['kind']
    if kind == 'build':
        return dict(case=case, sites=atom_list(case, seed))
    if kind == 'corrector':
        feats, dmaps, flat = corrector_inputs(case, seed)
        net = engine.Corrector(case['n'], case['n'], 6, case['channels'], case['layers'], case['modes_x'],
                               case['modes_y'], max_samples=case['samples'])
        net.params.copy_(flat)
        return dict(case=case, net=net, feats=feats, dmaps=dmaps)
    if kind == 'batch':
        jobs = []
        for k, s in enumerate(batch_specs(case)):
            j = scan_inputs(s, seed * 1000 + k, 0.12)
            j['out'] = torch.empty((s['probes'], s['ny'], s['nx']), dtype=torch.float32, device=DEV)
            jobs.append(j)
        return dict(case=case, batch=engine.Batch(), jobs=jobs)
    i = scan_inputs(case, seed)
    st = dict(case=case, i=i, plan=engine.Plan(case['ny'], case['nx']))
    if kind == 'detect':
        st['maps'] = detector_maps(case, i['kmax'])
        return st
    if kind == 'host':
        for k in ('trans', 'psik', 'positions'):
            i[k] = i[k].cpu().pin_memory()
        i['norm'] = float(i['norm'].item())
        st['out'] = torch.empty((case['probes'], case['crop_y'], case['crop_x']), dtype=torch.float32, pin_memory=True)
        return st
    st['out'] = torch.empty((case['probes'], case['crop_y'], case['crop_x']), dtype=torch.float32,
                            device=DEV) if case['keep_out'] else None
    return st


def run(state):
    c = state['case']
    kind = c['kind']
    if kind == 'build':
        sim = MSAGPU(c['kv'], c['semi'], state['sites'], sampling=np.array([c['n'], c['n']]), debye_waller=False)
        sim.setup_device(torch.cuda.current_device())
        sim.calc_atomic_potentials()
        sim.build_potential_slices(c['slice_t'])
        sim.build_probe(PROBE)
        return dict(trans=sim.trans, windows=sim.windows, psik=sim.psi_k_dev, aperture=sim.apert_dev, norm=sim.norm_dev)
    if kind == 'corrector':
        net = state['net']
        maps = net.forward(state['feats'])
        if not c['train']:
            return maps
        net.backward(state['dmaps'])
        return dict(maps=maps, grads=net.grads.clone())  # the network's own buffer changes with its next step
    if kind == 'batch':
        return state['batch'].run(state['jobs'])
    i, plan = state['i'], state['plan']
    args = (i['trans'], i['psik'], i['norm'], i['positions'], i['kmax'], i['lam'], i['slice_t'], i['k_band'])
    if kind == 'detect':
        return plan.detect(*args, state['maps'])
    crop = (c['crop_y'], c['crop_x'])
    if kind == 'host':
        out = plan.multislice_host(*args, crop=crop, out=state['out'])
        torch.cuda.current_stream().synchronize()  # the call is asynchronous: its host result is read after this
        return out
    return plan.multislice(*args, crop=crop, out=state['out'])


def scan_work(c, out_words):
    """Inputs and outputs once; per probe and slice the transforms of every row (both
    ways), of the two thirds of the columns inside the band (both ways), and the two
    element-wise complex products."""
    n = c['ny'] * c['nx']
    fl = 10.0 * n * (math.log2(c['nx']) + 2 / 3 * math.log2(c['ny'])) + 10.0 * n
    return dict(bytes=8.0 * n * (c['slices'] + 1) + 8.0 * c['probes'] + 4.0 * out_words,
                flops=fl * c['slices'] * c['probes'])


def work(case):
    kind = case['kind']
    if kind == 'batch':
        w = [scan_work(s, s['probes'] * s['ny'] * s['nx']) for s in batch_specs(case)]
        return dict(bytes=sum(x['bytes'] for x in w), flops=sum(x['flops'] for x in w))
    if kind == 'build':
        s = math.floor(case['layers'] * case['a'] / case['slice_t'])
        return dict(bytes=8.0 * s * case['n'] ** 2 + 12.0 * case['n'] ** 2, flops=0)
    if kind == 'corrector':
        C, L, n, S = case['channels'], case['layers'], case['n'], case['samples']
        mx, my = case['modes_x'], case['modes_y']
        px = S * n * n
        # one layer: pointwise product, x transforms, y transforms and mode mixing
        layer = 2.0 * px * C * C + 2 * 2.0 * px * C * 2 * mx + 2 * 8.0 * S * C * mx * my * n + 8.0 * S * mx * my * C * C
        fwd = L * layer + 2.0 * px * C * (6 + C + 4)
        params = L * (2.0 * mx * my * C * C + C * C)
        return dict(bytes=4.0 * (px * (6 + 4 + (4 if case['train'] else 0)) + params * (2 if case['train'] else 1)),
                    flops=fwd * (3 if case['train'] else 1))
    if kind == 'detect':
        w = scan_work(case, case['probes'] * case['detectors'])
        w['bytes'] += 4.0 * case['detectors'] * case['ny'] * case['nx']
        return w
    return scan_work(case, case['probes'] * case['crop_y'] * case['crop_x'])


# ----------------------------------------------------------------------------- 64-bit values
def exact_scan(c, i, crop=None, maps=None):
    """CBED patterns (or detector signals) by complex128 transforms."""
    ny, nx = i['trans'].shape[1:]
    dev = DEV
    ky, kx = centred(ny, i['kmax']), centred(nx, i['kmax'])
    k = torch.sqrt(ky[:, None] ** 2 + kx[None] ** 2)
    turns = 0.5 * i['lam'] * i['slice_t'] * k * k
    prop = torch.polar(torch.ones_like(turns), -2 * math.pi * (turns - turns.round()))
    prop = prop * (k.float() < float(i['k_band']))
    sign = 1 - 2 * ((torch.arange(ny, device=dev)[:, None] + torch.arange(nx, device=dev)[None]) % 2).double()
    probe = i['psik'].to(dev).to(torch.complex128) * sign
    norm = float(i['norm'])
    pos = i['positions'].to(dev).double()
    trans = i['trans'].to(dev)
    y0, x0 = (0, 0) if crop is None else (ny // 2 - crop[0] // 2, nx // 2 - crop[1] // 2)
    cy, cx = (ny, nx) if crop is None else crop
    out = []
    step = max(1, (1 << 25) // (ny * nx))
    for p0 in range(0, pos.shape[0], step):
        p = pos[p0:p0 + step]
        ty, tx = -ky[None] * p[:, :1], -kx[None] * p[:, 1:]
        ey = torch.polar(torch.ones_like(ty), 2 * math.pi * (ty - ty.round()))
        ex = torch.polar(torch.ones_like(tx), 2 * math.pi * (tx - tx.round()))
        psi = torch.fft.ifft2(probe * ey[:, :, None] * ex[:, None, :]) * (ny * nx)
        for s in range(trans.shape[0]):
            f = torch.fft.fft2(psi * trans[s].to(torch.complex128)) * prop
            if s + 1 < trans.shape[0]:
                psi = torch.fft.ifft2(f)
        inten = f.abs().square() / norm / (ny * nx)
        if maps is None:
            out.append(inten[:, y0:y0 + cy, x0:x0 + cx].contiguous())
        else:
            out.append(torch.einsum('pyx,dyx->pd', inten, maps.double()))
    return torch.cat(out)


def exact_build(c, sites):
    """Kirkland windows, transmission slices and probe in double."""
    import namsa_gb300
    import os
    table = np.load(os.path.join(os.path.dirname(namsa_gb300.__file__), 'data', 'kirkland_params.npy'))
    n, os_, rng = c['n'], 2, 8
    xyz = np.column_stack([sites['x'], sites['y'], sites['z']]).astype(np.float32)
    Z = sites['atomic_number']
    uz = np.unique(Z)
    dims = xyz.max(0) - xyz.min(0)
    samp = np.array([n, n])
    kmax = np.min(samp / dims[:2])
    pix = dims[:2][::-1] / samp
    nn = np.floor(rng / pix).astype(np.int64) * os_
    g0 = torch.linspace(-rng / 2, rng / 2, int(nn[0]), dtype=torch.float64, device=DEV)
    g1 = torch.linspace(-rng / 2, rng / 2, int(nn[1]), dtype=torch.float64, device=DEV)
    r = torch.sqrt(g0[:, None] ** 2 + g1[None] ** 2)
    pre = 4 * math.pi ** 2 * 0.529 * 14.4
    wins = []
    for z in uz:
        a, b, cc, d = table[z - 1]
        v = torch.zeros_like(r)
        for q in range(3):
            v += pre * a[q] * torch.special.modified_bessel_k0(2 * math.pi * r * math.sqrt(b[q]) + 0.1)
            v += pre / 2 * cc[q] / d[q] * torch.exp(-math.pi ** 2 * r * r / d[q])
        v = v.view(int(nn[0]) // os_, os_, int(nn[1]) // os_, os_).mean((1, 3))
        wins.append(v - v.min())
    win = torch.stack(wins)
    H, W = win.shape[1:]
    v = c['kv'] * 1e3
    lam = wavelength(c['kv'])
    mc2, ev = 9.1093837139e-31 * 299792458.0 ** 2, 1.602176634e-19 * v
    sigma = float(np.float32(2 * math.pi * (mc2 + ev) / (2 * mc2 + ev) / (lam * v)))
    t = c['slice_t']
    S = int(np.int32(np.floor(np.float32(dims[-1]) / t)))
    px = (xyz[:, :2] / pix[::-1]).astype(np.int32)
    pot = torch.zeros((S, n, n), dtype=torch.float64, device=DEV)
    hy, hx = torch.arange(H, device=DEV), torch.arange(W, device=DEV)
    for s in range(S):
        m = np.logical_and(xyz[:, 2] >= s * t, xyz[:, 2] < (s + 1) * t)
        if not m.any():
            continue
        zi = torch.from_numpy(np.searchsorted(uz, Z[m])).to(DEV)
        ys = torch.from_numpy(np.rint(px[m, 1].astype(np.float32) - np.float32(H * 0.5)).astype(np.int64)).to(DEV)
        ye = torch.from_numpy(np.rint(px[m, 1].astype(np.float32) + np.float32(H * 0.5)).astype(np.int64)).to(DEV)
        xs = torch.from_numpy(np.rint(px[m, 0].astype(np.float32) - np.float32(W * 0.5)).astype(np.int64)).to(DEV)
        xe = torch.from_numpy(np.rint(px[m, 0].astype(np.float32) + np.float32(W * 0.5)).astype(np.int64)).to(DEV)
        yy, xx = ys[:, None] + hy, xs[:, None] + hx
        oky = (yy >= 0) & (yy < n) & (yy < ye[:, None])
        okx = (xx >= 0) & (xx < n) & (xx < xe[:, None])
        ok = oky[:, :, None] & okx[:, None, :]
        lin = (yy.clamp(0, n - 1)[:, :, None] * n + xx.clamp(0, n - 1)[:, None, :])
        pot[s].view(-1).index_add_(0, lin.reshape(-1), (win[zi] * ok).reshape(-1))
    trans = torch.polar(torch.ones_like(pot), pot * sigma)
    k = krad(n, n, np.float32(kmax))
    ks = float(np.float32(c['semi'] / lam))
    ap = 1 / (1 + torch.exp(-160.0 * (ks - k)))
    kl2 = (k * lam) ** 2
    psik = torch.polar(ap, -2 * math.pi / lam * 0.25 * 1e4 * kl2 * kl2)
    return dict(trans=trans, windows=win, psik=psik, aperture=ap, norm=(ap.square().sum() * (n * n)).reshape(1))


def exact_corrector(c, feats, dmaps, flat):
    """Maps and gradients of the network in double, without the bfloat16 rounding of its products."""
    C, L, n, mx, my = c['channels'], c['layers'], c['n'], c['modes_x'], c['modes_y']
    p = flat.double().requires_grad_(c['train'])
    at = [0]

    def take(*shape):
        k = math.prod(shape)
        at[0] += k
        return p[at[0] - k:at[0]].view(shape)

    def gelu(z):
        return torch.nn.functional.gelu(z, approximate='tanh')
    w0, b0 = take(C, 6), take(C)
    layers = [(take(mx, my, C, C, 2), take(C, C), take(C)) for _ in range(L)]
    p1, c1, p2, c2 = take(C, C), take(C), take(4, C), take(4)
    rows = torch.cat([torch.arange(my // 2, device=DEV), torch.arange(n - my // 2, n, device=DEV)])
    maps = []
    for s in range(feats.shape[0]):  # one slice at a time bounds the memory; gradients add up
        x = feats[s:s + 1].double()
        u = x @ w0.T + b0
        for R, w, b in layers:
            f = torch.fft.rfft2(u, dim=(1, 2))[:, rows, :mx]
            f = torch.einsum('xyoc,syxc->syxo', torch.view_as_complex(R.contiguous()), f)
            full = torch.zeros((1, n, n // 2 + 1, C), dtype=torch.complex128, device=DEV)
            full = full.index_put((torch.zeros(1, dtype=torch.long, device=DEV)[:, None, None], rows[None, :, None],
                                   torch.arange(mx, device=DEV)[None, None]), f)
            # real part of the sum over the kept modes, kx >= 1 counted twice
            g = torch.fft.ifft(full, dim=1)
            wt = torch.full((n // 2 + 1, 1), 2.0, dtype=torch.float64, device=DEV)
            wt[0] = 1
            e = 2 * math.pi * ((torch.arange(n, device=DEV)[:, None] * torch.arange(mx, device=DEV)[None]) % n) / n
            e = torch.polar(torch.ones_like(e, dtype=torch.float64), e.double())
            spec = torch.einsum('wx,sxyc->sywc', e, (g * wt)[:, :, :mx].permute(0, 2, 1, 3)).real / n
            u = gelu(spec + u @ w.T + b)
        o = gelu(u @ p1.T + c1) @ p2.T + c2
        if c['train']:
            o.backward(dmaps[s:s + 1].double())
        maps.append(o.detach())
    maps = torch.cat(maps)
    return dict(maps=maps, grads=p.grad) if c['train'] else maps


def exact(case, seed):
    kind = case['kind']
    if kind == 'build':
        return exact_build(case, atom_list(case, seed))
    if kind == 'corrector':
        return exact_corrector(case, *corrector_inputs(case, seed))
    if kind == 'batch':
        specs = batch_specs(case)
        if sum(s['probes'] * s['slices'] * s['ny'] * s['nx'] for s in specs) > 2.0e10:
            return None
        return [exact_scan(s, scan_inputs(s, seed * 1000 + k, 0.12)) for k, s in enumerate(specs)]
    if case['probes'] * case['slices'] * case['ny'] * case['nx'] > 2.0e10:
        return None  # over about 20 seconds of complex128 transforms
    i = scan_inputs(case, seed)
    if kind == 'detect':
        return exact_scan(case, i, maps=detector_maps(case, i['kmax']))
    return exact_scan(case, i, crop=(case['crop_y'], case['crop_x']))
