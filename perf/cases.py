"""Timing cases of the imaging path: what a self-calibration or imaging program
calls, at the sizes it calls them with.

A case names a call (``kind``) and its sizes.  Rows are a seeded disk array of
``nants`` antennas tracked for ``ntimes`` hour angles over +/-2 h in ``nfreq``
channels, ordered (time, baseline, channel); the longest baseline just reaches
the edge of the ``npixel`` uv-grid of a field ``fov`` radians wide, so every row
is imaged.  Sizes are those of this repository's five benchmark workloads and
its tests, scaled over the range in between.
"""
import functools
import importlib
import math

import numpy
import torch

arl = importlib.import_module('algorithm-reference-library_gb300')

C_M_S = 299792458.0
FRAMES = {1: 'stokesI', 2: 'linearnp', 4: 'linear'}
CDTYPE = {'fp32c': torch.complex64, 'fp64': torch.complex128}
RDTYPE = {'fp32c': torch.float32, 'fp64': torch.float64}
HA_MAX = math.pi / 6
W_SHARE = 0.37  # |w| <= sin(21.1 deg) of the longest baseline over the tracked hour angles


def _case(kind, nants, ntimes, nfreq, npixel, support=8, oversampling=8, npol=1, fov=0.2, precision='fp32c', **more):
    return dict(kind=kind, nants=nants, ntimes=ntimes, nfreq=nfreq, npixel=npixel, support=support,
                oversampling=oversampling, npol=npol, fov=fov, precision=precision, **more)


def listed():
    cases = {
        # The drop-in user: rows and images as NumPy data models, one dirty image of a
        # short observation (the 64-antenna, 60-time, 512^2 workload).
        'invert_host_small': _case('invert', 64, 60, 1, 512, fov=0.37, host=True),
        # A quick look inside a loop: a few thousand resident rows on 128^2.
        'predict_tiny': _case('predict', 24, 11, 1, 128, fov=0.4, host=False),
        # Reference precision, resident rows, two polarisations, an image size that is not a power of two.
        'invert_fp64': _case('invert', 96, 57, 4, 1000, npol=2, fov=0.3, precision='fp64', host=False),
        # W-projection of the 256-antenna, 4-channel workload: kernels of 8 to 32 taps on 64 w-planes.
        'wproj_grid': _case('grid', 256, 33, 4, 1024, support=32, fov=0.12, nw=64),
        'wproj_degrid': _case('degrid', 256, 33, 4, 1024, support=32, fov=0.12, nw=64),
        # One w-stacked dirty image of the 40 km array, resident between major cycles: the largest call.
        'wstack_invert_8k': _case('wstack_invert', 512, 3, 64, 8192, oversampling=16, fov=0.1, slices=32),
        # The four-polarisation w-stacked predict of a major cycle.
        'wstack_predict_4pol': _case('wstack_predict', 512, 2, 48, 4096, oversampling=16, npol=4, fov=0.23, slices=20),
        # One gradient step of a joint image and gain solve (128 antennas, 8 channels, 240 times).
        'gain_step': _case('gain', 128, 240, 8, 2048, fov=0.6),
        # Uniform weighting of a continuum observation before imaging.
        'uniform_weight': _case('weight', 256, 77, 4, 4096, fov=0.2),
        # Bright components subtracted from or added to the rows by direct transform.
        'dft_predict': _case('dft', 128, 41, 8, 1024, fov=0.2, ncomp=50),
        # The minor cycle between an invert and a predict.
        'hogbom': _case('clean', 0, 0, 0, 1024, niter=1000),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _npixel(rng, lo, hi):
    """Image sizes as users choose them: powers of two mostly, other even sizes too."""
    if rng.random() < 0.65:
        return 2 ** rng.randint(int(math.ceil(math.log2(lo))), int(math.log2(hi)))
    return 2 * _log(rng, lo / 2, hi / 2)


def draw(rng):
    kind = rng.choice(['invert', 'predict', 'grid', 'degrid', 'wstack_invert', 'wstack_predict', 'gain', 'weight',
                       'dft', 'clean'])
    if kind == 'clean':
        return _case('clean', 0, 0, 0, _npixel(rng, 128, 2048), niter=_log(rng, 100, 1500))
    nants, nfreq = _log(rng, 20, 400), _log(rng, 1, 16)
    precision, npol, more = 'fp32c', 1, {}
    support, oversampling, fov = rng.choice([6, 8, 8, 8, 10]), rng.choice([8, 8, 16]), rng.uniform(0.1, 0.5)
    if kind in ('invert', 'predict'):
        more['host'] = rng.random() < 0.3
        precision = rng.choice(['fp32c', 'fp32c', 'fp64'])
        npol = rng.choice([1, 1, 2, 4])
        rows, npixel = _log(rng, 2e3, 5e5 if more['host'] or precision == 'fp64' else 8e6), _npixel(rng, 128, 2048)
    elif kind in ('grid', 'degrid'):
        if rng.random() < 0.5:
            more['nw'], support, oversampling, nfreq = 2 * rng.randint(8, 32), 2 * rng.randint(8, 16), 8, rng.randint(1, 4)
        else:
            more['nw'], npol = 1, rng.choice([1, 1, 4])
        rows, npixel = _log(rng, 1e4, 4e6), _npixel(rng, 256, 2048)
    elif kind.startswith('wstack'):
        more['slices'], npol = rng.randint(3, 32), rng.choice([1, 1, 2, 4])
        rows, npixel = _log(rng, 1e5, 1e7 / npol), _npixel(rng, 512, 4096)
    elif kind == 'gain':
        rows, npixel = _log(rng, 1e4, 1.2e7), _npixel(rng, 256, 2048)
    elif kind == 'weight':
        precision, npol = rng.choice(['fp32c', 'fp32c', 'fp64']), rng.choice([1, 2, 4])
        rows, npixel = _log(rng, 1e4, 1e7), _npixel(rng, 256, 4096)
    else:
        precision, npol, more['ncomp'] = rng.choice(['fp32c', 'fp32c', 'fp64']), rng.choice([1, 1, 2, 4]), _log(rng, 1, 100)
        rows, npixel = _log(rng, 1e4, 3e6 if precision == 'fp32c' else 3e5), 1024
    nbase = nants * (nants - 1) // 2
    ntimes = max(1, int(rows // (nbase * nfreq)))
    while nbase * ntimes * nfreq > 1.3 * rows and nants > 8:
        nants -= 1
        nbase = nants * (nants - 1) // 2
    return _case(kind, nants, ntimes, nfreq, npixel, support, oversampling, npol, fov, precision, **more)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _nrows(case):
    return case['nants'] * (case['nants'] - 1) // 2 * case['ntimes'] * case['nfreq']


def _frequencies(case):
    return numpy.linspace(100e6, 120e6, case['nfreq']) if case['nfreq'] > 1 else numpy.array([100e6])


def _bmax(case):
    """Longest baseline in wavelengths: its kernel window touches the grid's edge."""
    return (0.5 - (case['support'] / 2 + 3) / case['npixel']) * case['npixel'] / case['fov']


def _wstep(case):
    return W_SHARE * _bmax(case) / max(1, case['nw'] // 2 - 1)


def _image(case):
    """Template image: one channel for each row channel under w-projection, else all channels in one."""
    f = _frequencies(case)
    step = f[1] - f[0] if f.size > 1 else 1e6
    if case.get('nw', 1) > 1:
        freq, width = f, step
    else:
        freq, width = f.mean()[None], 2.0 * (f[-1] - f[0]) + step
    return arl.create_image(npixel=case['npixel'], cellsize=case['fov'] / case['npixel'], frequency=freq,
                            channel_bandwidth=numpy.array([width]),
                            polarisation_frame=arl.PolarisationFrame(FRAMES[case['npol']]),
                            phasecentre=arl.PhaseCentre(0.0, -45.0))


@functools.lru_cache(maxsize=4)
def _kernel_of(items):
    """(gcf, cf) of an image geometry: a program makes them once and keeps them for all its rows."""
    case = dict(items)
    im = _image(case)
    if case.get('nw', 1) > 1:
        nw = case['nw']
        planes = (numpy.arange(nw) - nw // 2) * _wstep(case)
        gcf, cf = arl.create_awterm_convolutionfunction(
            im, nw=nw, wstep=_wstep(case), oversampling=case['oversampling'], support=case['support'],
            plane_support=arl.support_schedule(planes, 8, case['support']))
    else:
        gcf, cf = arl.create_pswf_convolutionfunction(im, oversampling=case['oversampling'], support=case['support'])
    if not case.get('host'):
        gcf.data = torch.as_tensor(gcf.data, device='cuda')
    return gcf, cf


def _kernel(case):
    keys = ('nfreq', 'npixel', 'support', 'oversampling', 'npol', 'fov', 'nw', 'host')
    return _kernel_of(tuple((k, case[k]) for k in keys if k in case))


def _rows(case, seed):
    """uvw [n, 3] (wavelengths), frequency [n], antenna1 [n], antenna2 [n] on the GPU."""
    rng = numpy.random.default_rng(seed)
    n, f = case['nants'], _frequencies(case)
    radius = 0.5 * _bmax(case) * C_M_S / f[-1]
    r, th = radius * numpy.sqrt(rng.uniform(size=n)), rng.uniform(0, 2 * numpy.pi, n)
    east, north = r * numpy.cos(th), r * numpy.sin(th)
    h = math.sqrt(0.5)  # latitude and declination -45 degrees
    xyz = torch.as_tensor(numpy.stack([east, -north * h, north * h]), device='cuda')
    ha = torch.linspace(-HA_MAX, HA_MAX, case['ntimes'], dtype=torch.float64, device='cuda')[:, None]
    x, y, z = xyz[:, None, :]
    u = x * ha.cos() - y * ha.sin()
    v0 = x * ha.sin() + y * ha.cos()
    ant = torch.stack([u, h * (z - v0), -h * (z + v0)], dim=-1)          # [time, antenna, 3]
    a1, a2 = (torch.as_tensor(a, device='cuda') for a in numpy.triu_indices(n, 1))
    k = torch.as_tensor(f / C_M_S, device='cuda')
    uvw = ((ant[:, a2] - ant[:, a1])[:, :, None, :] * k[:, None]).reshape(-1, 3)
    shape = (case['ntimes'], a1.numel(), f.size)
    rep = [a.to(torch.int32)[None, :, None].expand(shape).reshape(-1) for a in (a1, a2)]
    freq = torch.as_tensor(f, device='cuda').expand(shape).reshape(-1)
    return uvw.contiguous(), freq.contiguous(), rep[0], rep[1]


def _sources(case, seed, n):
    """(l, m, flux) of n point sources inside the field, flux log-uniform 0.1 to 10."""
    rng = numpy.random.default_rng(seed + 1)
    l, m = rng.uniform(-0.4, 0.4, (2, n)) * case['fov']
    return l, m, numpy.exp(rng.uniform(math.log(0.1), math.log(10.0), n))


def _observe(uvw, l, m, flux, chunk=1 << 19):
    """Sum of the sources' visibilities, 64 bits."""
    s = torch.as_tensor(numpy.stack([l, m, numpy.sqrt(1 - l ** 2 - m ** 2) - 1]), device='cuda')
    fl = torch.as_tensor(flux, device='cuda')
    out = torch.empty(uvw.shape[0], dtype=torch.complex128, device='cuda')
    for b in range(0, uvw.shape[0], chunk):
        ph = -2.0 * math.pi * (uvw[b:b + chunk] @ s)
        out[b:b + chunk] = torch.complex((ph.cos() * fl).sum(1), (ph.sin() * fl).sum(1))
    return out


def _weights(case, seed, n):
    g = torch.Generator(device='cuda').manual_seed(seed + 2)
    return 0.5 + torch.rand((n, case['npol']), generator=g, device='cuda', dtype=RDTYPE[case['precision']])


def _noise(case, seed, n, sigma):
    g = torch.Generator(device='cuda').manual_seed(seed + 3)
    return sigma * torch.randn((n, case['npol']), generator=g, device='cuda', dtype=CDTYPE[case['precision']])


def _model_image(case, seed):
    """[1 or nchan, npol, N, N] model: 100 slightly resolved sources, the polarisations scaled copies."""
    n = case['npixel']
    im = torch.zeros((n, n), dtype=torch.float64, device='cuda')
    l, m, flux = _sources(case, seed, 100)
    y, x = (torch.as_tensor(numpy.round(c / case['fov'] * n).astype(int) + n // 2, device='cuda') for c in (m, l))
    fl = torch.as_tensor(flux, device='cuda')
    for dy in range(-3, 4):
        for dx in range(-3, 4):
            im.index_put_((y + dy, x + dx), fl * math.exp(-0.5 * (dy * dy + dx * dx)), accumulate=True)
    p = torch.tensor([1.0, 0.2, -0.1, 0.05], dtype=torch.float64, device='cuda')[:case['npol']]
    return (im * p[:, None, None])[None].contiguous()


def _inputs(case, seed):
    """The arrays of a case, which prepare() hands to the framework and exact() computes with."""
    if case['kind'] == 'clean':
        return _clean_inputs(case, seed)
    uvw, freq, a1, a2 = _rows(case, seed)
    n, cdt = uvw.shape[0], CDTYPE[case['precision']]
    d = dict(uvw=uvw, freq=freq, a1=a1, a2=a2)
    if case['kind'] in ('invert', 'grid', 'wstack_invert'):
        v = _observe(uvw, *_sources(case, seed, 20))
        d['vis'] = v[:, None].to(cdt) + _noise(case, seed, n, 0.1)
    if case['kind'] == 'gain':
        rng = numpy.random.default_rng(seed + 4)
        g = rng.normal(1.0, 0.1, case['nants']) * numpy.exp(1j * rng.uniform(-math.pi, math.pi, case['nants']))
        g = torch.as_tensor(g, device='cuda')
        v = _observe(uvw, *_sources(case, seed, 20)) * g[a2] * g[a1].conj()
        d['vis'] = v[:, None].to(cdt) + _noise(case, seed, n, 0.01)
        d['gains'] = torch.ones(case['nants'], dtype=torch.complex128, device='cuda')
    if case['kind'] in ('predict', 'wstack_predict', 'gain'):
        d['model'] = _model_image(case, seed)
    if case['kind'] == 'degrid':
        nchan = case['nfreq'] if case['nw'] > 1 else 1
        m = _model_image(case, seed).expand(nchan, -1, -1, -1)
        d['grid'] = _fft(m)[:, :, None].to(cdt).contiguous()
    if case['kind'] == 'dft':
        l, m, flux = _sources(case, seed, case['ncomp'])
        f = _frequencies(case)
        pol = numpy.array([1.0, 0.2, -0.1, 0.05])[:case['npol']]
        d['lm'] = (l, m)
        d['flux'] = flux[:, None, None] * ((f / f[0]) ** -0.7)[None, :, None] * pol
    d['weight'] = _weights(case, seed, n)
    return d


def _clean_inputs(case, seed):
    """A dirty image and the PSF of a sampled uv-plane, peak 1 at the centre."""
    n = case['npixel']
    g = torch.Generator(device='cuda').manual_seed(seed)
    r = (torch.arange(n, device='cuda', dtype=torch.float64) - n // 2) / n
    keep = torch.rand((n, n), generator=g, device='cuda') < 0.5 * torch.exp(-12 * (r[:, None] ** 2 + r ** 2))
    keep = (keep | torch.roll(keep.flip(0, 1), (1, 1), (0, 1))).to(torch.float64)  # u and -u
    psf = _ifft(keep.to(torch.complex128)).real
    peak = float(psf.max())
    rng = numpy.random.default_rng(seed + 1)
    sky = torch.zeros((n, n), dtype=torch.float64, device='cuda')
    yx = torch.as_tensor(rng.integers(n // 4 + 8, 3 * n // 4 - 8, (2, 60)), device='cuda')
    sky.index_put_((yx[0], yx[1]), torch.as_tensor(numpy.exp(rng.uniform(-2.3, 2.3, 60)), device='cuda'),
                   accumulate=True)
    dirty = _ifft(_fft(sky) * keep).real / peak
    dirty = dirty + 1e-3 * torch.randn((n, n), generator=g, device='cuda', dtype=torch.float64)
    return dict(dirty=dirty[None, None].contiguous(), psf=(psf / peak)[None, None].contiguous())


# ---------------------------------------------------------------------------
# What a program has in hand, and the call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    d, kind = _inputs(case, seed), case['kind']
    im = _image(dict(case, nfreq=1) if kind == 'clean' else case)
    s = dict(case=case, im=im)
    if kind == 'clean':
        s['dirty'] = arl.create_image_from_array(d['dirty'], im.wcs, im.polarisation_frame)
        s['psf'] = arl.create_image_from_array(d['psf'], im.wcs, im.polarisation_frame)
        return s
    if kind != 'dft':
        s['gcfcf'] = _kernel(case)
    n, cdt = d['uvw'].shape[0], CDTYPE[case['precision']]
    v = d['vis'] if 'vis' in d else torch.zeros((n, case['npol']), dtype=cdt, device='cuda')
    s['vis'] = arl.DeviceVisibility(d['uvw'], d['freq'], v, d['weight'], im.polarisation_frame, im.phasecentre)
    s['weight'] = d['weight']
    if case.get('host'):
        s['vis'] = arl.Visibility(uvw=d['uvw'].cpu().numpy(), frequency=d['freq'].cpu().numpy(), vis=v.cpu().numpy(),
                                  weight=d['weight'].cpu().numpy(), polarisation_frame=im.polarisation_frame,
                                  phasecentre=im.phasecentre)
    if 'model' in d:
        m = d['model'].cpu().numpy() if case.get('host') else d['model']
        s['model'] = arl.create_image_from_array(m, im.wcs, im.polarisation_frame)
    if kind in ('grid', 'degrid'):
        s['grid'] = arl.create_griddata_on_device(im, precision=case['precision'])
        if 'grid' in d:
            s['grid'].data = d['grid']
    if kind.startswith('wstack'):
        s['imager'] = arl.WStackImager(s['vis'], im, case['slices'], gcfcf=s['gcfcf'], precision=case['precision'])
    if kind == 'gain':
        s['op'] = arl.autograd.GriddingOperator(s['vis'], im, s['gcfcf'], precision=case['precision'])
        s.update(gains=d['gains'], a1=d['a1'], a2=d['a2'])
    if kind == 'dft':
        s['components'] = _components(d, im, case)
    return s


def _components(d, im, case):
    dec0, out = im.phasecentre.dec_rad, []
    for l, m, flux in zip(*d['lm'], d['flux']):
        n = math.sqrt(1 - l * l - m * m)
        dec = math.asin(m * math.cos(dec0) + n * math.sin(dec0))
        ra = math.atan2(l, n * math.cos(dec0) - m * math.sin(dec0))
        out.append(arl.Skycomponent(arl.PhaseCentre(math.degrees(ra), math.degrees(dec)), _frequencies(case), flux=flux,
                                    polarisation_frame=im.polarisation_frame))
    return out


def run(s):
    case = s['case']
    kind, precision = case['kind'], case['precision']
    if kind == 'invert':
        image, sumwt = arl.invert_2d(s['vis'], s['im'], gcfcf=s['gcfcf'], precision=precision)
        return [image.data, sumwt]
    if kind == 'predict':
        return arl.predict_2d(s['vis'], s['model'], gcfcf=s['gcfcf'], precision=precision).vis
    if kind == 'grid':
        grid, sumwt = arl.grid_visibility_to_griddata(s['vis'], s['grid'], s['gcfcf'][1], precision=precision)
        return [grid.data, sumwt]
    if kind == 'degrid':
        return arl.degrid_visibility_from_griddata(s['vis'], s['grid'], s['gcfcf'][1], precision=precision).vis
    if kind == 'wstack_invert':
        return list(s['imager'].invert())
    if kind == 'wstack_predict':
        return s['imager'].predict(s['model'].data)
    if kind == 'gain':
        return list(arl.autograd.gain_chi2_step(s['model'].data, s['gains'], s['vis'].vis, s['op'], s['a1'], s['a2']))
    if kind == 'weight':  # the natural weights are kept, the uniform ones are a new column
        v = s['vis']
        v = arl.DeviceVisibility(v.uvw, v.frequency, v.vis, s['weight'].clone(), v.polarisation_frame, v.phasecentre)
        return arl.weight_visibility(v, s['im'], gcfcf=s['gcfcf']).imaging_weight
    if kind == 'dft':
        v = s['vis']
        v = arl.DeviceVisibility(v.uvw, v.frequency, torch.zeros_like(v.vis), v.imaging_weight, v.polarisation_frame,
                                 v.phasecentre)
        return arl.predict_skycomponent_visibility(v, s['components']).vis
    comp, resid = arl.deconvolve_cube(s['dirty'], s['psf'], algorithm='hogbom', niter=case['niter'], gain=0.1,
                                      threshold=0.0, fractional_threshold=1e-4, window_shape='quarter',
                                      psf_support=case['npixel'] // 4)
    return [comp.data, resid.data]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind, npix = case['kind'], case['npixel'] ** 2
    n, npol = _nrows(case), case['npol']
    c = 16 if case['precision'] == 'fp64' else 8
    if kind == 'clean':
        # each iteration searches the window and subtracts the PSF patch from the residual
        return {'bytes': 8.0 * (3 * npix + npix // 4), 'flops': case['niter'] * 3.0 * npix / 4}
    row, tap = 32, case['support'] ** 2
    if case.get('nw', 1) > 1:  # supports grow with |w|; most rows lie near the small ones
        tap = ((8 + case['support']) / 2) ** 2
    conv = 8.0 * n * npol * tap
    nchan = case['nfreq'] if case.get('nw', 1) > 1 else 1
    plane = nchan * npol * npix
    fft = plane * 5 * math.log2(npix)
    table = case.get('nw', 1) * (case['oversampling'] * case['support']) ** 2 * c
    into, out = n * (row + npol * 1.5 * c), n * (row + npol * c)
    if kind == 'invert':
        return {'bytes': into + table + plane * 8 * 2, 'flops': conv + fft}
    if kind == 'predict':
        return {'bytes': out + table + plane * 8 * 2, 'flops': conv + fft}
    if kind == 'grid':
        return {'bytes': into + table + plane * c, 'flops': conv}
    if kind == 'degrid':
        return {'bytes': out + table + plane * c, 'flops': conv}
    if kind == 'wstack_invert':
        return {'bytes': into + table + plane * (2 * 8 + case['slices'] * c), 'flops': conv + fft * case['slices']}
    if kind == 'wstack_predict':
        return {'bytes': out + table + plane * (2 * 8 + case['slices'] * c), 'flops': conv + fft * case['slices']}
    if kind == 'gain':  # predict, residuals and their gradients, the adjoint
        return {'bytes': 2 * n * row + 8 * n + 4 * n * c + 4 * plane * 8, 'flops': 2 * conv + 2 * fft + 60.0 * n}
    if kind == 'weight':
        return {'bytes': n * (row + npol * c) + 2 * plane * 8, 'flops': 20.0 * n}
    return {'bytes': n * (row + 2 * npol * c), 'flops': n * case['ncomp'] * (10.0 + 4 * npol)}


# ---------------------------------------------------------------------------
# The same in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _fft(a):
    return torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(a, dim=(-2, -1))), dim=(-2, -1))


def _ifft(a):
    return torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(a, dim=(-2, -1))), dim=(-2, -1))


class _Map:
    """Grid cell, kernel offset and channel of each row, each operation rounded on its own as NumPy does."""

    def __init__(self, case, d, cf):
        n, cell = case['npixel'], case['fov'] / case['npixel']
        deg = math.pi / 180.0
        self.n, self.s, self.o = n, case['support'], case['oversampling']
        self.uf, self.u = self._axis(d['uvw'][:, 0], 1.0 / (n * deg * (-cell * 180.0 / math.pi)))
        self.vf, self.v = self._axis(d['uvw'][:, 1], 1.0 / (n * deg * (cell * 180.0 / math.pi)))
        self.ch = torch.zeros_like(self.u)
        self.z = torch.zeros_like(self.u)
        sup = numpy.array([self.s])
        if case.get('nw', 1) > 1:
            f = _frequencies(case)
            step = f[1] - f[0] if f.size > 1 else 1e6
            self.ch = torch.round((d['freq'] - f[0]) / step).long()
            self.z = torch.round((d['uvw'][:, 2] / _wstep(case) + (case['nw'] // 2 + 1.0)) - 1.0).long()
            sup = numpy.asarray(cf.plane_support)
        self.sup = torch.as_tensor(sup, device='cuda').long()[self.z]
        taps = torch.as_tensor(numpy.ascontiguousarray(cf.data[0, 0]), device='cuda')
        self.taps = taps.reshape(-1, self.o, self.o, self.s, self.s)

    def _axis(self, x, cdelt):
        p = torch.round((x / cdelt + float(self.n // 2 + 1)) - 1.0)
        off = x - ((p + 1.0) - float(self.n // 2 + 1)) * cdelt
        f = torch.floor((off / (cdelt / self.o) + float(self.o // 2 + 1)) - 1.0)
        return f.long(), p.long()

    def blocks(self, rows=None):
        """(rows, flat cells [n, sz, sz] in [channel][y][x], taps [n, sz, sz]) of rows of one support."""
        for sz in torch.unique(self.sup).tolist():
            r = self.sup == sz if rows is None else rows & (self.sup == sz)
            r = torch.nonzero(r)[:, 0]
            j = torch.arange(sz, device='cuda') - sz // 2
            lo = self.s // 2 - sz // 2
            step = max(1, (1 << 25) // (sz * sz))
            for b in range(0, r.numel(), step):
                q = r[b:b + step]
                y = (self.ch[q] * self.n + self.v[q])[:, None] + j
                cells = y[:, :, None] * self.n + (self.u[q][:, None] + j)[:, None, :]
                yield q, cells, self.taps[self.z[q], self.vf[q], self.uf[q], lo:lo + sz, lo:lo + sz]

    def grid(self, vis, nchan, rows=None):
        """[nchan, n, n] of one polarisation's weighted visibilities."""
        out = torch.zeros((nchan * self.n * self.n, 2), dtype=torch.float64, device='cuda')
        for q, cells, taps in self.blocks(rows):
            val = torch.view_as_real(taps.conj().resolve_conj() * vis[q][:, None, None])
            out.index_add_(0, cells.reshape(-1), val.reshape(-1, 2))
        return torch.view_as_complex(out).reshape(nchan, self.n, self.n)

    def degrid(self, grid, out, rows=None):
        flat = grid.reshape(-1)
        for q, cells, taps in self.blocks(rows):
            out[q] = (flat[cells] * taps).sum((1, 2))
        return out


def _slices(case, d):
    """Plane of each row, the planes' mean w and a plane's w-beam."""
    w, k = d['uvw'][:, 2], case['slices']
    wmax = float(w.abs().max())
    step = 2.0 * wmax / (k - 1)
    plane = torch.round(((w + wmax) / step + 1.0) - 1.0).long()  # many rows of a planar array sit on a tie at transit
    n = case['npixel']
    x = (torch.arange(n, device='cuda', dtype=torch.float64) - n // 2) / n
    r2 = case['fov'] ** 2 * (x[:, None] ** 2 + x ** 2)
    nterm = torch.where(r2 < 1.0, 1.0 - torch.sqrt((1.0 - r2).clamp_min(0.0)), 0.0)

    def beam(s):
        rows = plane == s
        mean = float(w[rows].mean()) if bool(rows.any()) else 0.0
        return rows, torch.polar((r2 < 1.0).double(), -2.0 * math.pi * mean * nterm)
    return beam


def _exact_clean(case, d):
    n, h = case['npixel'], case['npixel'] // 4
    res = d['dirty'][0, 0].clone()
    psf = d['psf'][0, 0][n // 2 - h:n // 2 + h, n // 2 - h:n // 2 + h].contiguous()
    i = torch.arange(n, device='cuda')
    band = ((i >= n // 4 + 1) & (i < 3 * (n // 4))).to(torch.float64)
    window = band[:, None] * band
    comp, pmax = torch.zeros_like(res), float(psf.max())
    stop = 0.9 * 1e-4 * float(res.abs().max())
    for _ in range(case['niter']):
        at = int((res * window).abs().argmax())
        y, x = at // n, at % n
        mval = float(res[y, x]) * 0.1 / pmax
        comp[y, x] += mval
        y0, y1, x0, x1 = max(0, y - h), min(n, y + h), max(0, x - h), min(n, x + h)
        res[y0:y1, x0:x1] -= psf[y0 - y + h:y1 - y + h, x0 - x + h:x1 - x + h] * mval
        if abs(float(res[y, x])) < stop:
            break
    return [comp[None, None], res[None, None]]


def exact(case, seed):
    d, kind, npol, n2 = _inputs(case, seed), case['kind'], case['npol'], case['npixel'] ** 2
    if kind == 'clean':
        return _exact_clean(case, d)
    uvw, wt = d['uvw'], d['weight'].double()
    if kind == 'dft':
        out = torch.empty((uvw.shape[0], npol), dtype=torch.complex128, device='cuda')
        per = torch.as_tensor(d['flux'], device='cuda')
        ch = torch.arange(uvw.shape[0], device='cuda') % case['nfreq']
        out.zero_()
        for k, (l, m) in enumerate(zip(*d['lm'])):
            ph = -2.0 * math.pi * (uvw[:, 0] * l + uvw[:, 1] * m + uvw[:, 2] * (math.sqrt(1 - l * l - m * m) - 1))
            out += torch.complex(ph.cos(), ph.sin())[:, None] * per[k][ch]
        return out
    gcf, cf = _kernel(case)
    mp = _Map(case, d, cf)
    nchan = case['nfreq'] if case.get('nw', 1) > 1 else 1
    if kind == 'weight':
        cell = mp.v * mp.n + mp.u
        sums = torch.zeros((n2, npol), dtype=torch.float64, device='cuda').index_add_(0, cell, wt)[cell]
        return torch.where((sums != 0).all(1, keepdim=True), wt / sums, wt)
    g = torch.as_tensor(gcf.data, device='cuda')[0, 0]
    sumwt = torch.zeros((nchan, npol), dtype=torch.float64, device='cuda').index_add_(0, mp.ch, wt)
    if kind in ('invert', 'grid', 'wstack_invert'):
        vw = d['vis'].to(torch.complex128) * wt
    if kind == 'grid':
        return [torch.stack([mp.grid(vw[:, p], nchan) for p in range(npol)], 1)[:, :, None], sumwt]
    if kind == 'invert':
        image = torch.stack([_ifft(mp.grid(vw[:, p], nchan)).real for p in range(npol)], 1) * g * n2
        return [image / sumwt[:, :, None, None], sumwt]
    if kind == 'wstack_invert':
        beam, image = _slices(case, d), torch.zeros((1, npol, mp.n, mp.n), dtype=torch.float64, device='cuda')
        for s in range(case['slices']):
            rows, wb = beam(s)
            for p in range(npol):
                image[0, p] += (wb * _ifft(mp.grid(vw[:, p], 1, rows)[0])).real
        return [image * g * n2 / sumwt[:, :, None, None], sumwt]
    out = torch.zeros((uvw.shape[0], npol), dtype=torch.complex128, device='cuda')
    if kind == 'degrid':
        for p in range(npol):
            mp.degrid(d['grid'][:, p, 0].to(torch.complex128), out[:, p])
        return out
    if kind == 'wstack_predict':
        beam = _slices(case, d)
        for s in range(case['slices']):
            rows, wb = beam(s)
            for p in range(npol):
                mp.degrid(_fft(wb.conj() * d['model'][0, p] * g), out[:, p], rows)
        return out
    for p in range(npol):
        mp.degrid(_fft(d['model'][0, p] * g), out[:, p])
    if kind == 'predict':
        return out
    # gain step at unit gains: chi^2 and 2 d/d conj of the image and the gains
    r = d['vis'].to(torch.complex128) - out
    gains = torch.zeros((case['nants'], 2), dtype=torch.float64, device='cuda')
    for at, val in ((d['a2'], -2.0 * r * out.conj()), (d['a1'], -2.0 * r.conj() * out)):
        gains.index_add_(0, at.long(), torch.view_as_real(val[:, 0].contiguous()))
    image = _ifft(mp.grid(-2.0 * r[:, 0], 1)[0]).real * n2 * g
    return [r.abs().square().sum(), image[None, None], torch.view_as_complex(gains)]
