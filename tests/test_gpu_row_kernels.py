"""Row kernels at the sizes and values where their fast forms change to the
general ones: the fixed-point DFT phases, the channel ranks, the integer row
mapping (checked through the weight grid and the degridder) and the run sums of
the gain chi^2.  Against the oracle or NumPy in 64 bits."""
import ctypes

import numpy
import pytest
import torch

from helpers import rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


def _cuda(a):
    return torch.as_tensor(numpy.ascontiguousarray(a), device='cuda')


@pytest.mark.parametrize('n,ncomp,nchan,npol', [(1, 1, 1, 1), (255, 127, 1, 2), (513, 129, 7, 4),
                                                (300, 5, 6500, 1), (155649, 3, 2, 1)])
def test_dft_fixed_point_phase(arl, n, ncomp, nchan, npol):
    """FP32C predict against 64 bits.  Per term the phase rounding (2^-26 turns),
    sine / cosine, flux and product roundings stay below 6 units of 2^-24 of the
    flux, and the sum of ncomp terms adds at most one unit of the flux sum each."""
    rng = numpy.random.default_rng(n)
    uvw = rng.uniform(-1, 1, (n, 3)) * 10.0 ** rng.uniform(0, 5, (n, 1))
    l, m = rng.uniform(-0.6, 0.6, (2, ncomp))
    lmn = numpy.stack([l, m, numpy.sqrt(1 - l * l - m * m) - 1], 1)
    lmn[0] = (0.6, -0.8, -1.0)  # the horizon: n = -1 lies outside the fixed-point range
    flux = rng.uniform(0.1, 3.0, (ncomp, nchan, npol))
    chan = rng.integers(0, nchan, n).astype(numpy.int32)
    vis = torch.zeros((n, npol), dtype=torch.complex64, device='cuda')
    arl.skycomponents.dft_predict(_cuda(uvw), _cuda(chan), _cuda(lmn), _cuda(flux), vis, 'fp32c')
    ph = -2 * numpy.pi * (uvw.astype(numpy.longdouble) @ lmn.T.astype(numpy.longdouble))
    want = numpy.einsum('nk,knp->np', numpy.exp(1j * (ph % (2 * numpy.pi)).astype(float)), flux[:, chan])
    bound = (6 + ncomp) * 2.0 ** -24 * flux[:, chan].sum(0)
    assert numpy.all(numpy.abs(vis.cpu().numpy() - want) <= bound)


def test_dft_coordinates_beyond_fixed_point(arl):
    """Rows of 2^31 wavelengths and more: exact phases by construction (multiples of
    1/8 turn), so the FP64 fallback is off by the FP32 sine and cosine alone."""
    u = numpy.array([2.0 ** 31, 2.0 ** 31 - 0.5, -2.0 ** 31, 2.0 ** 40 + 4, 5.0])
    uvw = numpy.stack([u, u, numpy.zeros(5)], 1)
    lmn = numpy.array([[0.25, -0.125, 0.0]])
    vis = torch.zeros((5, 1), dtype=torch.complex64, device='cuda')
    arl.skycomponents.dft_predict(_cuda(uvw), None, _cuda(lmn), _cuda(numpy.ones((1, 1, 1))), vis, 'fp32c')
    want = numpy.exp(-2j * numpy.pi * ((u * 0.125) % 1.0))
    assert numpy.max(numpy.abs(vis.cpu().numpy()[:, 0] - want)) <= 4 * 2.0 ** -24
    vis = torch.zeros((1, 1), dtype=torch.complex64, device='cuda')
    arl.skycomponents.dft_predict(_cuda([[numpy.nan, 1.0, 1.0]]), None, _cuda(lmn), _cuda(numpy.ones((1, 1, 1))), vis,
                                  'fp32c')
    assert bool(torch.isnan(torch.view_as_real(vis)).all())


@pytest.mark.parametrize('values,n', [([1e8], 5), ([-0.0, 0.0, 2.0, -3.0, numpy.inf, -numpy.inf, numpy.nan], 4097),
                                      (list(numpy.linspace(1e8, 2e8, 300)), 20000)])
@pytest.mark.parametrize('slow_axis', [False, True])
def test_row_channels_are_unique_ranks(arl, values, n, slow_axis):
    f = numpy.resize(numpy.asarray(values), n)
    if slow_axis:
        f = numpy.sort(f)[::-1].copy()
    uniq, inv = numpy.unique(f, return_inverse=True)
    got, nchan = arl.skycomponents._device_row_channels(_cuda(f), uniq.size, 'cuda')
    assert nchan == uniq.size
    assert numpy.array_equal(got.cpu().numpy(), inv)
    if uniq.size > 1:
        assert arl.skycomponents._device_row_channels(_cuda(f), uniq.size - 1, 'cuda')[1] > uniq.size - 1


def _edge_rows(arl, gd, cf, O):
    """u, v at, and within a few ulps and 2^-19 sub-pixels of, every kind of
    boundary; planes and channels on their ties; values out of range."""
    cu, cv = gd.grid_wcs.wcs.cdelt[0], gd.grid_wcs.wcs.cdelt[1]
    k = numpy.arange(-9 * O, 9 * O) / (2.0 * O)
    near = numpy.concatenate([[0.0], 2.0 ** -21 * numpy.array([1, -1, 3, -3, 9, -9]) / O])
    u = ((k[:, None] + near) * cu).reshape(-1)
    u = numpy.concatenate([u, numpy.nextafter(u, numpy.inf), numpy.nextafter(u, -numpy.inf)])
    v = numpy.roll(u / cu * cv, 17)
    n = u.size
    w = numpy.resize(numpy.array([0.0, 0.5, -0.5, 1.5, 0.25, -1.0, 0.49999999999, -1.5000000001]), n) * \
        cf.grid_wcs.wcs.cdelt[4]
    f = numpy.resize(numpy.array([1.0e8, 1.05e8, 1.1e8, 1.0499999999e8, 1.15e8]), n)
    return numpy.stack([u, v, w], 1), f


@pytest.mark.parametrize('O,npix', [(8, 64), (16, 100), (2, 64), (6, 64)])
def test_row_mapping_at_boundaries(arl, oracle, O, npix):
    """Degridding a grid of ones with taps that spell each kernel's index gives the
    (sub-pixel, plane) index of every row; the weight grid gives its cell."""
    im = arl.create_image(npixel=npix, cellsize=1e-3, frequency=numpy.array([1.0e8, 1.1e8]),
                          channel_bandwidth=numpy.array([1e7]), phasecentre=arl.PhaseCentre(0.0, -45.0))
    S, nz = 4, 5
    cf = arl.create_convolutionfunction_from_image(im, nz=nz, zstep=37.5, oversampling=O, support=S)
    cf.grid_wcs.wcs.crpix[4] = nz // 2 + 1.0
    idx = numpy.arange(nz)[:, None, None] * O * O + numpy.arange(O)[:, None] * O + numpy.arange(O)
    cf.data = numpy.broadcast_to((idx + 1.0)[None, None, :, :, :, None, None] / S ** 2,
                                 (2, 1, nz, O, O, S, S)).astype(complex)
    gd = arl.create_griddata_from_image(im)
    uvw, f = _edge_rows(arl, gd, cf, O)
    img = oracle.image_geometry(npix, 1e-3, nchan=2, frequency0=1.0e8, channel_bandwidth=1e7)
    gax = oracle.grid_axes(img)
    cax = oracle.cf_axes(img, O, S, nz=nz, zstep=37.5)
    pu, puo, pv, pvo, pwg, pwc, pf = oracle.convolution_mapping(uvw, f, gax, cax)
    ok = oracle.rows_in_grid((pu, puo, pv, pvo, pwg, pwc, pf), gax['shape'], cax['shape'])
    assert 0.3 < ok.mean() < 1.0
    bad = numpy.array([[numpy.nan, 0, 0], [numpy.inf, 0, 0], [1e30, 0, 0], [0, -1e12, 0], [0, 0, numpy.nan]])
    uvw, f = numpy.concatenate([uvw, bad]), numpy.concatenate([f, numpy.full(len(bad), 1e8)])
    n = uvw.shape[0]
    vis = arl.DeviceVisibility(_cuda(uvw), _cuda(f), torch.zeros((n, 1), dtype=torch.complex128, device='cuda'),
                               torch.ones((n, 1), dtype=torch.float64, device='cuda'), im.polarisation_frame,
                               im.phasecentre)
    gd.data[...] = 1.0
    got = arl.degrid_visibility_from_griddata(vis, gd, cf, precision='fp64', check=False).vis.cpu().numpy()[:, 0].real
    want = numpy.zeros(n)
    want[:ok.size][ok] = (pwc * O * O + pvo * O + puo + 1.0)[ok]
    assert numpy.array_equal(numpy.round(got * 64) / 64, want)
    # nearest cells: distinct powers are not needed, a weight per row sums to the oracle's grid
    keep = (numpy.minimum(pu, pv) >= 0) & (numpy.maximum(pu, pv) < npix) & (pwc >= 0) & (pwc < nz) & (pf >= 0) & (pf < 2)
    wt = numpy.random.default_rng(3).integers(1, 100, (ok.size, 1)).astype(float)[keep]
    sub = arl.DeviceVisibility(_cuda(uvw[:ok.size][keep]), _cuda(f[:ok.size][keep]),
                               torch.zeros((len(wt), 1), dtype=torch.complex128, device='cuda'), _cuda(wt),
                               im.polarisation_frame, im.phasecentre)
    grid, sumwt = arl.grid_weight_to_griddata(sub, arl.create_griddata_from_image(im), cf)
    want_g, want_s = oracle.grid_weight(wt, [a[keep] for a in (pu, puo, pv, pvo, pwg, pwc, pf)], gax['shape'])
    assert numpy.array_equal(grid.data, want_g)
    assert numpy.array_equal(sumwt.cpu().numpy(), want_s)


@pytest.mark.parametrize('n,nant,nfreq,npol,offset', [(1, 2, 1, 1, 0), (7, 5, 1, 1, 0), (263, 6, 8, 1, 0),
                                                      (2049, 20, 3, 1, 1), (777, 9, 5, 2, 0)])
@pytest.mark.parametrize('dtype', [numpy.complex64, numpy.complex128])
def test_gain_chi2_runs(arl, n, nant, nfreq, npol, offset, dtype):
    """Runs of one baseline cut at every place, arrays off the 16-byte boundary
    (offset) and baselines in random order.  The sums are FP64: relative to their
    absolute sums they differ from NumPy's by rounding alone (n 2^-52); the
    model gradient is rounded once to its own type."""
    rng = numpy.random.default_rng(n)
    a1, a2 = numpy.triu_indices(nant, 1)
    pick = numpy.repeat(numpy.arange(n) % a1.size if n != 777 else rng.integers(0, a1.size, n), nfreq)[:n]
    a1, a2 = a1[pick].astype(numpy.int32), a2[pick].astype(numpy.int32)
    rnd = lambda *s: rng.normal(size=s) + 1j * rng.normal(size=s)  # noqa: E731
    g, v, m = rnd(nant), rnd(n, npol).astype(dtype), rnd(n, npol).astype(dtype)
    w = rng.uniform(0.1, 2.0, (n, npol)) if npol == 2 else None

    def put(a):
        t = torch.empty(a.size + offset, dtype=_cuda(a).dtype, device='cuda')
        t[offset:] = _cuda(a).reshape(-1)
        return t[offset:].reshape(a.shape)
    M, G = put(m).requires_grad_(True), _cuda(g).requires_grad_(True)
    c = arl.autograd.GainChi2.apply(M, G, put(v), put(a1), put(a2), None if w is None else _cuda(w))
    c.backward()
    r = v.astype(complex) - (g[a2] * g[a1].conj())[:, None] * m
    ww = 1.0 if w is None else w
    assert abs(float(c.detach()) - (ww * abs(r) ** 2).sum()) <= n * 2.0 ** -52 * (ww * abs(r) ** 2).sum() + 1e-300
    want = -2 * ww * (g[a2].conj() * g[a1])[:, None] * r
    eps = 2.0 ** -24 if dtype == numpy.complex64 else 2.0 ** -50
    assert numpy.all(abs(M.grad.cpu().numpy() - want) <= 2 * eps * (abs(want) + 1e-3 * abs(want).max()))
    want_g, scale = numpy.zeros(nant, complex), numpy.zeros(nant)
    d2, d1 = (-2 * ww * r * g[a1][:, None] * m.conj()).sum(1), (-2 * ww * r.conj() * g[a2][:, None] * m).sum(1)
    for a, d in ((a2, d2), (a1, d1)):
        numpy.add.at(want_g, a, d)
        numpy.add.at(scale, a, abs(d))
    # the run sums Q lose the cancellation inside a run: bound by the antenna's absolute sum, a few ulps a row
    assert numpy.all(abs(G.grad.cpu().numpy() - want_g) <= 16 * n * 2.0 ** -53 * (scale + 1e-300))


@pytest.mark.parametrize('nchan,npol,n', [(1, 1, 1), (1, 4, 700), (3, 2, 5000), (4, 1, 8195)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
def test_uniform_weights(arl, nchan, npol, n, dtype):
    """Weights of integers (sums exact in any order), some zero: a row's quotient is
    the FP64 one rounded to its type."""
    rng = numpy.random.default_rng(n + npol)
    N, cell = 32, 2e-3
    frame = {1: 'stokesI', 2: 'linearnp', 4: 'linear'}[npol]
    fr = 1e8 + 1e6 * numpy.arange(nchan)
    im = arl.create_image(npixel=N, cellsize=cell, frequency=fr, channel_bandwidth=numpy.array([1e6]),
                          polarisation_frame=arl.PolarisationFrame(frame), phasecentre=arl.PhaseCentre(0.0, -45.0))
    gcf, cf = arl.create_pswf_convolutionfunction(im, oversampling=8, support=6)
    uvw = rng.uniform(-0.4, 0.4, (n, 3)) / cell
    f = rng.choice(fr, n)
    w = rng.integers(0, 50, (n, npol)).astype(float)
    vis = arl.DeviceVisibility(_cuda(uvw), _cuda(f), torch.zeros((n, npol), dtype=torch.complex64, device='cuda'),
                               _cuda(w).to(dtype), im.polarisation_frame, im.phasecentre)
    got = arl.weight_visibility(vis, im, gcfcf=(gcf, cf)).imaging_weight.cpu().numpy()
    cu = 1.0 / (N * numpy.pi / 180.0 * (-cell * 180.0 / numpy.pi))
    cv = 1.0 / (N * numpy.pi / 180.0 * (cell * 180.0 / numpy.pi))
    pu = numpy.round((uvw[:, 0] / cu + (N // 2 + 1)) - 1.0).astype(int)
    pv = numpy.round((uvw[:, 1] / cv + (N // 2 + 1)) - 1.0).astype(int)
    ch = numpy.round((f - 1e8) / 1e6).astype(int)
    sums = numpy.zeros((nchan, N, N, npol))
    numpy.add.at(sums, (ch, pv, pu), w)
    s = sums[ch, pv, pu]
    want = numpy.where((s != 0).all(1, keepdims=True), w / numpy.where(s != 0, s, 1.0), w)
    assert numpy.array_equal(got, want.astype(got.dtype))
