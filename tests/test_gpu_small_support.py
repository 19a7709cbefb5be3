"""The one-warp gridder and the 32-cell subgrid it plans with: supports up to 10, real
and complex taps, rows below and above one batch, one chunk and the direct path,
windows on the tiles' and the grid's edges, non-finite visibilities.  Against the
oracle in 64 bits: relative to the grid's largest cell FP64 sums stay within the rows
per cell times 2^-52, FP32C ones within 1e-6, as everywhere in the suite (its
products round at 2^-24 and sums are compensated).

FP32C takes it from 2 Mi rows: rows repeated that often have the oracle's sums times
the repeats.  A cell of 512^2 then has up to four tiles of up to sixteen chunks added,
each rounded at 2^-25 of the sum and the products at 2^-24: 64 2^-24 + 12 2^-24 < 5e-6."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


def _axes(oracle, npix, nchan, S, O):
    img = oracle.image_geometry(npix, 2e-3, nchan=nchan, npol=1, frequency0=1e8, channel_bandwidth=1e7)
    return oracle.grid_axes(img), oracle.cf_axes(img, O, S)


def _case(arl, oracle, n, S, O, npix, npol, nchan, per_pol, real, seed):
    rng = numpy.random.default_rng(seed)
    cell = 2e-3
    frame = {1: 'stokesI', 2: 'linearnp', 4: 'linear'}[npol]
    freq = 1e8 + 1e7 * numpy.arange(nchan)
    im = arl.create_image(npixel=npix, cellsize=cell, frequency=freq, channel_bandwidth=numpy.array([1e7]),
                          polarisation_frame=arl.PolarisationFrame(frame), phasecentre=arl.PhaseCentre(0.0, -45.0))
    cf = arl.create_convolutionfunction_from_image(im, oversampling=O, support=S)
    shape = (nchan, npol if per_pol else 1, 1, O, O, S, S)
    k = rng.normal(size=shape) + (0 if real else 1j) * rng.normal(size=shape)
    cf.data = numpy.broadcast_to(k, (nchan, npol, 1, O, O, S, S)).astype(complex)
    # pixels from the first to the last position whose window fits, both ends included
    lo, hi = -(npix // 2 - S // 2), npix - S // 2 - npix // 2
    cu, cv = 1.0 / (npix * cell), 1.0 / (npix * cell)
    uv = rng.integers(lo, hi + 1, (n, 2)).astype(float)
    uv[:4] = [[lo, lo], [lo, hi], [hi, lo], [hi, hi]][:n]
    uv = numpy.clip(uv + rng.uniform(-0.45, 0.45, (n, 2)), lo - 0.45, hi + 0.45)
    uvw = numpy.concatenate([uv * [-cu, cv], numpy.zeros((n, 1))], 1)
    f = rng.choice(freq, n)
    v = rng.normal(size=(n, npol)) + 1j * rng.normal(size=(n, npol))
    w = rng.uniform(0.0, 2.0, (n, npol))
    img = oracle.image_geometry(npix, cell, nchan=nchan, npol=npol, frequency0=1e8, channel_bandwidth=1e7)
    gax, cax = oracle.grid_axes(img), oracle.cf_axes(img, O, S)
    maps = oracle.convolution_mapping(uvw, f, gax, cax)
    keep = oracle.rows_in_grid(maps, gax['shape'], cax['shape'])
    uvw, f, v, w, maps = uvw[keep], f[keep], v[keep], w[keep], [m[keep] for m in maps]
    return im, cf, uvw, f, v, w, maps, gax['shape'], arl.PolarisationFrame(frame)


@pytest.mark.parametrize('precision', ['fp32c', 'fp64'])
@pytest.mark.parametrize('n,S,npix,npol,nchan,per_pol,real', [
    (1, 8, 64, 1, 1, False, True), (3, 6, 64, 2, 1, False, False), (33, 2, 32, 1, 1, False, True),
    (300, 4, 48, 1, 3, True, False), (5000, 8, 40, 1, 1, False, True), (5000, 8, 100, 2, 1, True, True),
    (4097, 6, 56, 1, 2, True, False), (4000, 10, 64, 1, 1, False, False), (4000, 10, 64, 2, 1, True, True),
    (700, 8, 64, 4, 1, False, True)])
def test_grid_and_degrid_vs_oracle(arl, oracle, precision, n, S, npix, npol, nchan, per_pol, real):
    im, cf, uvw, f, v, w, maps, shape, frame = _case(arl, oracle, n, S, 4, npix, npol, nchan, per_pol, real, n + S)
    vis = arl.Visibility(uvw=uvw, frequency=f, vis=v, weight=w, imaging_weight=w, polarisation_frame=frame)
    gd, sw = arl.grid_visibility_to_griddata(vis, arl.create_griddata_from_image(im), cf, precision=precision)
    want, want_sw = oracle.grid_vec(v, w, maps, cf.data, shape)
    tol = 1e-6 if precision == 'fp32c' else 1e-12
    assert numpy.max(numpy.abs(gd.data - want)) <= tol * numpy.max(numpy.abs(want))
    assert numpy.allclose(sw, want_sw, rtol=1e-6 if precision == 'fp32c' else 1e-12)
    gd.data[...] = want
    out = arl.degrid_visibility_from_griddata(vis, gd, cf, precision=precision)
    d = oracle.degrid_vec(want, maps, cf.data)
    assert numpy.max(numpy.abs(out.vis - d)) <= 4 * tol * numpy.max(numpy.abs(d))


@pytest.mark.parametrize('S,O,reps,drop,nchan,real', [
    (8, 4, 128, 0, 1, True), (8, 4, 128, 1, 1, True), (8, 16, 128, 0, 3, False), (6, 4, 131, 7, 1, False),
    (4, 2, 128, 0, 2, True), (2, 4, 129, 33, 1, False)])
def test_many_rows_vs_oracle(arl, oracle, S, O, reps, drop, nchan, real):
    im, cf, uvw, f, v, w, maps, shape, frame = _case(arl, oracle, 16384, S, O, 512, 1, nchan, nchan > 1, real, S + O)
    assert len(f) == 16384
    if nchan > 2:  # the last channel: a few rows alone in their tiles, not repeated with the others
        few = numpy.flatnonzero(f == f.max())[3:]
        f = f.copy()
        f[few] = f.min()
        maps = oracle.convolution_mapping(uvw, f, *_axes(oracle, 512, nchan, S, O))
    n = 16384 * reps - drop
    rep = lambda a: numpy.concatenate([a] * reps)[:n]
    vis = arl.Visibility(uvw=rep(uvw), frequency=rep(f), vis=rep(v), weight=rep(w), imaging_weight=rep(w),
                         polarisation_frame=frame)
    gd, sw = arl.grid_visibility_to_griddata(vis, arl.create_griddata_from_image(im), cf, precision='fp32c')
    want, want_sw = oracle.grid_vec(v, w, maps, cf.data, shape)
    want, want_sw = reps * want, reps * want_sw
    if drop:
        less, less_sw = oracle.grid_vec(v[-drop:], w[-drop:], [m[-drop:] for m in maps], cf.data, shape)
        want, want_sw = want - less, want_sw - less_sw
    assert numpy.max(numpy.abs(gd.data - want)) <= 5e-6 * numpy.max(numpy.abs(want))
    assert numpy.allclose(sw, want_sw, rtol=1e-6)
    gd.data[...] = want
    out = arl.degrid_visibility_from_griddata(vis, gd, cf, precision='fp32c')
    d = rep(oracle.degrid_vec(want, maps, cf.data))
    assert numpy.max(numpy.abs(out.vis - d)) <= 4e-6 * numpy.max(numpy.abs(d))


@pytest.mark.parametrize('precision', ['fp64'])
@pytest.mark.parametrize('rows', [1, 200])
def test_non_finite_visibilities_reach_their_cells(arl, oracle, precision, rows):
    """Real taps: a visibility with an infinite real part makes NaN or infinity of the
    window's cells, as the whole complex product does, and of no others."""
    im, cf, uvw, f, v, w, maps, shape, frame = _case(arl, oracle, rows, 8, 4, 64, 1, 1, False, True, 5)
    v = v.copy()
    v[0, 0] = complex(numpy.inf, 1.0)
    vis = arl.Visibility(uvw=uvw, frequency=f, vis=v, weight=w + 0.1, imaging_weight=w + 0.1, polarisation_frame=frame)
    gd, _ = arl.grid_visibility_to_griddata(vis, arl.create_griddata_from_image(im), cf, precision=precision)
    pu, pv = int(maps[0][0]), int(maps[2][0])
    hit = numpy.zeros((64, 64), bool)
    hit[pv - 4:pv + 4, pu - 4:pu + 4] = True
    got = gd.data[0, 0, 0]
    assert not numpy.isfinite(got.real[hit]).any() and not numpy.isfinite(got.imag[hit]).any()
    assert numpy.isfinite(got[~hit]).all()


@pytest.mark.parametrize('rows', [1, 200])
def test_degrid_of_non_finite_cells(arl, oracle, rows):
    """FP64, real taps: an infinite cell makes its rows non-finite in both parts, as the
    whole complex product does, and no others."""
    im, cf, uvw, f, v, w, maps, shape, frame = _case(arl, oracle, rows, 8, 4, 64, 1, 1, False, True, 6)
    vis = arl.Visibility(uvw=uvw, frequency=f, vis=v, weight=w, imaging_weight=w, polarisation_frame=frame)
    gd = arl.create_griddata_from_image(im)
    pu, pv = maps[0].astype(int), maps[2].astype(int)
    x, y = pu[0] - 1, pv[0] + 2
    gd.data[...] = 1 + 1j
    gd.data[0, 0, 0, y, x] = complex(numpy.inf, 1.0)
    out = arl.degrid_visibility_from_griddata(vis, gd, cf, precision='fp64').vis[:, 0]
    hit = (x >= pu - 4) & (x < pu + 4) & (y >= pv - 4) & (y < pv + 4)
    assert hit[0] and not numpy.isfinite(out.real[hit]).any() and not numpy.isfinite(out.imag[hit]).any()
    assert numpy.isfinite(out[~hit]).all()
