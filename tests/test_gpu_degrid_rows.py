"""The degridder of small-subgrid plans (one polarisation, supports 4 to 8, 2^21 rows and
more): rows find their cells across tiles, planes and channels, rejected rows give zero,
the last warp is short; infinite cells; the gridder's direct rule for few rows."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu

FULL = 1 << 21


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


def _setup(arl, oracle, npix, S, O, nchan, nw, n, seed, span=None):
    rng = numpy.random.default_rng(seed)
    cell, wstep = 1e-3, 50.0
    fr = 1e8 + 1e7 * numpy.arange(nchan)
    im = arl.create_image(npixel=npix, cellsize=cell, frequency=fr, channel_bandwidth=numpy.full(nchan, 1e7),
                          phasecentre=arl.PhaseCentre(0.0, -45.0))
    cf = arl.create_convolutionfunction_from_image(im, oversampling=O, support=S)
    span = npix // 2 - S if span is None else span
    uvw = numpy.concatenate([rng.uniform(-span, span, (n, 2)) / (npix * cell),
                             rng.integers(-(nw // 2), (nw + 1) // 2, (n, 1)) * wstep], 1)
    f = rng.choice(fr, n)
    img = oracle.image_geometry(npix, cell, nchan=nchan, frequency0=1e8, channel_bandwidth=1e7)
    maps = oracle.convolution_mapping(uvw, f, oracle.grid_axes(img, nw, wstep), oracle.cf_axes(img, O, S))
    return im, cf, arl.create_griddata_from_image(im, nw=nw, wstep=wstep), uvw, f, maps


def _rows(arl, im, uvw, f, precision, vis=None):
    n = len(f)
    v = torch.zeros((n, 1), dtype=arl.device.CDTYPE[precision], device='cuda') if vis is None else vis
    return arl.DeviceVisibility(torch.as_tensor(uvw, device='cuda'), torch.as_tensor(f, device='cuda'), v,
                                torch.ones((n, 1), dtype=arl.device.RDTYPE[precision], device='cuda'),
                                im.polarisation_frame, im.phasecentre)


@pytest.mark.parametrize('precision', ['fp32c', 'fp64'])
@pytest.mark.parametrize('S,npix,nchan,nw,extra', [(8, 1000, 1, 1, 0), (8, 257, 2, 3, 37), (6, 300, 1, 2, 1),
                                                   (4, 300, 3, 1, 255)])
def test_rows_find_their_cells(arl, oracle, precision, S, npix, nchan, nw, extra):
    """Taps that pick one cell of the window: a row gives its cell's number exactly."""
    n = FULL + extra
    im, cf, gd, uvw, f, maps = _setup(arl, oracle, npix, S, 4, nchan, nw, n, S + npix)
    cf.data = numpy.zeros(cf.data.shape, complex)
    cf.data[..., S // 2, S // 2] = 1.0
    bad = numpy.arange(n) % 11 == 5
    bad[-40:] = True  # a last warp of rejected rows
    uvw[bad, 0] += 10.0 / 1e-3
    cells = torch.arange(npix, dtype=torch.float64, device='cuda')
    plane = 2000.0 * torch.arange(nchan * nw, dtype=torch.float64, device='cuda').reshape(nchan, 1, nw, 1, 1)
    gd.data = torch.complex(cells.expand(nchan, 1, nw, npix, npix),
                            cells[:, None] + plane.expand(nchan, 1, nw, npix, npix)).to(arl.device.CDTYPE[precision])
    out = arl.degrid_visibility_from_griddata(_rows(arl, im, uvw, f, precision), gd, cf, precision=precision,
                                              check=False).vis.cpu().numpy()[:, 0]
    want = maps[0] + 1j * (maps[2] + 2000.0 * (maps[6] * nw + maps[4]))
    assert numpy.array_equal(out, numpy.where(bad, 0, want))


@pytest.mark.parametrize('precision', ['fp32c', 'fp64'])
@pytest.mark.parametrize('real', [True, False])
def test_infinite_cell(arl, oracle, precision, real):
    """Rows whose window holds the cell are not finite in both parts, no others."""
    n, npix, S = FULL + 3, 300, 8
    im, cf, gd, uvw, f, maps = _setup(arl, oracle, npix, S, 4, 1, 1, n, 7)
    rng = numpy.random.default_rng(1)
    cf.data = rng.uniform(0.5, 1.0, cf.data.shape) + (0 if real else 1j) * rng.uniform(0.5, 1.0, cf.data.shape)
    gd.data[...] = 1 + 1j
    gd.data[0, 0, 0, 140, 160] = complex(numpy.inf, 1.0)
    out = arl.degrid_visibility_from_griddata(_rows(arl, im, uvw, f, precision), gd, cf,
                                              precision=precision).vis.cpu().numpy()[:, 0]
    dx, dy = 160 - maps[0], 140 - maps[2]
    hit = (dx >= -S // 2) & (dx < S // 2) & (dy >= -S // 2) & (dy < S // 2)
    assert hit.any() and not numpy.isfinite(out.real[hit]).any() and not numpy.isfinite(out.imag[hit]).any()
    assert numpy.isfinite(out[~hit]).all()


@pytest.mark.parametrize('S', [2, 4, 6])
@pytest.mark.parametrize('n,span', [(15, 0.4), (16, 0.4), (64, 0.4), (64, 20.0), (71, 3.0), (300, 1.0), (300, 25.0)])
def test_few_rows_near_and_apart(arl, oracle, S, n, span):
    """FP64 gridding of a bin's few rows, through the subgrid or straight to the grid:
    within the rows per cell times 2^-52 of the largest cell."""
    npix = 64
    im, cf, gd, uvw, f, maps = _setup(arl, oracle, npix, S, 4, 1, 1, n, n + S, span)
    rng = numpy.random.default_rng(n)
    cf.data = rng.normal(size=cf.data.shape) + 1j * rng.normal(size=cf.data.shape)
    v = rng.normal(size=(n, 1)) + 1j * rng.normal(size=(n, 1))
    g, sw = arl.grid_visibility_to_griddata(_rows(arl, im, uvw, f, 'fp64', torch.as_tensor(v, device='cuda')), gd, cf,
                                            precision='fp64')
    want, want_sw = oracle.grid_vec(v, numpy.ones((n, 1)), maps, cf.data, (1, 1, 1, npix, npix))
    got = numpy.asarray(torch.as_tensor(g.data).cpu())
    assert numpy.max(numpy.abs(got - want)) <= 4 * n * 2.0 ** -52 * numpy.max(numpy.abs(want))
    assert numpy.allclose(torch.as_tensor(sw).cpu(), want_sw, rtol=1e-14)
