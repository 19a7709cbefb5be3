"""Row preparation at its limits: more distinct frequencies than channels (the table
fills), histograms on either side of the one-CTA scan's forms, rows on either side of
a block, and non-finite visibilities in the FP32C one-warp gridder."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


@pytest.mark.parametrize('n', [300, 4097, 200000])
@pytest.mark.parametrize('max_chan', [0, 1, 127])
def test_more_frequencies_than_channels(arl, n, max_chan):
    f = torch.as_tensor(numpy.random.default_rng(n).permutation(n) * 1.0, device='cuda')
    assert arl.skycomponents._device_row_channels(f, max_chan, 'cuda')[1] > max_chan


def _pixel_grid(npix):
    """Cell (y, x) holds x + i y."""
    a = torch.arange(npix, dtype=torch.float32, device='cuda')
    return torch.complex(a[None, :].expand(npix, npix), a[:, None].expand(npix, npix))[None, None, None].contiguous()


@pytest.mark.parametrize('npix,subgrid,n', [(64, 16, 1), (64, 16, 255), (64, 16, 257), (1200, 16, 50000),
                                            (1600, 16, 50001)])
def test_rows_find_their_pixels(arl, oracle, npix, subgrid, n):
    """Taps that pick one cell of the window: a row degrids to its pixel's numbers
    exactly.  Bins: 64 (8 a thread in the scan), 22,500 (32 a thread), 40,000 (the
    three-pass scan)."""
    before = arl.tune.get_tuning()
    try:
        arl.tune.set_tuning(subgrid=subgrid)
        cell, S, O = 1e-4, 8, 2
        im = arl.create_image(npixel=npix, cellsize=cell, frequency=numpy.array([1e8]),
                              channel_bandwidth=numpy.array([1e7]), phasecentre=arl.PhaseCentre(0.0, -45.0))
        cf = arl.create_convolutionfunction_from_image(im, oversampling=O, support=S)
        cf.data = numpy.zeros(cf.data.shape, complex)
        cf.data[..., S // 2, S // 2] = 1.0
        rng = numpy.random.default_rng(n)
        uv = rng.uniform(-npix // 2 + 8, npix // 2 - 8, (n, 2)) / (npix * cell)
        uvw = numpy.concatenate([uv, numpy.zeros((n, 1))], 1)
        f = numpy.full(n, 1e8)
        img = oracle.image_geometry(npix, cell)
        maps = oracle.convolution_mapping(uvw, f, oracle.grid_axes(img), oracle.cf_axes(img, O, S))
        bad = numpy.arange(n) % 7 == 3 if n > 1 else numpy.zeros(n, bool)
        uvw[bad] *= 1e6
        gd = arl.create_griddata_from_image(im, nw=1)
        gd.data = _pixel_grid(npix)
        vis = arl.DeviceVisibility(torch.as_tensor(uvw, device='cuda'), torch.as_tensor(f, device='cuda'),
                                   torch.zeros((n, 1), dtype=torch.complex64, device='cuda'),
                                   torch.ones((n, 1), dtype=torch.float32, device='cuda'), im.polarisation_frame,
                                   im.phasecentre)
        out = arl.degrid_visibility_from_griddata(vis, gd, cf, precision='fp32c', check=False).vis.cpu().numpy()[:, 0]
        assert numpy.array_equal(out, numpy.where(bad, 0, maps[0] + 1j * maps[2]))
    finally:
        arl.tune.set_tuning(**before)


@pytest.mark.parametrize('value', [complex(numpy.inf, 1.0), complex(1.0, numpy.nan)])
def test_non_finite_visibility_in_many_rows(arl, oracle, value):
    """2^21 rows (the one-warp gridder's FP32C form), one of them not finite: its window's
    cells are not finite, no others, and those equal the grid without the row."""
    n, npix, cell, S, O = 1 << 21, 512, 1e-3, 8, 4
    rng = numpy.random.default_rng(5)
    im = arl.create_image(npixel=npix, cellsize=cell, frequency=numpy.array([1e8]),
                          channel_bandwidth=numpy.array([1e7]), phasecentre=arl.PhaseCentre(0.0, -45.0))
    cf = arl.create_convolutionfunction_from_image(im, oversampling=O, support=S)
    cf.data = numpy.broadcast_to(rng.uniform(0.5, 1.0, (1, 1, 1, O, O, S, S)), cf.data.shape).astype(complex)
    px = rng.integers(-240, 240, (n, 2))
    uvw = torch.as_tensor(numpy.concatenate([px / (npix * cell), numpy.zeros((n, 1))], 1), device='cuda')
    f = torch.full((n,), 1e8, dtype=torch.float64, device='cuda')
    v = torch.view_as_complex(torch.randn((n, 1, 2), device='cuda', generator=torch.Generator('cuda').manual_seed(1)))
    w = torch.ones((n, 1), dtype=torch.float32, device='cuda')
    row = n // 3

    def grid(x):
        v[row, 0] = x
        vis = arl.DeviceVisibility(uvw, f, v, w, im.polarisation_frame, im.phasecentre)
        g, sw = arl.grid_visibility_to_griddata(vis, arl.create_griddata_from_image(im), cf, precision='fp32c')
        return numpy.asarray(torch.as_tensor(g.data).cpu())[0, 0, 0], float(torch.as_tensor(sw).reshape(-1)[0])
    got, sw = grid(value)
    want, want_sw = grid(0.0)
    img = oracle.image_geometry(npix, cell)
    maps = oracle.convolution_mapping(uvw[row:row + 1].cpu().numpy(), numpy.array([1e8]), oracle.grid_axes(img),
                                      oracle.cf_axes(img, O, S))
    x, y = int(maps[0][0]), int(maps[2][0])
    hit = numpy.zeros((npix, npix), bool)
    hit[y - 4:y + 4, x - 4:x + 4] = True
    assert not numpy.isfinite(got[hit]).any() and numpy.isfinite(got[~hit]).all()
    assert numpy.max(numpy.abs(got[~hit] - want[~hit])) <= 1e-5 * numpy.max(numpy.abs(want))
    assert sw == want_sw == float(n)
