"""The four-polarisation degridder on either side of the rows per bin where it is bounded to
three CTAs an SM (24), with eight and sixteen lanes a row."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


@pytest.mark.parametrize('small_rows_degrid', [2, 4])
@pytest.mark.parametrize('n', [1, 33, 383, 384, 600])  # 96^2 pixels: 16 bins
@pytest.mark.parametrize('S', [6, 8])
def test_four_polarisations_vs_oracle(arl, oracle, S, n, small_rows_degrid):
    before = arl.tune.get_tuning()
    try:
        arl.tune.set_tuning(small_rows_degrid=small_rows_degrid)
        rng = numpy.random.default_rng(n + S)
        npix, cell, O = 96, 2e-3, 4
        im = arl.create_image(npixel=npix, cellsize=cell, frequency=numpy.array([1e8]),
                              channel_bandwidth=numpy.array([1e7]), phasecentre=arl.PhaseCentre(0.0, -45.0),
                              polarisation_frame=arl.PolarisationFrame('linear'))
        cf = arl.create_convolutionfunction_from_image(im, oversampling=O, support=S)
        cf.data = rng.normal(size=cf.data.shape) + 1j * rng.normal(size=cf.data.shape)
        uvw = numpy.concatenate([rng.uniform(-40, 40, (n, 2)) / (npix * cell), numpy.zeros((n, 1))], 1)
        f = numpy.full(n, 1e8)
        img = oracle.image_geometry(npix, cell, npol=4, frequency0=1e8, channel_bandwidth=1e7)
        maps = oracle.convolution_mapping(uvw, f, oracle.grid_axes(img), oracle.cf_axes(img, O, S))
        gd = arl.create_griddata_from_image(im)
        gd.data = rng.normal(size=gd.data.shape) + 1j * rng.normal(size=gd.data.shape)
        vis = arl.Visibility(uvw=uvw, frequency=f, vis=numpy.zeros((n, 4), complex), weight=numpy.ones((n, 4)),
                             imaging_weight=numpy.ones((n, 4)), polarisation_frame=im.polarisation_frame)
        out = arl.degrid_visibility_from_griddata(vis, gd, cf, precision='fp32c')
        want = oracle.degrid_vec(gd.data, maps, cf.data)
        assert numpy.max(numpy.abs(out.vis - want)) <= 4e-6 * numpy.max(numpy.abs(want))
    finally:
        arl.tune.set_tuning(**before)
