"""Uniform weights in FP32: a row's quotient is the FP64 one rounded to its type, also
where that lies at a rounding boundary of FP32 (a double-single quotient's 46 bits do
not tell on which side)."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


def _boundary_weights(rng, ncell):
    """Three FP32 weights a cell: the first over their sum lies within 2^-49 of a midpoint
    of two FP32 numbers, on either side or at it.  The sum needs 52 bits, so FP64 adds
    it exactly in any order."""
    mid = (rng.integers(2 ** 23, 2 ** 24, ncell) * 2.0 + 1) * 2.0 ** -25  # 25 bits, in [0.5, 1)
    w1 = rng.integers(2 ** 23, 2 ** 24, ncell) * 2.0 ** -24
    s = w1 / mid
    w2 = numpy.floor((s - w1) * 2.0 ** 24) * 2.0 ** -24
    w3 = numpy.round((s - w1 - w2) * 2.0 ** 49) * 2.0 ** -49 + rng.integers(-1, 2, ncell) * 2.0 ** -49
    w = numpy.stack([w1, w2, w3], 1)
    ok = (w3 > 2.0 ** -30) & (w3 < 2.0 ** -24) & (w2 > 0)
    w = w[ok].astype(numpy.float32)
    assert w.shape[0] > ncell // 4
    return w


@pytest.mark.parametrize('npol', [1, 2])
def test_quotients_at_rounding_boundaries(arl, npol):
    rng = numpy.random.default_rng(npol)
    N, cell = 128, 2e-3
    w = _boundary_weights(rng, 120 * 120)
    n = w.shape[0]
    im = arl.create_image(npixel=N, cellsize=cell, frequency=numpy.array([1e8]), channel_bandwidth=numpy.array([1e7]),
                          polarisation_frame=arl.PolarisationFrame({1: 'stokesI', 2: 'linearnp'}[npol]),
                          phasecentre=arl.PhaseCentre(0.0, -45.0))
    gcf, cf = arl.create_pswf_convolutionfunction(im, oversampling=8, support=6)
    at = rng.permutation(120 * 120)[:n]
    uv = numpy.stack([at % 120 - 60.0, at // 120 - 60.0, numpy.zeros(n)], 1) / (N * cell)
    uvw = numpy.repeat(uv, 3, axis=0)
    flat = numpy.repeat(w.reshape(-1, 1), npol, axis=1)
    vis = arl.DeviceVisibility(torch.as_tensor(uvw, device='cuda'),
                               torch.full((3 * n,), 1e8, dtype=torch.float64, device='cuda'),
                               torch.zeros((3 * n, npol), dtype=torch.complex64, device='cuda'),
                               torch.as_tensor(flat, device='cuda'), im.polarisation_frame, im.phasecentre)
    got = arl.weight_visibility(vis, im, gcfcf=(gcf, cf)).imaging_weight.cpu().numpy()
    w64 = w.astype(numpy.float64)
    want = (w64 / w64.sum(1, keepdims=True)).astype(numpy.float32)
    assert numpy.array_equal(got, numpy.repeat(want.reshape(-1, 1), npol, axis=1))


def test_quotients_near_the_smallest_normal(arl):
    """One heavy and one faint weight a cell: the faint one's quotient is so small that the
    low part of a double-single one would be a few units of the smallest FP32 number."""
    rng = numpy.random.default_rng(5)
    N, cell, n = 128, 2e-3, 14000
    w = numpy.stack([rng.uniform(1e17, 9e17, n), 10.0 ** rng.uniform(-17.9, -11, n)], 1).astype(numpy.float32)
    im = arl.create_image(npixel=N, cellsize=cell, frequency=numpy.array([1e8]), channel_bandwidth=numpy.array([1e7]),
                          phasecentre=arl.PhaseCentre(0.0, -45.0))
    gcf, cf = arl.create_pswf_convolutionfunction(im, oversampling=8, support=6)
    at = rng.permutation(120 * 120)[:n]
    uv = numpy.stack([at % 120 - 60.0, at // 120 - 60.0, numpy.zeros(n)], 1) / (N * cell)
    vis = arl.DeviceVisibility(torch.as_tensor(numpy.repeat(uv, 2, axis=0), device='cuda'),
                               torch.full((2 * n,), 1e8, dtype=torch.float64, device='cuda'),
                               torch.zeros((2 * n, 1), dtype=torch.complex64, device='cuda'),
                               torch.as_tensor(w.reshape(-1, 1), device='cuda'), im.polarisation_frame, im.phasecentre)
    got = arl.weight_visibility(vis, im, gcfcf=(gcf, cf)).imaging_weight.cpu().numpy()
    w64 = w.astype(numpy.float64)
    want = (w64 / w64.sum(1, keepdims=True)).astype(numpy.float32)
    assert numpy.array_equal(got, want.reshape(-1, 1))
