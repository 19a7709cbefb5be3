"""Hogbom CLEAN where its one-launch minor cycle changes form: rows that are not
whole segments, fewer segments than CTAs, windows other than 0 and 1, a PSF
larger than the image or of odd size, the residual in global memory, more
iterations than one launch takes.  Bit-identical to the oracle's loop."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


def _case(nx, ny, pnx, pny, seed):
    rng = numpy.random.default_rng(seed)
    dirty = rng.normal(size=(nx, ny))
    psf = 0.05 * rng.normal(size=(pnx, pny))
    psf[pnx // 2, pny // 2] = 1.3
    return dirty, psf, rng


@pytest.mark.parametrize('nx,ny,pnx,pny,window,niter', [
    (2, 3, 2, 2, None, 5), (16, 16, 8, 8, None, 20050), (40, 300, 20, 600, 'general', 200),
    (300, 257, 31, 33, '01', 300), (5, 4000, 4, 1000, 'zero', 3), (700, 512, 256, 256, 'negative', 400),
    (2048, 2048, 64, 64, '01', 30), (2300, 2100, 300, 200, 'general', 40), (1, 9, 2, 2, None, 12)])
def test_hogbom_forms(arl, oracle, nx, ny, pnx, pny, window, niter):
    dirty, psf, rng = _case(nx, ny, pnx, pny, nx + ny)
    w = {None: lambda: None, '01': lambda: (rng.random((nx, ny)) < 0.5).astype(float),
         'general': lambda: rng.choice([0.0, 1.0, 0.5, -0.25], (nx, ny)), 'zero': lambda: numpy.zeros((nx, ny)),
         'negative': lambda: -rng.random((nx, ny))}[window]()
    got = arl.hogbom(dirty, psf, w, 0.2, 0.0, niter, 1e-6)
    want = oracle.hogbom(dirty, psf, w, 0.2, 0.0, niter, 1e-6)
    for g, x in zip(got, want):
        assert numpy.array_equal(g, x)


def test_hogbom_stops_at_the_threshold(arl, oracle):
    """Ties (a dirty image of equal peaks, one negative) go to the first pixel."""
    dirty, psf, _ = _case(64, 64, 16, 16, 1)
    dirty[:] = 0.01
    dirty[[50, 7, 7], [3, 60, 21]] = (2.0, -2.0, 2.0)
    got = arl.deconvolution.hogbom_device(dirty, psf, None, 0.5, 0.3, 1000, 0.001)
    want = oracle.hogbom(dirty, psf, None, 0.5, 0.3, 1000, 0.001)
    assert 3 <= got[2] < 1000
    assert numpy.array_equal(got[0].cpu().numpy(), want[0]) and numpy.array_equal(got[1].cpu().numpy(), want[1])


@pytest.mark.parametrize('scale', [1e-280, 1e280])
def test_hogbom_extreme_magnitudes(arl, oracle, scale):
    """Peaks outside the range of the two-step quotient."""
    dirty, psf, _ = _case(64, 64, 16, 16, 2)
    got = arl.hogbom(dirty * scale, psf, None, 0.1, 0.0, 50, 1e-6)
    want = oracle.hogbom(dirty * scale, psf, None, 0.1, 0.0, 50, 1e-6)
    assert numpy.array_equal(got[0], want[0]) and numpy.array_equal(got[1], want[1])
