"""What ``deconvolve_cube`` refuses, and a blank PSF, for which it has nothing to do:
decided before any device is looked for, as the arguments alone decide it."""
import numpy
import pytest
import torch


def _images(arl):
    def make():
        im = arl.create_image(npixel=16, cellsize=1e-3, frequency=numpy.array([1e8]),
                              channel_bandwidth=numpy.array([1e7]), phasecentre=arl.PhaseCentre(0.0, -45.0))
        im.data = numpy.random.default_rng(1).normal(size=im.data.shape)
        return im
    return make(), make()


@pytest.mark.parametrize('algorithm', ['hogbom', 'msclean'])
@pytest.mark.parametrize('bad,error', [(dict(gain=2.5), AssertionError), (dict(threshold=-1.0), AssertionError),
                                       (dict(niter=0), AssertionError),
                                       (dict(fractional_threshold=1.5), AssertionError),
                                       (dict(window_shape='round'), ValueError)])
def test_bad_arguments(arl, monkeypatch, algorithm, bad, error):
    def none():
        raise RuntimeError('no CUDA device')
    monkeypatch.setattr(arl.device, 'require_cuda', none)
    dirty, psf = _images(arl)
    with pytest.raises(error):
        arl.deconvolve_cube(dirty, psf, algorithm=algorithm, **bad)


@pytest.mark.parametrize('algorithm', ['hogbom', 'msclean'])
@pytest.mark.parametrize('which', [0, 1])
def test_images_that_require_gradients(arl, monkeypatch, algorithm, which):
    monkeypatch.setattr(arl.device, 'require_cuda', lambda: pytest.fail('a device was looked for'))
    images = _images(arl)
    images[which].data = torch.from_numpy(images[which].data).requires_grad_(True)
    with pytest.raises(RuntimeError):
        arl.deconvolve_cube(*images, algorithm=algorithm)


@pytest.mark.parametrize('algorithm', ['hogbom', 'msclean'])
def test_blank_psf(arl, monkeypatch, algorithm):
    monkeypatch.setattr(arl.device, 'require_cuda', lambda: pytest.fail('a device was looked for'))
    dirty, psf = _images(arl)
    psf.data[:] = 0.0
    for im in arl.deconvolve_cube(dirty, psf, algorithm=algorithm, window_shape='quarter'):
        assert im.data.shape == dirty.data.shape and not im.data.any()
