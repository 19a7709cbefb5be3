"""DFT predict where the phase is zero: a component at the phase centre and a row at
the origin give the flux with an imaginary part of exactly zero, as exp(0) does."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


@pytest.mark.parametrize('precision', ['fp32c', 'fp64'])
@pytest.mark.parametrize('n,npol', [(1, 1), (700, 4), (155649, 1)])
def test_component_at_the_phase_centre(arl, n, npol, precision):
    rng = numpy.random.default_rng(n)
    uvw = torch.as_tensor(rng.uniform(-1, 1, (n, 3)) * 10.0 ** rng.uniform(0, 5, (n, 1)), device='cuda')
    flux = rng.integers(1, 100, (1, 1, npol)).astype(float)
    vis = torch.zeros((n, npol), dtype=arl.device.CDTYPE[precision], device='cuda')
    arl.skycomponents.dft_predict(uvw, None, torch.zeros((1, 3), dtype=torch.float64, device='cuda'),
                                  torch.as_tensor(flux, device='cuda'), vis, precision)
    assert numpy.array_equal(vis.cpu().numpy(), numpy.broadcast_to(flux[0, 0], (n, npol)).astype(complex))


@pytest.mark.parametrize('precision', ['fp32c', 'fp64'])
def test_row_at_the_origin(arl, precision):
    """And components on one axis, rows on another: every product of the phase is zero."""
    rng = numpy.random.default_rng(2)
    uvw = torch.zeros((300, 3), dtype=torch.float64, device='cuda')
    uvw[100:, 1] = torch.as_tensor(rng.uniform(-1e4, 1e4, 200), device='cuda')
    lmn = torch.zeros((9, 3), dtype=torch.float64, device='cuda')
    lmn[:, 0] = torch.as_tensor(rng.uniform(-0.5, 0.5, 9), device='cuda')
    flux = torch.ones((9, 1, 1), dtype=torch.float64, device='cuda')
    vis = torch.zeros((300, 1), dtype=arl.device.CDTYPE[precision], device='cuda')
    arl.skycomponents.dft_predict(uvw, None, lmn, flux, vis, precision)
    assert numpy.array_equal(vis.cpu().numpy(), numpy.full((300, 1), 9.0 + 0j))
