"""DFT predict, FP32C, on either side of the channel counts up to which a block stages
the components' fluxes (128 with one row a thread, 256 with two).  Per term the phase,
sine / cosine, flux and product roundings stay below 6 units of 2^-24 of the flux, and
the sum of ncomp terms adds at most one unit of the flux sum each."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


@pytest.mark.parametrize('n,nchan', [(700, 128), (700, 129), (155649, 256), (155649, 257)])
@pytest.mark.parametrize('npol', [1, 2, 4])
def test_dft_flux_staging(arl, n, nchan, npol):
    rng = numpy.random.default_rng(n + npol)
    ncomp = 13
    put = lambda a: torch.as_tensor(numpy.ascontiguousarray(a), device='cuda')  # noqa: E731
    uvw = rng.uniform(-1e3, 1e3, (n, 3))
    l, m = rng.uniform(-0.6, 0.6, (2, ncomp))
    lmn = numpy.stack([l, m, numpy.sqrt(1 - l * l - m * m) - 1], 1)
    flux = rng.uniform(0.1, 3.0, (ncomp, nchan, npol))
    chan = rng.integers(0, nchan, n).astype(numpy.int32)
    vis = torch.zeros((n, npol), dtype=torch.complex64, device='cuda')
    arl.skycomponents.dft_predict(put(uvw), put(chan), put(lmn), put(flux), vis, 'fp32c')
    want = numpy.einsum('nk,knp->np', numpy.exp(-2j * numpy.pi * (uvw @ lmn.T)), flux[:, chan])
    bound = (6 + ncomp) * 2.0 ** -24 * flux[:, chan].sum(0)
    assert numpy.all(numpy.abs(vis.cpu().numpy() - want) <= bound)
