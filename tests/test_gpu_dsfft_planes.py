"""The FP32C inverse transform of w-planes whose sum cancels in its high part: what is
left in the low part is the whole signal, also in a tile that is otherwise empty."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


@pytest.mark.parametrize('ny,nx', [(64, 64), (64, 4096), (64, 8192), (512, 256)])
def test_planes_that_cancel(arl, ny, nx):
    """One cell holds 1, small and -1 in three planes.  A double-single sum is exact here
    and every later value a product with a twiddle: 24 roundings of 2^-24 at most."""
    small = float(numpy.float32(1e-9))
    grid = torch.zeros((1, 1, 3, ny, nx), dtype=torch.complex64, device='cuda')
    y, x = ny // 2 + 5, nx // 2 - 3
    grid[0, 0, :, y, x] = torch.tensor([1.0, small, -1.0], dtype=torch.complex64, device='cuda')
    im = arl.create_image(npixel=64, cellsize=1e-3, frequency=numpy.array([1e8]),
                          channel_bandwidth=numpy.array([1e7]), phasecentre=arl.PhaseCentre(0.0, -45.0))
    wcs = arl.create_griddata_from_image(im, nw=3).grid_wcs
    gd = arl.device.grid_desc(wcs, grid.shape)
    gcf = torch.ones((1, 1, ny, nx), dtype=torch.float64, device='cuda')
    re, imag = arl.device.fft_grid_to_image(grid, gd, gcf, 'fp32c', imaginary=True)
    ph = 2 * numpy.pi * ((5 * (numpy.arange(ny) - ny // 2) % ny)[:, None] / ny -
                         (3 * (numpy.arange(nx) - nx // 2) % nx)[None, :] / nx)
    got = re[0, 0].cpu().numpy() + 1j * imag[0, 0].cpu().numpy()
    assert numpy.max(numpy.abs(got - small * numpy.exp(1j * ph))) <= 24 * 2.0 ** -24 * small
