"""Host Visibility tables on the device: the unpacked records equal the columns
gathered on the host, for tables that take the records' way and those that cannot."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


def _table(arl, n, npol, form):
    rng = numpy.random.default_rng(n + npol)
    c = rng.normal(size=(n, npol)) + 1j * rng.normal(size=(n, npol))
    frame = {1: 'stokesI', 2: 'linearnp', 4: 'linear'}[npol]
    vis = arl.Visibility(uvw=rng.normal(size=(n, 3)) * 1e3, frequency=rng.uniform(1e8, 2e8, n), vis=c,
                         weight=numpy.ones((n, npol)), imaging_weight=rng.uniform(0, 2, (n, npol)),
                         polarisation_frame=arl.PolarisationFrame(frame))
    if form == 'narrow field':  # records that are not whole 64-bit words
        d = numpy.zeros(n, dtype=vis.data.dtype.descr + [('flag', 'i2')])
        for k in vis.data.dtype.names:
            d[k] = vis.data[k]
        vis.data = d
    elif form == 'every other row':
        vis.data = numpy.repeat(vis.data, 2)[::2]
    elif form == 'other byte order':
        vis.data = vis.data.astype(vis.data.dtype.newbyteorder('S'))
    elif form == 'read-only':
        vis.data.flags.writeable = False
    return vis


@pytest.mark.parametrize('precision', ['fp32c', 'fp64'])
@pytest.mark.parametrize('n,npol,form', [(1, 1, 'plain'), (777, 4, 'plain'), (300, 2, 'narrow field'),
                                         (300, 1, 'every other row'), (300, 1, 'read-only')])
def test_columns_equal_the_host_ones(arl, monkeypatch, n, npol, form, precision):
    vis = _table(arl, n, npol, form)
    monkeypatch.setattr(arl.device, '_UNPACK_ROWS', 256)  # several pieces, the last one short
    uvw, f, v, w = arl.device.host_rows(vis, precision, torch.device('cuda', 0))
    cdt, rdt = ('c8', 'f4') if precision == 'fp32c' else ('c16', 'f8')
    for got, want in ((uvw, vis.uvw), (f, vis.frequency), (v, vis.vis.astype(cdt)), (w, vis.imaging_weight.astype(rdt))):
        assert numpy.array_equal(got.cpu().numpy(), want)
    uvw, f, v, w = arl.device.host_rows(vis, precision, torch.device('cuda', 0), need_vis=False)
    assert numpy.array_equal(uvw.cpu().numpy(), vis.uvw) and v is None and w is None


def test_other_byte_order_stays_refused(arl):
    with pytest.raises(ValueError):
        arl.device.host_rows(_table(arl, 10, 1, 'other byte order'), 'fp32c', torch.device('cuda', 0))
