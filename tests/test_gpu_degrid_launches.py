"""A degrid call runs one degridding kernel, whichever variant is chosen and
whether or not it applies, so that a variant's parity test tests that variant."""
import ctypes

import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


@pytest.mark.parametrize('subgrid', [48, 64])  # the TMA kernel takes 48 alone
@pytest.mark.parametrize('degrid_kernel', [2, 3, 4])
def test_one_degrid_kernel_a_call(arl, degrid_kernel, subgrid):
    before = arl.tune.get_tuning()
    nat, dv, dev = arl._native, arl.device, torch.device('cuda')
    try:
        arl.tune.set_tuning(degrid_kernel=degrid_kernel, subgrid=subgrid)
        im = arl.create_image(npixel=128, cellsize=2e-3, frequency=numpy.array([1e8]),
                              channel_bandwidth=numpy.array([1e7]), phasecentre=arl.PhaseCentre(0.0, -45.0))
        _, cf = arl.create_pswf_convolutionfunction(im, oversampling=8, support=8)
        cf_t, cs, ps, psup = dv.device_cf(cf, 'fp32c', dev)
        cd = dv.cf_desc(cf.grid_wcs, cf.data.shape, cs, ps, psup, table=cf_t)
        gdh = arl.create_griddata_from_image(im)
        gd = dv.grid_desc(gdh.grid_wcs, gdh.data.shape)
        n = 4000
        rng = numpy.random.default_rng(1)
        uvw = torch.as_tensor(rng.uniform(-0.35, 0.35, (n, 3)) / 2e-3, device=dev)
        f = torch.full((n,), 1e8, dtype=torch.float64, device=dev)
        g = torch.ones(gdh.data.shape, dtype=torch.complex64, device=dev)
        ws = torch.empty(dv.plan_bytes(n, gd, cd), dtype=torch.uint8, device=dev)
        out = torch.empty((n, 1), dtype=torch.complex64, device=dev)
        nat.call('arlgpu_plan_build', nat.ptr(uvw), nat.ptr(f), n, ctypes.byref(gd), ctypes.byref(cd), nat.ptr(ws),
                 ws.numel(), None, nat.stream_ptr())
        launches = nat.load().arlgpu_kernel_launches()
        nat.call('arlgpu_degrid_planned', n, nat.PRECISIONS['fp32c'], nat.ptr(cf_t), ctypes.byref(cd), nat.ptr(g),
                 ctypes.byref(gd), nat.ptr(out), nat.ptr(ws), ws.numel(), nat.stream_ptr())
        assert nat.load().arlgpu_kernel_launches() - launches == 1
        torch.cuda.synchronize()
    finally:
        arl.tune.set_tuning(**before)
