"""Gain chi^2 on either side of the row counts where a thread takes more rows (65,536 and
155,648), pairs of rows in one access and not, one polarisation and several."""
import numpy
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def need_cuda(arl):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    arl._native.load()


@pytest.mark.parametrize('n', [65535, 65539, 155648, 155655])
@pytest.mark.parametrize('npol,offset,nfreq', [(1, 0, 8), (1, 1, 1), (2, 0, 3)])
@pytest.mark.parametrize('dtype', [torch.complex64, torch.complex128])
def test_gain_chi2_at_the_row_counts(arl, n, npol, offset, nfreq, dtype):
    """Against PyTorch in 64 bits: FP64 sums of n terms in another order, so relative to
    the absolute sums within n 2^-52; the model gradient is rounded once to its type."""
    dev = torch.device('cuda')
    gen = torch.Generator(dev).manual_seed(n)
    nant = 20
    i, j = numpy.triu_indices(nant, 1)
    pick = numpy.arange(n) // nfreq % i.size

    def put(t):
        out = torch.empty(t.numel() + offset, dtype=t.dtype, device=dev)
        out[offset:] = t.reshape(-1)
        return out[offset:].reshape(t.shape)
    a1, a2 = (put(torch.as_tensor(a[pick].astype('i4'), device=dev)) for a in (i, j))
    rnd = lambda *s: torch.view_as_complex(torch.randn(s + (2,), dtype=torch.float64, device=dev, generator=gen))  # noqa: E731
    g, v, m = rnd(nant), put(rnd(n, npol).to(dtype)), put(rnd(n, npol).to(dtype))
    w = put(torch.rand((n, npol), dtype=torch.float64, device=dev, generator=gen) + 0.1)
    M, G = m.clone().requires_grad_(True) if offset == 0 else m.requires_grad_(True), g.requires_grad_(True)
    c = arl.autograd.GainChi2.apply(M, G, v, a1, a2, w)
    c.backward()
    with torch.no_grad():
        g1, g2 = g[a1.long()][:, None], g[a2.long()][:, None]
        mm, r = m.to(torch.complex128), v.to(torch.complex128) - g2 * g1.conj() * m.to(torch.complex128)
        want = (w * r.abs() ** 2).sum()
        assert abs(c - want) <= n * 2.0 ** -52 * want
        gm = -2 * w * g2.conj() * g1 * r
        eps = 2.0 ** -23 if dtype == torch.complex64 else 2.0 ** -48
        assert bool(((M.grad.to(torch.complex128) - gm).abs() <= eps * (gm.abs() + 1e-3 * gm.abs().max())).all())
        wg, scale = torch.zeros_like(g), torch.zeros(nant, dtype=torch.float64, device=dev)
        for a, d in ((a2, (-2 * w * r * g1 * mm.conj()).sum(1)), (a1, (-2 * w * r.conj() * g2 * mm).sum(1))):
            wg.index_add_(0, a.long(), d)
            scale.index_add_(0, a.long(), d.abs())
        assert bool(((G.grad - wg).abs() <= n * 2.0 ** -52 * scale).all())
