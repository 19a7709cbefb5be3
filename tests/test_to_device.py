"""Host arrays on their way to the device: the copy is done with the host's memory
when ``to_device`` returns, because the memory may be a temporary or be written by
the caller next."""
import numpy
import pytest
import torch


@pytest.fixture
def moves(monkeypatch):
    """Records of every ``Tensor.to`` that names a device: (device, non_blocking,
    whether the source is pinned).  The data stay where they are."""
    seen = []
    to = torch.Tensor.to

    def spy(self, *args, **kwargs):
        device = next((a for a in args if isinstance(a, torch.device)), kwargs.get('device'))
        if device is None:
            return to(self, *args, **kwargs)
        seen.append((device, bool(kwargs.get('non_blocking', False)), type(self).__name__ == 'Pinned'))
        dtype = next((a for a in args if isinstance(a, torch.dtype)), kwargs.get('dtype'))
        return to(self, dtype or self.dtype)
    monkeypatch.setattr(torch.Tensor, 'to', spy)
    return seen


@pytest.mark.parametrize('shape,strided', [((5,), False), ((6, 3), True), ((0, 3), False), ((), False)])
def test_pageable_copies_block(arl, moves, shape, strided):
    a = numpy.arange(2.0 * max(1, int(numpy.prod(shape)))).reshape(-1)[:2 * int(numpy.prod(shape))]
    a = a.reshape(shape + (2,))[..., 0] if strided else a[::2].reshape(shape).copy()
    dev = torch.device('cuda', 0)
    out = arl.device.to_device(a, torch.float32, dev)
    assert out.dtype == torch.float32 and numpy.array_equal(out.numpy().reshape(a.shape), a.astype('f4'))
    assert [m for m in moves if m[0] == dev and m[1] and not m[2]] == []


@pytest.mark.gpu
@pytest.mark.parametrize('n', [7, 1 << 12, 1 << 20])
def test_array_may_change_after_the_call(arl, n):
    """Behind work that keeps the stream busy: the device tensor holds what the array
    held at the call."""
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    dev = torch.device('cuda', 0)
    x = torch.zeros(1 << 28, device=dev)
    a = numpy.arange(float(n))
    for _ in range(20):
        x.add_(1.0)
    t = arl.device.to_device(a, torch.float64, dev)
    a[:] = -1.0
    assert numpy.array_equal(t.cpu().numpy(), numpy.arange(float(n)))
