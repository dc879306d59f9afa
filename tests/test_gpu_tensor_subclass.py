"""Tensor subclasses go to the autograd.Function classes: the result keeps the type that the torch
operations inside give it, and __torch_function__ sees those operations.  Parameters are plain."""
import pytest

pytestmark = pytest.mark.gpu


def test_type_and_torch_function(cuda):
    import torch
    import bfly
    from bfly import ops

    class Tagged(torch.Tensor):
        seen = 0

        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            Tagged.seen += 1
            return super().__torch_function__(func, types, args, kwargs or {})

    x = torch.randn(4, 64, 64, dtype=torch.complex64, device=cuda)
    for f in (bfly.fft, bfly.ifft, bfly.fft2, bfly.ifft2, lambda t: bfly.fft(t, dim=1)):
        before = Tagged.seen
        y = f(x.as_subclass(Tagged))
        assert type(y) is Tagged and Tagged.seen > before
        assert torch.equal(y.as_subclass(torch.Tensor), f(x))
    r, w = torch.randn(2, 4000, device=cuda), torch.hann_window(256, device=cuda)
    spec = bfly.stft(r, 256, window=w)
    for f, t in ((bfly.rfft, r[:, :64]), (bfly.irfft, x[..., :33]), (bfly.rfft2, r[:, :2048].reshape(2, 32, 64)),
                 (bfly.irfft2, x[..., :33]), (lambda t: bfly.stft(t, 256, window=w), r),
                 (lambda t: bfly.stft(r, 256, window=t), w), (lambda t: bfly.istft(t, 256, window=w), spec),
                 (lambda t: bfly.istft(spec, 256, window=t), w)):
        before = Tagged.seen
        y = f(t.as_subclass(Tagged))
        assert Tagged.seen > before and torch.equal(y.as_subclass(torch.Tensor), f(t))


def test_parameters_are_plain(cuda):
    import torch
    import bfly
    p = torch.nn.Parameter(torch.randn(4, 64, dtype=torch.complex64, device=cuda))
    y = bfly.fft(p)
    assert type(y) is torch.Tensor and "C2CNode" in type(y.grad_fn).__name__ + y.grad_fn.name()
