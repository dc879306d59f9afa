"""Conjugate and negative views (z.conj(), z.conj().imag) hold other values than their memory.  Every
function and its gradient transforms the values, through the C++ module and through the
autograd.Function classes that stand in for it: the bits of the call on the resolved tensor."""
import pytest

pytestmark = pytest.mark.gpu


def _inputs(torch, dev):
    g = torch.Generator(device=dev).manual_seed(11)
    c = lambda *s: torch.randn(*s, dtype=torch.complex64, device=dev, generator=g).conj()   # noqa: E731
    neg = lambda *s: c(*s).imag                                                             # noqa: E731
    return c, neg


def _calls(torch, ops, dev):
    c, neg = _inputs(torch, dev)
    w = torch.hann_window(256, device=dev)
    wneg = torch.complex(w, -w).conj().imag   # the same window as a negative view
    assert wneg.is_neg() and torch.equal(wneg, w)
    spec = torch.stft(torch.randn(2, 4000, device=dev), 256, window=w, return_complex=True).conj()
    return [
        ("fft", c(3, 96), [lambda x: ops.fft(x), lambda x: ops._FFT.apply(x, -1, 1.0)]),
        ("ifft axis", c(2, 64, 5), [lambda x: ops.ifft(x, dim=1), lambda x: ops._FFTAxis.apply(x, 1, 1, 1 / 64)]),
        ("fft2", c(2, 32, 48), [lambda x: ops.fft2(x), lambda x: ops._FFT2.apply(x, -1, 1.0)]),
        ("rfft", neg(3, 400), [lambda x: ops.rfft(x), lambda x: ops._RFFT.apply(x, 1.0)]),
        ("irfft", c(4, 129), [lambda x: ops.irfft(x), lambda x: ops._IRFFT.apply(x, 256, 1 / 256)]),
        ("rfft2", neg(2, 32, 64), [lambda x: ops.rfft2(x), lambda x: ops._RFFT2.apply(x, 1.0)]),
        ("irfft2", c(2, 32, 33), [lambda x: ops.irfft2(x), lambda x: ops._IRFFT2.apply(x, 64, 1 / 2048)]),
        ("stft", neg(2, 4000), [lambda x: ops.stft(x, 256, window=wneg), lambda x: ops.stft(x, 400)]),
        ("istft", spec, [lambda x: ops.istft(x, 256, window=wneg, length=4000)]),
        ("istft 400", c(2, 201, 20), [lambda x: ops.istft(x, 400)]),
        ("tensor cores", c(2, 256), [lambda x: ops.c2c_tensor(x)]),
    ]


def test_views_are_transformed_as_their_values(cuda):
    import torch
    from bfly import ops
    for name, x, routes in _calls(torch, ops, cuda):
        assert x.is_conj() or x.is_neg()
        for k, f in enumerate(routes):
            want = f(x.resolve_conj().resolve_neg().clone())
            assert torch.equal(f(x), want), (name, k)


def test_gradients_that_are_views(cuda):
    import torch
    from bfly import ops
    c, neg = _inputs(torch, cuda)
    for name, x, routes in _calls(torch, ops, cuda):
        if name == "tensor cores":
            continue
        for k, f in enumerate(routes):
            a = x.resolve_conj().resolve_neg().clone().requires_grad_(True)
            y = f(a)
            g = (c if y.is_complex() else neg)(*y.shape)
            assert g.is_conj() or g.is_neg()
            want = torch.autograd.grad(f(a), a, g.resolve_conj().resolve_neg())[0]
            assert torch.equal(torch.autograd.grad(y, a, g)[0], want), (name, k)


def test_function_classes_of_the_short_time_transforms(cuda):
    """_STFT and _ISTFT on views, as ops.stft and ops.istft hand them calls the module leaves."""
    import torch
    from bfly import ops
    c, neg = _inputs(torch, cuda)
    for n in (256, 400):
        x, X = neg(2, 4000), c(2, 9, n // 2 + 1)
        for f, v in ((lambda t: ops._STFT.apply(t, n, n // 4, True, None), x),
                     (lambda t: ops._ISTFT.apply(t, n, n // 4, True, None, 8 * (n // 4), 1.0), X)):
            r = v.resolve_conj().resolve_neg().clone()
            assert torch.equal(f(v), f(r)), n
            a = r.requires_grad_(True)
            y = f(a)
            g = (c if y.is_complex() else neg)(*y.shape)
            want = torch.autograd.grad(f(a), a, g.resolve_conj().resolve_neg())[0]
            assert torch.equal(torch.autograd.grad(y, a, g)[0], want), n
