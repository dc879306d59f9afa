"""Gradients of gradients through bfly's functions (a gradient penalty), by the C++ module and by the
autograd.Function classes, against torch's FP64 transforms.  Tolerance: rel L2 <= 1e-5, this
repository's bound for fp32 gradients."""
import pytest

pytestmark = pytest.mark.gpu


def _second(torch, f, x, weight, probe):
    """Gradient of <grad of a quartic of f, probe>: it has a term through f and one through f's gradient."""
    a = x.clone().requires_grad_(True)
    y = f(a)
    p = y.real.square() + (y.imag.square() if y.is_complex() else 0)
    loss = (p * p * weight).sum() / p.detach().mean()
    g = torch.autograd.grad(loss, a, create_graph=True)[0]
    dot = (g * probe.conj()).real.sum() if x.is_complex() else (g * probe).sum()
    return torch.autograd.grad(dot, a)[0]


def _cases(torch, ops, dev):
    T = torch.fft
    w, w4 = torch.hann_window(256, device=dev), torch.hann_window(400, device=dev)
    wd, wd4 = w.double(), w4.double()
    st = lambda n, win: lambda t: torch.stft(t, n, n // 4, window=win, return_complex=True)   # noqa: E731
    one = torch.ones(256, device=dev, dtype=torch.float64)
    return [
        ("fft", (3, 96), True, ops.fft, lambda t: ops._FFT.apply(t, -1, 1.0), T.fft),
        ("ifft axis", (2, 64, 5), True, lambda t: ops.ifft(t, dim=1), lambda t: ops._FFTAxis.apply(t, 1, 1, 1 / 64),
         lambda t: T.ifft(t, dim=1)),
        ("fft2", (2, 32, 48), True, ops.fft2, lambda t: ops._FFT2.apply(t, -1, 1.0), T.fft2),
        ("rfft", (3, 400), False, ops.rfft, lambda t: ops._RFFT.apply(t, 1.0), T.rfft),
        ("rfft ortho", (3, 256), False, lambda t: ops.rfft(t, "ortho"), lambda t: ops._RFFT.apply(t, 1 / 16),
         lambda t: T.rfft(t, norm="ortho")),
        ("irfft", (4, 129), True, ops.irfft, lambda t: ops._IRFFT.apply(t, 256, 1 / 256), T.irfft),
        ("rfft2", (2, 32, 64), False, ops.rfft2, lambda t: ops._RFFT2.apply(t, 1.0), T.rfft2),
        ("irfft2", (2, 32, 33), True, ops.irfft2, lambda t: ops._IRFFT2.apply(t, 64, 1 / 2048), T.irfft2),
        ("stft", (2, 3000), False, lambda t: ops.stft(t, 256, window=w),
         lambda t: ops._STFT.apply(t, 256, 64, True, w).transpose(1, 2), st(256, wd)),
        ("stft no window", (2, 3000), False, lambda t: ops.stft(t, 256),
         lambda t: ops._STFT.apply(t, 256, 64, True, None).transpose(1, 2), st(256, one)),
        ("stft 400", (2, 3000), False, lambda t: ops.stft(t, 400, window=w4),
         lambda t: ops._STFT.apply(t, 400, 100, True, w4).transpose(1, 2), st(400, wd4)),
        ("istft", (2, 129, 20), True, lambda t: ops.istft(t, 256, window=w),
         lambda t: ops._ISTFT.apply(t.transpose(1, 2).contiguous(), 256, 64, True, w, 19 * 64, 1.0),
         lambda t: torch.istft(t, 256, window=wd)),
        ("istft 400", (2, 201, 20), True, lambda t: ops.istft(t, 400, window=w4),
         lambda t: ops._ISTFT.apply(t.transpose(1, 2).contiguous(), 400, 100, True, w4, 19 * 100, 1.0),
         lambda t: torch.istft(t, 400, window=wd4)),
    ]


def test_gradient_of_the_gradient(cuda):
    import torch
    from bfly import ops
    gen = torch.Generator(device=cuda).manual_seed(3)
    for name, shape, cplx, native, function, ref in _cases(torch, ops, cuda):
        dt = torch.complex64 if cplx else torch.float32
        x, probe = (torch.randn(*shape, dtype=dt, device=cuda, generator=gen) for _ in range(2))
        with torch.no_grad():
            out = native(x)
        weight = torch.rand(out.shape, device=cuda, generator=gen)
        wide = torch.complex128 if cplx else torch.float64
        want = _second(torch, ref, x.to(wide), weight.double(), probe.to(wide))
        for route, f in (("module", native), ("functions", function)):
            got = _second(torch, f, x, weight, probe)
            rel = ((got - want).norm() / want.norm()).item()
            assert rel <= 1e-5, (name, route, rel)


def test_first_gradient_has_no_graph_unless_asked(cuda):
    import torch
    import bfly
    x = torch.randn(2, 64, device=cuda, requires_grad=True)
    y = bfly.rfft(x)
    g = torch.autograd.grad(y, x, torch.ones_like(y))[0]
    assert not g.requires_grad
