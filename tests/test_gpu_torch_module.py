"""The C++ torch module behind bfly's functions against the autograd.Function classes it stands in
for: the same kernels, so equal bits, values and gradients; and what it has to leave to them."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _cases(torch, ops, dev):
    g = torch.Generator(device=dev).manual_seed(5)
    c = lambda *s: torch.randn(*s, dtype=torch.complex64, device=dev, generator=g)   # noqa: E731
    r = lambda *s: torch.randn(*s, device=dev, generator=g)                          # noqa: E731
    w = torch.hann_window(256, device=dev)
    spec = torch.stft(r(2, 4000), 256, window=w, return_complex=True)
    return [
        ("fft", c(3, 96), lambda x: ops.fft(x), lambda x: ops._FFT.apply(x, -1, 1.0)),
        ("fft rows strided", c(5, 64, 6).transpose(1, 2), lambda x: ops.fft(x), lambda x: ops._FFT.apply(x, -1, 1.0)),
        ("ifft axis", c(2, 64, 5), lambda x: ops.ifft(x, dim=1), lambda x: ops._FFTAxis.apply(x, 1, 1, 1.0 / 64)),
        ("fft axis ortho", c(64, 7), lambda x: ops.fft(x, "ortho", 0), lambda x: ops._FFTAxis.apply(x, 0, -1, 0.125)),
        ("fft2", c(2, 32, 48), lambda x: ops.fft2(x), lambda x: ops._FFT2.apply(x, -1, 1.0)),
        ("ifft2", c(32, 64), lambda x: ops.ifft2(x), lambda x: ops._FFT2.apply(x, 1, 1.0 / 2048)),
        ("rfft", r(2, 3, 400), lambda x: ops.rfft(x), lambda x: ops._RFFT.apply(x, 1.0)),
        ("irfft", c(4, 129), lambda x: ops.irfft(x), lambda x: ops._IRFFT.apply(x, 256, 1.0 / 256)),
        ("rfft2", r(2, 32, 64), lambda x: ops.rfft2(x), lambda x: ops._RFFT2.apply(x, 1.0)),
        ("irfft2", c(2, 32, 33), lambda x: ops.irfft2(x), lambda x: ops._IRFFT2.apply(x, 64, 1.0 / 2048)),
        ("stft", r(2, 4000), lambda x: ops.stft(x, 256, window=w),
         lambda x: ops._STFT.apply(x.contiguous(), 256, 64, True, w).transpose(-1, -2)),
        ("istft", spec, lambda x: ops.istft(x, 256, window=w, length=4000),
         lambda x: ops._ISTFT.apply(x.transpose(-1, -2).contiguous(), 256, 64, True, w, 4000, 1.0)),
    ]


def test_values_and_gradients_equal_the_functions(cuda):
    import torch
    from bfly import ops
    for name, x, native, function in _cases(torch, ops, cuda):
        with torch.no_grad():
            plain = native(x)
        a, b = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
        ya, yb = native(a), function(b)
        assert ya.grad_fn is not None and torch.equal(ya, yb) and torch.equal(plain, yb), name
        g = torch.randn_like(yb)
        ga, gb = torch.autograd.grad(ya, a, g)[0], torch.autograd.grad(yb, b, g)[0]
        assert torch.equal(ga, gb), name
        # a gradient that is neither contiguous nor, for complex results, held unconjugated
        ya = native(a)
        gs = torch.randn(*ya.shape, 2, device=cuda).to(ya.dtype)[..., 0]
        gs = gs.conj() if ya.is_complex() else gs
        ga = torch.autograd.grad(ya, a, gs)[0]
        gb = torch.autograd.grad(function(b), b, gs.resolve_conj().contiguous())[0]
        assert torch.equal(ga, gb), name


def test_a_conjugate_view_is_transformed_as_its_values(cuda):
    import torch
    import bfly
    x = torch.randn(3, 64, dtype=torch.complex64, device=cuda)
    assert torch.equal(bfly.fft(x.conj()), bfly.fft(x.conj().resolve_conj()))


def test_refusals_and_errors_stay(cuda):
    import torch
    import bfly
    from bfly import BflyError, ops
    x = torch.randn(2, 64, dtype=torch.complex64, device=cuda)
    for bad in (lambda: bfly.fft(x.cpu()), lambda: bfly.fft(x, norm="no"), lambda: bfly.irfft(x, 64)):
        with pytest.raises(ValueError):
            bad()
    for bad in (lambda: bfly.fft(x.to(torch.complex128)), lambda: bfly.rfft(x)):
        with pytest.raises(TypeError):
            bad()
    with pytest.raises(BflyError) as e:
        bfly.fft(torch.randn(1, 131072, dtype=torch.complex64, device=cuda))
    assert e.value.code == -8
    assert bfly.fft(x[:0]).shape == (0, 64)
    with pytest.raises(RuntimeError):      # no vmap rule, as the Function says
        torch.func.vmap(bfly.fft)(x)
    with torch.autograd.forward_ad.dual_level(), pytest.raises(RuntimeError):   # no jvp
        bfly.fft(torch.autograd.forward_ad.make_dual(x, x))
    assert ops._native.fft(x.cpu(), -1, -1, 0) is None


def test_saved_tensor_hooks_see_the_window(cuda):
    import torch
    import bfly
    w = torch.hann_window(256, device=cuda)
    x = torch.randn(2, 4000, device=cuda, requires_grad=True)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t, lambda t: t):
        y = bfly.stft(x, 256, window=w)
    assert any(torch.equal(t, w) for t in packed)
    assert torch.autograd.grad(y, x, torch.ones_like(y))[0].shape == x.shape


def test_threads_and_streams(cuda):
    """Two threads on streams of their own, plans looked up and forgotten meanwhile."""
    import torch
    import bfly
    from bfly import ops
    x = torch.randn(64, 512, dtype=torch.complex64, device=cuda)
    want = bfly.fft(x)
    bfly.ifft(x)
    torch.cuda.synchronize()
    bad = []

    def work():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for i in range(200):
                y = bfly.fft(x)
                if i % 50 == 0:
                    ops._native.forget_plans()
            if not torch.equal(y, want):
                bad.append(1)
        s.synchronize()

    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
