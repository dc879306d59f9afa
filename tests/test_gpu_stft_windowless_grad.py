"""Gradients through bfly.stft and bfly.istft where no window is given (the default), on every route a
length takes, against torch's FP64 short-time transforms.  Tolerance: rel L2 <= 1e-5, this
repository's bound for fp32 gradients."""
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a - b).norm() / b.norm()).item()


@pytest.mark.parametrize("n", [64, 256, 2048, 8192, 400])
@pytest.mark.parametrize("center", [True, False])
@pytest.mark.parametrize("lead", [(), (2,), (2, 3)])
def test_stft(cuda, n, center, lead):
    import torch
    import bfly
    g = torch.Generator(device=cuda).manual_seed(n)
    x = torch.randn(*lead, 6 * n + 3, device=cuda, generator=g).requires_grad_(True)
    xd = x.detach().double().requires_grad_(True)
    flat = xd.reshape(-1, xd.shape[-1])
    want = torch.stft(flat, n, center=center, return_complex=True, hop_length=n // 4, window=torch.ones(n, device=cuda).double())
    got = bfly.stft(x, n, center=center)
    gy = torch.randn(got.shape, dtype=torch.complex64, device=cuda, generator=g)
    a = torch.autograd.grad(got, x, gy)[0]
    b = torch.autograd.grad(want, xd, gy.to(torch.complex128).reshape(want.shape))[0]
    assert a.shape == x.shape and _rel(a, b) <= 1e-5


@pytest.mark.parametrize("n", [64, 256, 2048, 8192, 400])
@pytest.mark.parametrize("center", [True, False])
def test_istft(cuda, n, center):
    import torch
    import bfly
    g = torch.Generator(device=cuda).manual_seed(n)
    X = torch.randn(2, n // 2 + 1, 9, dtype=torch.complex64, device=cuda, generator=g).requires_grad_(True)
    Xd = X.detach().to(torch.complex128).requires_grad_(True)
    got = bfly.istft(X, n, center=center)
    want = torch.istft(Xd, n, center=center, window=torch.ones(n, device=cuda).double())
    gy = torch.randn(got.shape, device=cuda, generator=g)
    a = torch.autograd.grad(got, X, gy)[0]
    b = torch.autograd.grad(want, Xd, gy.double())[0]
    assert _rel(a, b) <= 1e-5
