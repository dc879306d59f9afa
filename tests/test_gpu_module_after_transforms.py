"""The C++ module answers plain calls after a thread's first torch.func transform and after
torch.compile, and leaves the calls inside a transform to the autograd.Function classes."""
import pytest

pytestmark = pytest.mark.gpu


def _all_answered(torch, ops, dev):
    c = torch.randn(2, 64, 64, dtype=torch.complex64, device=dev)
    r = torch.randn(2, 64, 64, device=dev)
    n = ops._native
    half = c[..., :33].contiguous()
    frames = torch.randn(2, 9, 33, dtype=torch.complex64, device=dev)
    return all(y is not None for y in (
        n.fft(c, -1, -1, 0), n.fft(c, 1, 1, 0), n.fft2(c, -1, 0), n.rfft(r, 0), n.irfft(half, 64, 0), n.rfft2(r, 0),
        n.irfft2(half, 64, 0), n.stft(r[:, 0].repeat(1, 9), 64, 16, True, None),
        n.istft(frames, 64, 16, True, None, 128, 1.0)))


def test_answered_after_functorch_and_compile(cuda):
    import torch
    import bfly
    from bfly import ops
    assert _all_answered(torch, ops, cuda)
    torch.func.vmap(lambda t: t * 2)(torch.randn(3, 4, device=cuda))
    assert _all_answered(torch, ops, cuda)
    torch.func.grad(lambda t: (t * t).sum())(torch.randn(4, device=cuda))
    assert _all_answered(torch, ops, cuda)
    f = torch.compile(lambda t: bfly.fft(t * 2) + 1, backend="eager")
    x = torch.randn(3, 64, dtype=torch.complex64, device=cuda)
    assert torch.equal(f(x), bfly.fft(x * 2) + 1)
    assert _all_answered(torch, ops, cuda)


def test_left_alone_inside_a_transform(cuda):
    import torch
    import bfly
    from bfly import ops
    x = torch.randn(3, 64, dtype=torch.complex64, device=cuda)
    inside = []

    def body(t):
        inside.append(ops._native.fft(x, -1, -1, 0) is None)   # a plain tensor, but inside a level
        return t * 2

    torch.func.vmap(body)(torch.randn(3, 4, device=cuda))
    torch.func.grad(lambda t: body(t).sum())(torch.randn(4, device=cuda))
    assert inside == [True, True]
    with pytest.raises(RuntimeError):
        torch.func.vmap(bfly.fft)(x)
    with pytest.raises(RuntimeError):   # the Function has no setup_context
        torch.func.grad(lambda t: bfly.fft(t).abs().sum())(x)
