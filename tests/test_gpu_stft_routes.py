"""Short-time transforms of 1024 and 2048 on both sides of the rule that chooses 16 or 32 values a thread:
the last frame count of one and the first of the other, hops that divide by 4, by 2 and odd ones,
against torch's FP64 transforms.  Tolerances are this repository's for these entries: rel L2 <= 1e-6 per
frame forward, 2e-6 inverse, 1e-5 for gradients."""
import pytest

pytestmark = pytest.mark.gpu


def _rel(torch, a, b, dim=None):
    d, n = (a - b).abs().square(), b.abs().square()
    return (d.sum(dim) / n.sum(dim)).sqrt().max().item()


# (n, hop, frames of one signal, signals): the frames in all lie at a side of 640, 2048, 4096, 8192 or 16384
CASES = [(1024, 256, 2047, 1), (1024, 256, 2048, 1), (1024, 258, 2048, 1), (1024, 129, 4100, 1), (2048, 512, 639, 1),
         (2048, 512, 640, 1), (1024, 256, 819, 5), (1024, 256, 1024, 4), (1024, 1024, 2047, 4), (1024, 1024, 2048, 4),
         (1024, 1024, 4096, 4), (1024, 258, 2047, 4), (1024, 258, 2048, 4), (1024, 129, 4095, 4), (1024, 129, 4096, 4),
         (2048, 512, 4095, 4), (2048, 512, 4096, 4), (2048, 1024, 4096, 4), (2048, 256, 2047, 4), (2048, 256, 2048, 4),
         (2048, 514, 4096, 4)]


@pytest.mark.parametrize("n,hop,frames,signals", CASES)
def test_against_fp64(cuda, n, hop, frames, signals):
    import torch
    import bfly
    g = torch.Generator(device=cuda).manual_seed(hop)
    length = hop * (frames - 1)
    w = torch.hann_window(n, device=cuda) + 0.1   # no zero envelope at hop n
    x = torch.randn(signals, length, device=cuda, generator=g).requires_grad_(True)
    xd = x.detach().double().requires_grad_(True)
    y = bfly.stft(x, n, hop_length=hop, window=w)
    ref = torch.stft(xd, n, hop_length=hop, window=w.double(), return_complex=True)
    assert y.shape == ref.shape == (signals, n // 2 + 1, frames)
    assert _rel(torch, y.detach(), ref.detach(), 1) <= 1e-6
    gy = torch.randn(y.shape, dtype=torch.complex64, device=cuda, generator=g)
    got = torch.autograd.grad(y, x, gy)[0]
    want = torch.autograd.grad(ref, xd, gy.to(torch.complex128))[0]
    assert _rel(torch, got, want) <= 1e-5
    del y, ref, got, want
    X = gy.requires_grad_(True)
    Xd = X.detach().to(torch.complex128).requires_grad_(True)
    z = bfly.istft(X, n, hop_length=hop, window=w)
    zr = torch.istft(Xd, n, hop_length=hop, window=w.double())
    assert z.shape == zr.shape and _rel(torch, z.detach(), zr.detach(), 1) <= 2e-6
    gz = torch.randn(z.shape, device=cuda, generator=g)
    got = torch.autograd.grad(z, X, gz)[0]
    want = torch.autograd.grad(zr, Xd, gz.double())[0]
    assert _rel(torch, got, want) <= 1e-5


@pytest.mark.parametrize("n", [1024, 2048])
def test_capture_on_the_other_side(ctx, cuda, n):
    """A call with few frames is all the warm-up that a captured one with many needs, on every kernel."""
    import torch
    plan = ctx.make_plan()
    hop, few, many = n // 4, 40, 20000
    w = torch.hann_window(n, device=cuda)
    x = torch.randn(1, hop * (many - 1), device=cuda)
    spec = torch.empty(1, many, n // 2 + 1, dtype=torch.complex64, device=cuda)
    y, gx, gs = torch.empty_like(x), torch.empty_like(x), torch.empty_like(spec)

    def run(frames, s):
        length = hop * (frames - 1)
        assert plan.exec_stft(x.data_ptr(), spec.data_ptr(), n, 1, length, hop, True, w.data_ptr(), s)[0] == 0
        assert plan.exec_istft(spec.data_ptr(), y.data_ptr(), n, 1, frames, hop, True, w.data_ptr(), length, 1.0, s) == 0
        assert plan.exec_stft_backward(spec.data_ptr(), gx.data_ptr(), n, 1, length, hop, True, w.data_ptr(), s) == 0
        assert plan.exec_istft_backward(x.data_ptr(), gs.data_ptr(), n, 1, frames, hop, True, w.data_ptr(), length, 1.0,
                                        s) == 0

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        run(few, stream.cuda_stream)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            run(many, stream.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert ((y - x).norm() / x.norm()).item() <= 2e-6
