"""irfft2 between streams and in graphs: the array between its two passes belongs to the call, so calls
on other streams and later, larger calls leave it alone."""
import pytest

pytestmark = pytest.mark.gpu


def _routes(ops):
    return (ops.irfft2, lambda X: ops._IRFFT2.apply(X, 2 * (X.shape[-1] - 1), 1.0 / (X.shape[-2] * 2 * (X.shape[-1] - 1))))


def test_two_streams(cuda):
    import torch
    from bfly import ops
    x = [torch.randn(16, 256, 256, device=cuda) for _ in range(2)]
    X = [torch.fft.rfft2(t) for t in x]
    for f in _routes(ops):
        want = [f(t) for t in X]
        torch.cuda.synchronize()
        streams, got = [torch.cuda.Stream() for _ in range(2)], [[], []]
        for _ in range(30):
            for k in range(2):
                with torch.cuda.stream(streams[k]):
                    got[k].append(f(X[k]))
        torch.cuda.synchronize()
        for k in range(2):
            assert all(torch.equal(y, want[k]) for y in got[k])
            assert (torch.linalg.vector_norm(want[k] - x[k]) / torch.linalg.vector_norm(x[k])).item() <= 2e-6


def test_graph_outlives_a_larger_call(cuda):
    import torch
    from bfly import ops
    small, large = (torch.fft.rfft2(torch.randn(b, 64, 128, device=cuda)) for b in (2, 64))
    for f in _routes(ops):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            want = f(small)
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                y = f(small)
        f(large)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)


def test_refusals_stay(cuda):
    import torch
    import bfly
    for shape in ((3, 48, 33), (2, 64, 18), (8192, 33), (16, 33)):   # no such columns, or rows of 34
        with pytest.raises(bfly.BflyError) as e:
            bfly.irfft2(torch.randn(*shape, dtype=torch.complex64, device=cuda))
        assert e.value.code == -8
