"""Short-time transforms that read what the kernel before them wrote into the same buffer, with no
synchronisation between them (an iterated phase reconstruction): a kernel may be launched while the
one before it drains, so it must not read the caller's arrays as constants.  The chain gives the same
bits as the same launches one at a time.

The scan runs without a GPU: read-only loads (__ldg) name tables alone, which are complete before any
kernel that reads them is launched."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ascend-fft_b200" / "csrc"
TABLES = {"tw", "twp", "twr", "wt", "wA", "chirp", "filt", "tlo", "thi", "tileMap", "dftTable"}


def test_read_only_loads_name_tables_alone():
    seen = set()
    for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        for m in re.finditer(r"__ldg\((?:reinterpret_cast<[^>]*>\()?\(?(\w+)", f.read_text()):
            assert m.group(1) in TABLES, f"{f.name}: __ldg of {m.group(1)}"
            seen.add(m.group(1))
    assert "twr" in seen


@pytest.mark.gpu
@pytest.mark.parametrize("n,hop", [(256, 64), (1024, 256), (4096, 512), (400, 100), (1200, 300)])
def test_iterated_reconstruction(plan, cuda, n, hop):
    import torch
    signals, frames = 8, 150
    length = hop * (frames - 1)
    g = torch.Generator(device=cuda).manual_seed(n)
    w = torch.hann_window(n, device=cuda)
    start = torch.randn(signals, length, device=cuda, generator=g)

    def chain(after):
        x = start.clone()
        spec = torch.empty(signals, frames, n // 2 + 1, dtype=torch.complex64, device=cuda)
        torch.cuda.synchronize()
        s = torch.cuda.current_stream().cuda_stream
        for _ in range(40):   # each step changes the signal: 0.97 of it comes back
            rc, got = plan.exec_stft(x.data_ptr(), spec.data_ptr(), n, signals, length, hop, True, w.data_ptr(), s)
            assert rc == 0 and got == frames
            after()
            assert plan.exec_istft(spec.data_ptr(), x.data_ptr(), n, signals, frames, hop, True, w.data_ptr(), length,
                                   0.97, s) == 0
            after()
        torch.cuda.synchronize()
        return x, spec

    for a, b in zip(chain(lambda: None), chain(torch.cuda.synchronize)):
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("n,hop", [(256, 64), (1024, 256)])
def test_gradient_chain(plan, cuda, n, hop):
    import torch
    signals, frames = 8, 150
    length = hop * (frames - 1)
    w = torch.hann_window(n, device=cuda)
    start = torch.randn(signals, length, device=cuda, generator=torch.Generator(device=cuda).manual_seed(n))

    def chain(after):
        x = start.clone()
        spec = torch.empty(signals, frames, n // 2 + 1, dtype=torch.complex64, device=cuda)
        torch.cuda.synchronize()
        s = torch.cuda.current_stream().cuda_stream
        for _ in range(20):   # the gradient of an inverse transform, and of a forward one, of each other's results
            assert plan.exec_istft_backward(x.data_ptr(), spec.data_ptr(), n, signals, frames, hop, True, w.data_ptr(),
                                            length, 1.0, s) == 0
            after()
            assert plan.exec_stft_backward(spec.data_ptr(), x.data_ptr(), n, signals, length, hop, True, w.data_ptr(),
                                           s) == 0
            after()
        torch.cuda.synchronize()
        return x, spec

    got, want = chain(lambda: None), chain(torch.cuda.synchronize)
    # the fold of the reflect padding adds by atomics, so the order of sums varies: the samples it
    # touches, and the frames that read them, to the rounding of a few sums through the chain
    for a, b in zip(got, want):
        assert (torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b)).item() <= 1e-5
