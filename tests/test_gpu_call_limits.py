"""What bfly's functions accept and refuse at the limits of their arguments: the same through the C++
module as through the autograd.Function classes."""
import pytest

pytestmark = pytest.mark.gpu


def test_empty_lengths(cuda):
    import torch
    import bfly
    empty = torch.empty(2, 0, dtype=torch.complex64, device=cuda)
    for bad in (lambda: bfly.ifft(empty), lambda: bfly.fft(empty, norm="ortho"), lambda: bfly.fft(empty, norm="forward"),
                lambda: bfly.ifft2(empty[None]), lambda: bfly.fft2(empty[None], norm="forward"),
                lambda: bfly.rfft(empty.real, norm="ortho"), lambda: bfly.rfft2(empty.real[None], norm="ortho"),
                lambda: bfly.irfft2(torch.empty(0, 33, dtype=torch.complex64, device=cuda))):
        with pytest.raises(ZeroDivisionError):
            bad()
    assert bfly.fft(empty).shape == (2, 0) and bfly.fft2(empty[None]).shape == (1, 2, 0)
    x = torch.empty(0, 64, dtype=torch.complex64, device=cuda)
    assert bfly.fft(x).shape == bfly.ifft(x).shape == (0, 64)
    assert bfly.irfft(x[:, :33], 64).shape == (0, 64) and bfly.rfft(x.real).shape == (0, 33)


def test_norms(cuda):
    import torch
    import bfly
    x = torch.randn(2, 64, dtype=torch.complex64, device=cuda)
    for norm in (None, "", False, 0, ()):   # all of them read as "backward"
        assert torch.equal(bfly.ifft(x, norm), bfly.ifft(x, "backward"))
    for norm in ("no", 1, ["ortho"], b"ortho"):
        with pytest.raises(ValueError):
            bfly.fft(x, norm)
