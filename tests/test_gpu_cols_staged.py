"""Column FFTs of 2048 and 4096 points around the rule that hands them to the persistent kernel: one
strip fewer and more than the GPU has SMs, a partial last strip, one strip per SM and a remainder,
rows off the 16-byte boundary, in place.  Tolerance: the column bound of this repository, rel L2 <=
1e-6 per column against FP64."""
import numpy as np
import pytest

import oracle.fft_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,outer,inner", [(2048, 148, 8), (2048, 149, 8), (2048, 20, 134), (2048, 21, 131),
                                           (4096, 37, 16), (4096, 75, 6), (4096, 149, 2)])
@pytest.mark.parametrize("direction", [-1, 1])
@pytest.mark.parametrize("shift", [0, 1])
def test_columns_match_fp64(plan, cuda, n, outer, inner, direction, shift):
    import torch
    g = torch.Generator(device=cuda).manual_seed(n + outer)
    flat = torch.randn(outer * n * inner + shift, dtype=torch.complex64, device=cuda, generator=g)
    x = flat[shift:].view(outer, n, inner)
    y = torch.full_like(x, float("nan"))
    scale = 1.0 if direction < 0 else 1.0 / n
    assert plan.exec_c2c_axis(x.data_ptr(), y.data_ptr(), n, outer, inner, direction, scale, 0) == 0
    xd = x.to(torch.complex128)
    assert plan.exec_c2c_axis(x.data_ptr(), x.data_ptr(), n, outer, inner, direction, scale, 0) == 0   # in place
    torch.cuda.synchronize()
    assert torch.equal(x, y)
    rows = O.sample_batches(outer, 3)
    xs = xd[rows].cpu().numpy()
    ref = np.fft.fft(xs, axis=1) if direction < 0 else np.fft.ifft(xs, axis=1)
    got = np.moveaxis(y[rows].cpu().numpy(), 1, -1).reshape(-1, n)
    assert O.rel_l2_rows(got, np.moveaxis(ref, 1, -1).reshape(-1, n)) <= 1e-6
