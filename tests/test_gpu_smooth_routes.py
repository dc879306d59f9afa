"""C2C of n = A*2^k on both sides of the rule that divides these lengths between the prime-factor and
the mixed-radix kernels, one row, a partial CTA and many CTAs.  Tolerance: rel L2 <= 1e-6 per row
against FP64, this repository's bound for them."""
import numpy as np
import pytest

import oracle.fft_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [48, 80, 96, 144, 160, 192, 240, 288, 320, 384, 480, 576, 960, 1920, 3840])
@pytest.mark.parametrize("batch", [1, 7, 1501])
@pytest.mark.parametrize("direction", [-1, 1])
def test_rows_match_fp64(plan, cuda, n, batch, direction):
    import torch
    x = torch.from_numpy(O.normal_input(n, batch, n + batch)).to(cuda).view(torch.complex64)
    y = torch.empty_like(x)
    scale = 1.0 if direction < 0 else 1.0 / n
    assert plan.exec_c2c(x.data_ptr(), y.data_ptr(), n, batch, direction, scale, 0) == 0
    torch.cuda.synchronize()
    rows = O.sample_batches(batch, 40)
    xd = x[rows].cpu().numpy().astype(np.complex128)
    ref = np.fft.fft(xd, axis=-1) if direction < 0 else np.fft.ifft(xd, axis=-1)
    assert O.rel_l2_rows(y[rows].cpu().numpy(), ref) <= 1e-6
