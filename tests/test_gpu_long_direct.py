"""The one-pass long C2C kernels (n = 8192 and 16384 on one CTA per row, 32768 and 65536 on one
cluster per row): batches below, at and past the distance they load ahead, both directions, in
place, and the four-step schedule as a second opinion.

Tolerances: the long-C2C bounds of this repository, rel L2 <= 2e-6 per row against FP64 and <= 1e-6
against another fp32 schedule of the same transform."""
import numpy as np
import pytest

import oracle.fft_oracle as O

pytestmark = pytest.mark.gpu

LONG = [8192, 16384, 32768, 65536]
FOUR_STEP = "r16_cta256_shared_fp32_four_step"


@pytest.mark.parametrize("n", LONG)
@pytest.mark.parametrize("batch", [1, 2, 38, 151])
@pytest.mark.parametrize("direction", [-1, 1])
def test_rows_match_oracle_and_four_step(ctx, cuda, n, batch, direction):
    import torch
    plan, four = ctx.make_plan(), ctx.make_plan(FOUR_STEP, 8192, 1)
    x = torch.from_numpy(O.normal_input(n, batch, n % 89 + batch)).to(cuda).view(torch.complex64)
    y, f, z = torch.empty_like(x), torch.empty_like(x), x.clone()
    scale = 1.0 if direction < 0 else 1.0 / n
    assert plan.exec_c2c(x.data_ptr(), y.data_ptr(), n, batch, direction, scale, 0) == 0
    assert four.exec_c2c(x.data_ptr(), f.data_ptr(), n, batch, direction, scale, 0) == 0
    assert plan.exec_c2c(z.data_ptr(), z.data_ptr(), n, batch, direction, scale, 0) == 0   # in place
    torch.cuda.synchronize()
    rows = O.sample_batches(batch, 4)
    xd = x[rows].cpu().numpy().astype(np.complex128)
    ref = np.fft.fft(xd, axis=-1) if direction < 0 else np.fft.ifft(xd, axis=-1)
    assert O.rel_l2_rows(y[rows].cpu().numpy(), ref) <= 2e-6
    worst = (torch.linalg.vector_norm(y - f, dim=-1) / torch.linalg.vector_norm(f, dim=-1)).max().item()
    assert worst <= 1e-6, worst
    assert torch.equal(y, z)


@pytest.mark.parametrize("n", [64, 1024, 4096])
@pytest.mark.parametrize("tiles_past", [0, 1])
def test_short_rows_around_the_load_ahead_distance(ctx, cuda, n, tiles_past):
    """One row more than a whole number of CTAs, at and past the distance: the last tile that is
    loaded ahead is a partial one."""
    import torch
    rows = max(1, 256 * 16 // n)
    batch = rows * (296 + tiles_past) + 1
    x = torch.from_numpy(O.normal_input(n, batch, n)).to(cuda).view(torch.complex64)
    y = torch.empty_like(x)
    assert ctx.make_plan().exec_c2c(x.data_ptr(), y.data_ptr(), n, batch, -1, 1.0, 0) == 0
    torch.cuda.synchronize()
    ref = np.fft.fft(x.cpu().numpy().astype(np.complex128), axis=-1)
    assert O.rel_l2_rows(y.cpu().numpy(), ref) <= 1e-6
