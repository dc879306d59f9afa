"""The C++ module's plan table: a plan that was asked for before the table was emptied (an autotune
that ends while another thread looks its plan up) does not come back into it."""
import pytest

pytestmark = pytest.mark.gpu


def test_an_old_plan_is_not_kept(cuda, monkeypatch):
    import torch
    from bfly import ops
    x = torch.randn(2, 512, dtype=torch.complex64, device=cuda)
    want = ops.fft(x)
    real, asked = ops.plan_for, []

    def plan_for(device, n=None, kind="c2c"):
        p = real(device, n, kind)
        asked.append(n)
        if len(asked) == 1:
            ops._native.forget_plans()   # between the question and the answer
        return p

    ops._native.forget_plans()
    monkeypatch.setattr(ops, "plan_for", plan_for)
    for _ in range(3):
        assert torch.equal(ops.fft(x), want)
    assert asked == [512, 512]   # asked again after the table was emptied, then kept
