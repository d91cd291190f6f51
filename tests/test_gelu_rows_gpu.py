"""The tanh form of gelu, row by row, over every bfloat16 value."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [512, 514])          # whole 16-byte vectors, and one value at a time
@pytest.mark.parametrize("gated", [False, True])
def test_every_bfloat16(columns, gated):
    from llmgen_b200.kernels import ops
    every = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda()
    rows = -(-every.numel() // columns)
    z = torch.zeros(rows * columns, dtype=torch.bfloat16, device="cuda")
    z[: every.numel()] = every
    z = z.view(rows, columns)
    out = torch.empty_like(z)
    if gated:
        # all gates, then all ups (a power of two, which rounds nothing)
        ops.act_rows(out, torch.cat([z, torch.full_like(z, 2.0)], dim=1), "gelu_tanh_glu")
    else:
        ops.act_rows(out, z, "gelu_tanh")
    x = z.double()
    want = x / (1 + torch.exp(-2 * 0.7978845608028654 * (x + 0.044715 * x ** 3))) * (2.0 if gated else 1.0)
    usual = torch.isfinite(x) & (want.abs() > 1e-30) & (want.abs() < 3e38)
    # one rounding to bfloat16 (2^-8 of the value at most); float32's exponential of |2 u| < 80 adds 80 of its units (2^-24 each) and a few more
    assert float(((out.double() - want)[usual] / want[usual]).abs().max()) <= 2.0 ** -8 + 100 * 2.0 ** -24
    assert float(out.double()[torch.isfinite(x) & (want.abs() <= 1e-30)].abs().max()) <= 1e-29
    assert torch.equal(torch.isnan(out), torch.isnan(x) | (x == -float("inf")))
