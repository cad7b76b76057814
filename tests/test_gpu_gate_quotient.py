"""The gated products' activation at its edges: gates far out on both sides, infinite and no
numbers, against the division in float32 that it stands for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [4, 40, 300])
def test_silu_of_any_gate(rows):
    from foundry_b200.kernels import ops
    K, F = 64, 128
    gates = torch.cat([torch.linspace(-120, 120, F - 8), torch.tensor(
        [0.0, -0.0, 3e38, -3e38, float("inf"), -float("inf"), float("nan"), 1e-30])]).bfloat16()
    x = torch.zeros(rows, K, dtype=torch.bfloat16)
    x[:, 0] = 1
    w = torch.zeros(2 * F, K, dtype=torch.bfloat16)  # one weight a row: the sums are exact
    w[0::2, 0], w[1::2, 0] = gates, 1.0
    out = torch.empty(rows, F, dtype=torch.bfloat16, device="cuda")
    ops.gemm_bf16_silu_mul(x.cuda(), w.cuda(), out)
    g = gates.double()
    want = (g / (1 + torch.exp(-g))).expand(rows, F).cuda()
    want[:, F - 3] = float("nan")  # -inf / inf
    got = out.double()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    at = torch.isfinite(want)
    # bfloat16's rounding; gates below about -87 meet an exponential that float32 does not hold
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + 1e-35)[at].all())
