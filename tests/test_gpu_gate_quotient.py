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


def spread(count, low, high, gen):
    """Positive float32 numbers, their logarithms even over [low, high] (powers of two)."""
    return torch.exp2(torch.rand(count, generator=gen, dtype=torch.float64) * (high - low) + low).float()


@pytest.mark.parametrize("span", [(0, 1), (0, 24), (20, 125), (125, 127.99)])
def test_quotient_alone(span):
    """Rounded once: the Newton step and the correction leave the exact quotient's rounding but for
    2^-19 of the last place. (The plain product with the approximate reciprocal is up to one and a
    half places off, without the second of the two steps as much.)"""
    from foundry_b200.kernels import ops
    gen = torch.Generator().manual_seed(int(span[1]))
    d = spread(1 << 20, *span, gen).clamp(1.0, 3.4e38)
    n = spread(1 << 20, -20, 100, gen) * torch.where(torch.rand(1 << 20, generator=gen) < 0.5, -1.0, 1.0)
    got = ops.quotients(n.cuda(), d.cuda()).cpu()
    want = n.double() / d.double()
    place = torch.exp2(torch.floor(torch.log2(want.abs())).clamp(min=-126.0) - 23)
    assert float(((got.double() - want).abs() / place).max()) <= 0.5 + 2.0 ** -10
    # as the division rounds, but where the exact quotient lies between two numbers
    assert int((got != n / d).sum()) <= 2


def test_quotient_at_the_edges():
    from foundry_b200.kernels import ops
    inf, nan, small = float("inf"), float("nan"), 2.0 ** -140
    n, d = torch.meshgrid(torch.tensor([0.0, -0.0, 1.0, -1.0, 88.0, -88.5, small, -small, 3.4e38, -3.4e38,
                                        inf, -inf, nan]),
                          torch.tensor([1.0, 1.0 + 2.0 ** -23, 2.0, 3.0, 1e20, 1.7e38, 3.4e38, inf, nan]),
                          indexing="ij")
    got = ops.quotients(n.contiguous().cuda(), d.contiguous().cuda()).cpu()
    want = n / d
    assert torch.equal(got.isnan(), want.isnan())
    here = ~want.isnan()
    assert torch.equal(got.signbit()[here], want.signbit()[here])  # a zero keeps its sign
    same = (got == want) | ((got - want).abs() <= 2.0 ** -149)     # (the last place of subnormal numbers)
    assert bool(same[here].all()), (n[here][~same[here]], d[here][~same[here]])


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("limit,alpha,shift", [(7.0, 1.702, 1.0), (float("inf"), 1.0, 0.0)])
def test_clamped_gates_of_the_experts_products(form, limit, alpha, shift):
    """Extreme gates through every form of the grouped product: min(g, limit) times its sigmoid."""
    from foundry_b200.kernels import ops
    K, F, E, rows = 64, 128, 2, 300
    gates = torch.cat([torch.linspace(-120, 120, F - 8), torch.tensor(
        [0.0, -0.0, 3e38, -3e38, float("inf"), -float("inf"), float("nan"), 1e-30])]).bfloat16()
    x = torch.zeros(E * rows, K, dtype=torch.bfloat16)
    x[:, 0] = 1
    w = torch.zeros(E, 2 * F, K, dtype=torch.bfloat16)  # one weight a row: the sums are exact
    w[:, :F, 0], w[:, F:, 0] = gates, 1.0
    chosen = torch.arange(E, dtype=torch.int32).repeat_interleave(rows).view(-1, 1).cuda()
    order = ops.ExpertOrder(chosen, E)
    got = ops.gemm_tc_grouped(x.cuda(), w.cuda(), order, glu=(limit, alpha, shift), persistent=form).cpu().double()
    g = torch.minimum(gates.double().nan_to_num(limit, float("inf"), -float("inf")), torch.tensor(limit).double())
    want = (g / (1 + torch.exp(-alpha * g)) * (1.0 + shift)).expand(E * rows, F).clone()
    want[:, F - 3] = float("nan")  # -inf / inf
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    at = torch.isfinite(want)
    # bfloat16's rounding; gates far below zero meet an exponential that float32 does not hold
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + 1e-34)[at].all())
