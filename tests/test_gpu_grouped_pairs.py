"""The experts' products with two SMs on a tile (weights as the instruction's rows, an expert's
tokens as its columns): cuts of the tokens, empty experts, both epilogues, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from foundry_b200.kernels import ops as o
    return o


class Order:
    def __init__(self, counts):
        starts = [0]
        for c in counts:
            starts.append(starts[-1] + c)
        self.experts, self.pairs, self.host = len(counts), starts[-1], starts
        self.starts = torch.tensor(starts, dtype=torch.int32, device="cuda")


COUNTS = [[1], [31, 0, 33], [128, 129, 64, 65], [256, 257, 0, 511, 513], [700, 1, 1, 0, 32],
          [16] * 96, [0, 0, 5]]


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("K,N", [(64, 256), (200, 512), (576, 768)])
def test_against_float64(ops, counts, K, N):
    order = Order(counts)
    gen = torch.Generator().manual_seed(sum(counts) + K)
    rows = torch.randn(order.pairs, K, generator=gen).bfloat16().cuda()
    w = (torch.randn(len(counts), N, K, generator=gen) / K ** 0.5).bfloat16().cuda()
    exact = torch.cat([rows[a:b].double() @ w[e].double().T for e, (a, b) in
                       enumerate(zip(order.host, order.host[1:]))])
    got = ops.gemm_tc_grouped(rows, w, order, persistent=2)
    # K float32 sums of products of about one: well inside 2^-18 of the largest partial sum
    assert float((got.double() - exact).abs().max()) < 2.0 ** -18 * 16
    # the form that smaller steps take gives the same bits (a padded step may take the other one)
    assert torch.equal(got, ops.gemm_tc_grouped(rows, w, order, persistent=1))
    half = ops.gemm_tc_grouped(rows, w, order, torch.bfloat16, persistent=2)
    assert torch.equal(half, got.bfloat16())
    limit, alpha, shift = 1.5, 1.7, 1.0
    got = ops.gemm_tc_grouped(rows, w, order, glu=(limit, alpha, shift), persistent=2)
    assert torch.equal(got, ops.gemm_tc_grouped(rows, w, order, glu=(limit, alpha, shift), persistent=1))
    gate, up = exact[:, :N // 2].clamp(max=limit), exact[:, N // 2:].clamp(-limit, limit)
    want = gate * torch.sigmoid(alpha * gate) * (up + shift)
    # rounded to bfloat16 (2^-9 of the value), products of errors of 2^-14
    assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -12).all())


def test_an_experts_rows_do_not_depend_on_the_others(ops):
    order = Order([100, 40, 300])
    gen = torch.Generator().manual_seed(2)
    rows = torch.randn(440, 128, generator=gen).bfloat16().cuda()
    w = torch.randn(3, 256, 128, generator=gen).bfloat16().cuda()
    first = ops.gemm_tc_grouped(rows, w, order, persistent=2)[100:140].clone()
    rows[:100], rows[140:] = float("nan"), float("inf")
    assert torch.equal(first, ops.gemm_tc_grouped(rows, w, order, persistent=2)[100:140])
