"""The 32-bit products and attentions that take 16-byte loads, at the edges of their tiles, rows
and ranges, against float64. The bounds are those of sums in 32 bits: a sum of n products is off
by at most n * 2^-24 of the sum of their magnitudes, whatever the order."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
PAGE = 64


@pytest.fixture(scope="module")
def ops():
    from foundry_b200.kernels import ops as o
    return o


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed + sum(shape))).to(DEV)


def check_product(x, w, out):
    want = x.double() @ w.double().transpose(-1, -2)
    size = x.double().abs() @ w.double().abs().transpose(-1, -2)
    excess = ((out.double() - want).abs() - (x.shape[-1] + 2) * 2.0 ** -24 * size).max()
    assert float(excess) <= 0, float(excess)


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 129])
@pytest.mark.parametrize("N,K", [(1, 4), (7, 132), (65, 516), (130, 1028), (8196, 260), (8190, 128),
                                 (3, 4096)])
def test_product_of_16_byte_rows(ops, M, N, K):
    x, w = rnd(M, K), rnd(N, K, seed=1)
    wide = torch.full((M + 1, N + 5), 7.0, device=DEV)
    ops.gemm_simt(x, w, wide[:M, :N])
    check_product(x, w, wide[:M, :N])
    assert bool((wide[:, N:] == 7.0).all()) and bool((wide[M] == 7.0).all())  # nothing beyond


@pytest.mark.parametrize("M,N,K", [(3000, 4700, 64), (700, 70, 20)])
def test_product_of_large_tiles_and_views(ops, M, N, K):
    x, w = rnd(M, K + 8)[:, 4:K + 4], rnd(N, K + 12, seed=2)[:, 8:K + 8]  # strides, 16-byte bases
    out = torch.empty(M, N, device=DEV)
    ops.gemm_simt(x, w, out)
    check_product(x, w, out)


@pytest.mark.parametrize("M,off", [(3, 1), (40, 2), (5, 0)])
def test_views_without_16_byte_rows_take_the_general_kernel(ops, M, off):
    K = 130 if off == 0 else 128  # a K of no whole pieces, or a base that is not aligned
    x, w = rnd(M, 256)[:, off:off + K], rnd(50, 256, seed=3)[:, off:off + K]
    out = torch.empty(M, 50, device=DEV)
    ops.gemm_simt(x, w, out)
    check_product(x, w, out)


@pytest.mark.parametrize("M", [5, 16, 17, 70])
@pytest.mark.parametrize("K", [64, 300, 1100])
def test_batched_products(ops, M, K):
    x, w = rnd(M, 3, K), rnd(3, 66, K, seed=4)
    out = torch.empty(M, 3, 66, device=DEV)
    ops.gemm_simt_batched(x, w, out)
    for b in range(3):
        check_product(x[:, b], w[b], out[:, b])
