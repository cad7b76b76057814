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
                                 (3, 4096), (8193, 64), (8200, 200), (34, 124)])
def test_product_of_16_byte_rows(ops, M, N, K):
    x, w = rnd(M, K), rnd(N, K, seed=1)
    wide = torch.full((M + 1, N + 5), 7.0, device=DEV)
    ops.gemm_simt(x, w, wide[:M, :N])
    check_product(x, w, wide[:M, :N])
    assert bool((wide[:, N:] == 7.0).all()) and bool((wide[M] == 7.0).all())  # nothing beyond


@pytest.mark.parametrize("M", [1, 8, 16, 32, 33, 64, 129])
@pytest.mark.parametrize("K", [1028, 4096, 4100])
def test_no_term_of_a_long_sum_is_lost(ops, M, K):
    """Products of independent signs: a sum of i of them is about sqrt(i) of their root mean square,
    |x||w| / K, and each addition rounds it by up to 2^-24, errors of independent signs again: 0.41 *
    2^-24 * |x||w| in the root mean square where they are added one by one. Seven times that is far
    below one product."""
    x, w = rnd(M, K), rnd(70, K, seed=1)
    out = torch.empty(M, 70, device=DEV)
    ops.gemm_simt(x, w, out)
    want = x.double() @ w.double().T
    norms = x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)
    assert float(((out.double() - want).abs() / norms).max()) < 3 * 2.0 ** -24


@pytest.mark.parametrize("M,N,K", [(3000, 4700, 64), (700, 70, 20)])
def test_product_of_large_tiles_and_views(ops, M, N, K):
    x, w = rnd(M, K + 8)[:, 4:K + 4], rnd(N, K + 12, seed=2)[:, 8:K + 8]  # strides, 16-byte bases
    out = torch.empty(M, N, device=DEV)
    ops.gemm_simt(x, w, out)
    check_product(x, w, out)


@pytest.mark.parametrize("M", [33, 64, 65, 128, 209, 417])
@pytest.mark.parametrize("N,K", [(128, 1024), (257, 1028), (300, 4100), (2100, 1056), (8200, 1060)])
def test_product_of_pieces(ops, M, N, K):
    """Edges of the tensor cores' tiles (256 weight rows, 16 to 208 tokens, 32 of K), with and without
    several pairs of SMs on a tile's K, as a view into a wider matrix."""
    x, w = rnd(M, K + 8)[:, 4:K + 4], rnd(N, K, seed=1)
    wide = torch.full((M + 1, N + 5), 7.0, device=DEV)
    ops.gemm_simt(x, w, wide[:M, :N])
    check_product(x, w, wide[:M, :N])
    assert bool((wide[:, N:] == 7.0).all()) and bool((wide[M] == 7.0).all())  # nothing beyond
    assert ops.gemm_tc_status() == 0


@pytest.mark.parametrize("M", [17, 32])
@pytest.mark.parametrize("N,K", [(10504, 200), (21900, 96), (11000, 204)])
def test_up_to_32_rows_are_multiplied_and_added(ops, M, N, K):
    """However many columns: the bits are those of the first 8,200 columns alone, which are too few for the
    tensor cores."""
    x, w = rnd(M, K), rnd(N, K, seed=1)
    out, few = torch.empty(M, N, device=DEV), torch.empty(M, 8200, device=DEV)
    ops.gemm_simt(x, w, out)
    ops.gemm_simt(x, w[:8200], few)
    check_product(x, w, out)
    assert torch.equal(out[:, :8200], few)


@pytest.mark.parametrize("N", [300, 9000])
def test_product_of_pieces_rounds_no_more_than_a_chain(ops, N):
    """A chain of K additions is off by about 0.41 * 2^-24 * |x||w| in the root mean square (see
    test_no_term_of_a_long_sum_is_lost); 32 of K at a time, a sum is off by less than half of that."""
    x, w = rnd(100, 4096), rnd(N, 4096, seed=1)
    out = torch.empty(100, N, device=DEV)
    ops.gemm_simt(x, w, out)
    norms = x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)
    off = (out.double() - x.double() @ w.double().T) / norms
    assert float(off.square().mean().sqrt()) < 0.2 * 2.0 ** -24


@pytest.mark.parametrize("N", [300, 9000])
def test_product_of_pieces_of_what_pieces_cannot_carry(ops, N):
    """Infinities, NaN, overflow and operands near the smallest normal number come out as a chain of
    32-bit FMAs gives them."""
    x, w = rnd(64, 1024), rnd(N, 1024, seed=1)
    x[3, 5], x[7, 9], w[100, 77] = float("inf"), float("nan"), float("-inf")
    w[5] = 2.0 ** torch.randint(-3, 3, (1024,)).float()  # one piece each: the others are zero
    x[9], w[11] = 3e38, 1.0
    x[20] *= 1e-36
    w[21] *= 1e-35
    out = torch.empty(64, N, device=DEV)
    ops.gemm_simt(x, w, out)
    plain = torch.empty(64, N, device=DEV)
    for r in range(0, 64, 32):  # up to 32 rows: FMAs
        ops.gemm_simt(x[r:r + 32], w, plain[r:r + 32])
    assert float(out[9, 11]) == float("inf")
    out[9], plain[9] = 0, 0  # elsewhere in the row the order decides what overflows first
    assert torch.equal(out.isnan(), plain.isnan()) and torch.equal(out.isinf(), plain.isinf())
    assert torch.equal(out.isposinf(), plain.isposinf())
    whole = plain.isfinite()
    size = (x.double().abs() @ w.double().abs().T)[whole]
    # (1024 + 2) * 2^-24 of the magnitudes for either sum, and what rounding below 2^-126 takes
    gap = (out.double() - plain.double()).abs()[whole] - 2 * 1026 * 2.0 ** -24 * size
    assert float(gap.max()) <= 2.0 ** -126


@pytest.mark.parametrize("N", [300, 9000])
@pytest.mark.parametrize("of_x,of_w", [(1e-34, 1e8), (1e-36, 1e10), (1e-38, 1e12), (3e-40, 1e15),
                                       (1e-39, 1e30), (1e-43, 1e30), (1e10, 1e-36), (1e-20, 1e-18)])
def test_product_of_pieces_of_small_times_large(ops, N, of_x, of_w):
    """Operands whose pieces are below the smallest normal number, times operands that make results of
    any size of them: all tokens, one of them, one number of a token."""
    for rows, cols in ((slice(None), slice(None)), (slice(5, 6), slice(None)), (slice(40, 41), slice(9, 10))):
        x, w = rnd(64, 1024), rnd(N, 1024, seed=1) * of_w
        x[rows, cols] *= of_x
        x[50] = 0.0
        out = torch.empty(64, N, device=DEV)
        ops.gemm_simt(x, w, out)
        size = x.double().abs() @ w.double().abs().T
        # products of 2^-24 of their magnitude each; below the smallest normal number, 2^-149 each
        gap = (out.double() - x.double() @ w.double().T).abs() - 1026 * (2.0 ** -24 * size + 2.0 ** -149)
        assert float(gap.max()) <= 0, float(gap.max())


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("M,N,K", [(100, 300, 4096), (777, 300, 1024), (777, 9000, 1028), (1500, 20000, 512)])
def test_product_of_pieces_of_tokens_that_are_no_numbers(ops, M, N, K, value):
    """Every result of every tile falls (with and without several pairs on a tile's K, several tiles a
    pair): they are summed again behind the tiles, and no wait of the others runs out meanwhile."""
    x, w = torch.full((M, K), value, device=DEV), rnd(N, K, seed=1).abs() + 0.1
    w[7, 3] = 0.0
    out = torch.zeros(M, N, device=DEV)
    ops.gemm_simt(x, w, out)
    want = torch.full((M, N), value, device=DEV)
    want[:, 7] = float("nan")
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isposinf(), want.isposinf())
    assert ops.gemm_tc_status() == 0


@pytest.mark.parametrize("M,N,K", [(900, 500, 64), (700, 300, 1028)])
def test_many_batched_products(ops, M, N, K):
    x, w = rnd(M, 32, K), rnd(32, N, K, seed=4)
    out = torch.empty(M, 32, N, device=DEV)
    ops.gemm_simt_batched(x, w, out)
    for b in (0, 13, 31):
        check_product(x[:, b], w[b], out[:, b])


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


def paged_case(runs, Kh, G, D, ring=0, seed=5):
    """`runs`: (sequence, first position, tokens) in token order; -1 = padding rows."""
    n_seqs = max(s for s, _, _ in runs) + 1
    longest = max(a + n for _, a, n in runs)
    width = ring or (longest + PAGE - 1) // PAGE
    order = torch.randperm(n_seqs * width, generator=torch.Generator().manual_seed(seed))
    table = order.view(n_seqs, width).to(torch.int32).to(DEV)
    k, v = rnd(n_seqs * width, Kh, PAGE, D, seed=6), rnd(n_seqs * width, Kh, PAGE, D, seed=7)
    seq = torch.cat([torch.full((n,), s, dtype=torch.int32) for s, _, n in runs]).to(DEV)
    pos = torch.cat([torch.arange(a, a + n, dtype=torch.int32) for _, a, n in runs]).to(DEV)
    return dict(q=rnd(seq.numel(), Kh * G * D, seed=8), table=table, k=k, v=v, seq=seq, pos=pos)


def check_attention(ops, case, Kh, G, D, window=0, ring=0):
    T = case["seq"].numel()
    out = torch.full((T, Kh * G * D), 9.0, device=DEV)
    scale = D ** -0.5
    ops.attention_simt(case["q"], out, case["pos"], case["seq"], case["table"], case["k"], case["v"],
                       Kh * G, Kh, D, scale, window, ring)
    q = case["q"].double().view(T, Kh * G, D)
    worst = 0.0
    for t in range(T):
        s, p = int(case["seq"][t]), int(case["pos"][t])
        if s < 0:
            assert bool((out[t] == 0).all())
            continue
        j = torch.arange(max(0, p - window + 1) if window else 0, p + 1, device=DEV)
        page = j // PAGE % ring if ring else j // PAGE
        pages = case["table"][s][page].long()
        k, v = case["k"][pages, :, j % PAGE].double(), case["v"][pages, :, j % PAGE].double()
        k, v = k.repeat_interleave(G, 1), v.repeat_interleave(G, 1)  # [keys, heads, D]
        w = torch.softmax(torch.einsum("hd,jhd->hj", q[t], k) * scale, -1)
        want = torch.einsum("hj,jhd->hd", w, v)
        worst = max(worst, float((out[t].double().view(-1, D) - want).abs().max()))
    # scores of a few units, off by D * 2^-24 of |q||k| * scale <= 30; weights by as much; their sums
    # by the number of keys * 2^-24 of |v| <= 5
    assert worst < (30 * D + 5 * 600) * 2.0 ** -24, worst


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("G", [1, 3, 4, 6])
def test_attention_of_single_tokens(ops, D, G):
    runs = [(0, 0, 1), (1, 599, 1), (2, 63, 1), (-1, 0, 1), (3, 64, 1), (4, 15, 1)]
    check_attention(ops, paged_case(runs, 2, G, D), 2, G, D)


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("runs", [
    [(0, 0, 130)],                                                     # blocks' and tiles' edges
    [(0, 37, 64), (1, 0, 65)],                                         # continued; ends in a block
    [(0, 0, 17), (1, 200, 20), (2, 3, 16), (3, 0, 40), (-1, 0, 30)],   # runs in one block, padding
    [(0, 0, 65), (-1, 0, 63)], [(0, 590, 1), (-1, 0, 20), (0, 591, 50)],  # blocks that share the keys
])
def test_attention_of_prompts(ops, D, runs):
    check_attention(ops, paged_case(runs, 2, 2, D), 2, 2, D)


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("Kh,G", [(1, 1), (2, 3), (8, 4), (3, 6)])
@pytest.mark.parametrize("runs", [
    [(0, 0, 8), (1, 0, 3), (2, 61, 9), (3, 250, 2)],                     # one or two warps a pair
    [(i, 3 * i, 1 + i % 16) for i in range(18)] + [(-1, 0, 5)],
    [(i, 0, 17) for i in range(5)] + [(5, 30, 20)],                      # runs between warps' rows
])
def test_attention_of_short_prompts(ops, D, Kh, G, runs):
    check_attention(ops, paged_case(runs, Kh, G, D), Kh, G, D)


def test_attention_of_short_prompts_with_a_window(ops):
    runs = [(i, 7 * i, 6) for i in range(12)]
    check_attention(ops, paged_case(runs, 2, 4, 64, ring=3), 2, 4, 64, 5, 3)


@pytest.mark.parametrize("runs", [[(0, 0, 1), (1, 250, 1)], [(0, 180, 70)]])
@pytest.mark.parametrize("window", [1, 20, 90])
def test_attention_with_a_window_on_a_ring(ops, runs, window):
    ring = (window + PAGE - 1) // PAGE + 2
    check_attention(ops, paged_case(runs, 1, 2, 64, ring=ring), 1, 2, 64, window, ring)


@pytest.mark.parametrize("tokens", [100, 12])  # tiles; ranges
def test_a_later_token_that_is_no_number_does_not_reach_earlier_ones(ops, tokens):
    case = paged_case([(0, 0, tokens)], 1, 1, 64)
    bad = tokens * 7 // 10
    for name in ("k", "v"):
        case[name][case["table"][0][bad // PAGE].long(), 0, bad % PAGE] = float("nan")
    out = torch.empty(tokens, 64, device=DEV)
    ops.attention_simt(case["q"], out, case["pos"], case["seq"], case["table"], case["k"], case["v"],
                       1, 1, 64, 0.125)
    assert bool(torch.isfinite(out[:bad]).all()) and bool(torch.isnan(out[bad:]).all())
