"""Prompt attention over the step's own rows on tcgen05 (keys from two sources), against float64:
edges of blocks and key tiles, several sequences side by side, sizes, the sink, strided views."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from foundry_b200.kernels import ops as o
    return o


def step_of(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    as_int = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    return types.SimpleNamespace(n_seqs=len(lens), cu_tokens=as_int(cu), kv_lens=as_int(lens),
                                 cu_tokens_host=cu, query_blocks_bound=None), cu


@pytest.mark.parametrize("lens", [[64], [65], [127], [128], [129, 1, 63], [300, 70, 5]])
@pytest.mark.parametrize("k1,k2,e", [(64, 32, 64), (64, 64, 128), (64, 8, 72), (128, 64, 128), (128, 16, 64)])
def test_rows(ops, lens, k1, k2, e):
    H, T = 3, sum(lens)
    ctx, cu = step_of(lens)
    gen = torch.Generator().manual_seed(k1 + k2 + T)
    rnd = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16).to(DEV)  # noqa: E731
    q, kv, low = rnd(T, H * (k1 + k2)), rnd(T, H, k1 + e), rnd(T, 24 + k2)
    k, v, shared = kv[:, :, :k1], kv[:, :, k1:], low[:, 24:]
    scale, sink = (k1 + k2) ** -0.5, torch.randn(H, generator=gen).to(DEV)
    for s in (None, sink):
        out = torch.full((T, H * e), 9.0, dtype=torch.bfloat16, device=DEV)
        before = dict(ops.PROFILER.snapshot_counts())
        ops.PROFILER.start("steps")
        ops.attention_maps_rows(ctx, q, out, k, shared, v, H, k1 + k2, e, scale, sink_logits=s)
        counts = ops.PROFILER.take()["kernels"]
        ops.PROFILER.start(None)
        assert counts["attention_prefill_rows"]["dispatch_count"] == 1, (counts, before)
        for a, b in zip(cu, cu[1:]):
            n = b - a
            keys = torch.cat([k[a:b], shared[a:b, None].expand(n, H, k2)], -1).double()
            w = torch.einsum("ihd,jhd->hij", q[a:b].double().view(n, H, -1), keys) * scale
            w = w.masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool, device=DEV), 1), -torch.inf)
            if s is not None:
                w = torch.cat([w, s.double()[:, None, None].expand(H, n, 1)], -1)
            w = torch.softmax(w, -1)[..., :n]
            want = torch.einsum("hij,jhe->ihe", w, v[a:b].double()).reshape(n, -1)
            # weights and outputs rounded to bfloat16 (2^-9 each) of values of up to about four
            assert float((out[a:b].double() - want).abs().max()) < 4 * 2.0 ** -7


def test_another_sequences_numbers_do_not_matter(ops):
    """Rows of a sequence that are no numbers, behind and in front of one whose tiles touch them."""
    lens, H, T = [100, 90, 70], 2, 260
    ctx, cu = step_of(lens)
    gen = torch.Generator().manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16).to(DEV)  # noqa: E731
    q, kv, low = rnd(T, H * 96), rnd(T, H, 128), rnd(T, 32)
    results = []
    for spoil in (False, True):
        if spoil:
            for a, b in ((cu[0], cu[1]), (cu[2], cu[3])):
                kv[a:b] = float("nan")
                low[a:b] = float("inf")
        out = torch.empty(T, H * 64, dtype=torch.bfloat16, device=DEV)
        ops.attention_maps_rows(ctx, q, out, kv[:, :, :64], low, kv[:, :, 64:], H, 96, 64, 0.1)
        results.append(out[cu[1]:cu[2]].clone())
    assert bool(torch.isfinite(results[0]).all()) and torch.equal(*results)


@pytest.mark.parametrize("k1,k2,e", [(64, 32, 64), (64, 8, 72), (128, 16, 64)])
def test_another_heads_numbers_do_not_matter(ops, k1, k2, e):
    """Queries, keys and values of one head that are no numbers leave the other heads as they are."""
    H, T = 3, 200
    ctx, _ = step_of([T])
    gen = torch.Generator().manual_seed(11)
    rnd = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16).to(DEV)  # noqa: E731
    q, kv, low = rnd(T, H, k1 + k2), rnd(T, H, k1 + e), rnd(T, k2)
    results = []
    for spoil in (False, True):
        if spoil:
            q[:, 1], kv[:, 1] = float("nan"), float("inf")
        out = torch.empty(T, H, e, dtype=torch.bfloat16, device=DEV)
        ops.attention_maps_rows(ctx, q.view(T, -1), out.view(T, -1), kv[:, :, :k1], low, kv[:, :, k1:], H,
                                k1 + k2, e, 0.1)
        results.append(out[:, [0, 2]].clone())
    assert bool(torch.isfinite(results[0]).all()) and torch.equal(*results)


def plain(q, k, shared, v, H, scale):
    n = q.shape[0]
    keys = torch.cat([k, shared[:, None].expand(n, H, shared.shape[1])], -1).double()
    w = torch.einsum("ihd,jhd->hij", q.double().view(n, H, -1), keys) * scale
    w = w.masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool, device=DEV), 1), -torch.inf)
    return torch.einsum("hij,jhe->ihe", torch.softmax(w, -1), v.double()).reshape(n, -1)


@pytest.mark.parametrize("form", ["one head's keys for all", "one head's values for all", "one row of keys",
                                  "overlapping heads", "heads outside"])
def test_views_of_any_strides(ops, form):
    """Views whose heads or rows are no boxes side by side, too, as the kernel without tensor maps
    reads them."""
    H, T, e = 3, 96, 64
    ctx, _ = step_of([T])
    gen = torch.Generator().manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16).to(DEV)  # noqa: E731
    q, k, v, shared = rnd(T, H * 96), rnd(T, H, 64), rnd(T, H, e), rnd(T, 32)
    if form == "one head's keys for all":
        k = k[:, :1].expand(T, H, 64)
    elif form == "one head's values for all":
        v = v[:, :1].expand(T, H, e)
    elif form == "one row of keys":
        k, shared = k[:1].expand(T, H, 64), shared[:1].expand(T, 32)
    elif form == "overlapping heads":
        k = rnd(T, 96).as_strided((T, H, 64), (96, 16, 1))
    else:  # a head's rows together
        k, v = rnd(H, T, 64).transpose(0, 1), rnd(H, T, e).transpose(0, 1)
    out = torch.full((T, H * e), 9.0, dtype=torch.bfloat16, device=DEV)
    ops.attention_maps_rows(ctx, q, out, k, shared, v, H, 96, e, 0.1)
    want = plain(q, k, shared, v, H, 0.1)
    # weights and outputs rounded to bfloat16 (2^-9 each) of values of up to about four
    assert float((out.double() - want).abs().max()) < 4 * 2.0 ** -7


@pytest.mark.parametrize("k1,k2,e", [(64, 32, 64), (128, 64, 128)])
def test_as_close_to_float64_as_the_kernel_without_tensor_maps(ops, k1, k2, e, monkeypatch):
    """Both round weights and outputs to bfloat16; a weight of one, a row's largest, is exact in both."""
    H, T = 8, 900
    ctx, _ = step_of([T])
    gen = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16).to(DEV)  # noqa: E731
    q, k, v, shared = rnd(T, H * (k1 + k2)), rnd(T, H, k1), rnd(T, H, e), rnd(T, k2)
    scale = (k1 + k2) ** -0.5
    want, off = plain(q, k, shared, v, H, scale), []
    for tensor_maps in (True, False):
        monkeypatch.setattr(ops, "PREFILL_TC", tensor_maps)
        out = torch.empty(T, H * e, dtype=torch.bfloat16, device=DEV)
        ops.attention_maps_rows(ctx, q, out, k, shared, v, H, k1 + k2, e, scale)
        off.append(float((out.double() - want).norm() / want.norm()))
    assert off[0] <= off[1], off
