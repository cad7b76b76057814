"""Prompt attention with two maps a head, and with masks, on tcgen05, at the edges of its 128-row blocks and 64-key
pages, against float64 and beside the mma.sync kernel that it takes the place of."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
PAGE = 64


@pytest.fixture(scope="module")
def ops():
    from foundry_b200.kernels import ops as o
    return o


def make(lens, starts, H, G, vdim, size=1.0, seed=1):
    g = torch.Generator().manual_seed(seed)
    as_int = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    T, n = sum(lens), len(lens)
    width = max((s + l + PAGE - 1) // PAGE for s, l in zip(starts, lens)) + 1
    table = torch.randperm(n * width, generator=g).view(n, width).to(torch.int32).to(DEV)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV).bfloat16()  # noqa: E731
    q = rnd(T, H * 128 + 8)[:, :H * 128] * size
    k, v = rnd(n * width, G, PAGE, 128), rnd(n * width, G, PAGE, vdim)
    cu = [0]
    for l in lens:
        cu.append(cu[-1] + l)
    ctx = types.SimpleNamespace(is_decode=False, n_seqs=n, n_tokens=T, cu_tokens=as_int(cu), cu_tokens_host=cu,
                                kv_lens=as_int([s + l for s, l in zip(starts, lens)]),
                                query_blocks_bound=None, long_queries=max(lens) >= 64)
    return ctx, q, k, v, table


def exact(q, k, v, table, lens, starts, H, G, vdim, scale, cap, sink, combine):
    """What float64 gives, and the sums of the values' magnitudes by both maps' weights."""
    lam, eps, post = combine
    outs, sizes, t0 = [], [], 0
    for i, (n, s) in enumerate(zip(lens, starts)):
        j = torch.arange(s + n, device=DEV)
        kk, vv = (c[table[i][j // PAGE].long(), :, j % PAGE].double().repeat_interleave(H // G, 1) for c in (k, v))
        qq = q[t0:t0 + n].double().view(n, H, 2, 64)
        t0 += n
        late = j[None] > (s + torch.arange(n, device=DEV))[:, None]
        a, m = [], []
        for mm in range(2):
            z = torch.einsum("thd,jhd->htj", qq[:, :, mm], kk[:, :, mm * 64:mm * 64 + 64]) * scale
            if cap:
                z = cap * torch.tanh(z / cap)
            z = z.masked_fill(late, -float("inf"))
            if sink is not None:
                z = torch.cat([z, sink.double()[:, None, None].expand(H, n, 1)], -1)
            w = torch.softmax(z, -1)[..., :s + n]
            a.append(torch.einsum("htj,jhe->the", w, vv))
            m.append(torch.einsum("htj,jhe->the", w, vv.abs()))
        o = a[0] - lam * a[1]
        r = post / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)
        outs.append((o * r).flatten(1))
        off = 2.0 ** -8 * (m[0] + lam * m[1])  # weights rounded to bfloat16, up to half a place each, twice
        rel = (off * off).mean(-1, keepdim=True).sqrt() / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)
        sizes.append((off * r + (o * r).abs() * (rel + 2.0 ** -8)).flatten(1))
    return torch.cat(outs), torch.cat(sizes)


@pytest.mark.parametrize("lens,starts", [([65], [0]), ([130], [0]), ([300, 65, 70], [0, 0, 0]),
                                         ([200, 64], [37, 128]), ([300, 1, 90], [0, 500, 63])])
@pytest.mark.parametrize("H,G,vdim,cap,size,sinks", [(4, 2, 128, 50.0, 1.0, False), (3, 1, 64, 0.0, 1.0, False),
                                                     (2, 2, 128, 3.0, 3.0, True), (8, 2, 64, 30.0, 0.3, True)])
def test_two_maps(ops, lens, starts, H, G, vdim, cap, size, sinks):
    ctx, q, k, v, table = make(lens, starts, H, G, vdim, size)
    combine, scale = (0.3, 1e-5, 0.2), 0.125
    sink = torch.randn(H, generator=torch.Generator().manual_seed(9)).to(DEV) if sinks else None
    out, old = (torch.full((sum(lens), H * vdim + 8), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    assert ops._tc_maps_blocks(ctx, q, out, k, v, G, 64, vdim, 2, scale) > 0
    args = (table, k, v, H, G, 64, vdim, 2, scale, cap, sink, combine)
    ops.attention_maps_paged(ctx, q, out[:, :H * vdim], *args)
    room, ops.MAPS_WORKSPACE = ops.MAPS_WORKSPACE, 0  # no room for both maps: mma.sync
    try:
        ops.attention_maps_paged(ctx, q, old[:, :H * vdim], *args)
    finally:
        ops.MAPS_WORKSPACE = room
    assert bool((out[:, H * vdim:] == 7).all()) and ops.gemm_tc_status() == 0
    want, bound = exact(q, k, v, table, lens, starts, H, G, vdim, scale, cap, sink, combine)
    off, before = (x[:, :H * vdim].double() - want for x in (out, old))
    assert bool((off.abs() <= bound).all())
    assert float(off.norm()) <= 1.05 * float(before.norm())  # the same roundings, in another order


@pytest.mark.parametrize("H,G,heads", [(8, 2, 4), (8, 2, 2), (8, 2, 1), (6, 6, 3), (3, 1, 1)])
def test_two_maps_with_little_memory(ops, monkeypatch, H, G, heads):
    """Where memory for all heads is missing, they are worked in parts, with the same bits; rows of padding
    tokens, which no block makes, are not written from what the memory held."""
    lens, vdim = [200, 65], 128
    ctx, q, k, v, table = make(lens, [37, 0], H, G, vdim)
    T = sum(lens)
    q = torch.cat([q, torch.zeros_like(q[:20])])[:, :H * 128]
    sink = torch.randn(H, generator=torch.Generator().manual_seed(9)).to(DEV)
    args = (table, k, v, H, G, 64, vdim, 2, 0.125, 50.0, sink, (0.3, 1e-5, 0.2))
    whole, parts = (torch.full((T + 20, H * vdim), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    assert ops._tc_maps_blocks(ctx, q, whole, k, v, G, 64, vdim, 2, 0.125) > 0
    ops.attention_maps_paged(ctx, q, whole, *args)
    empty, most = torch.empty, (T + 20) * heads * 2 * vdim
    asked = []

    def little(*size, **how):
        if how.get("dtype") == torch.float32:
            asked.append(size[0])
            if size[0] > most:
                raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **how)
    monkeypatch.setattr(ops.torch, "empty", little)
    ops.attention_maps_paged(ctx, q, parts, *args)
    monkeypatch.undo()
    assert asked[-1] == most and len(asked) > 1 and torch.equal(parts, whole)
    assert bool((whole[T:] == 7).all())


def test_what_the_form_does_not_take_stays(ops):
    ctx, q, k, v, table = make([100, 20, 1], [0, 0, 0], 4, 2, 128)
    out = torch.empty(121, 512, dtype=torch.bfloat16, device=DEV)
    takes = lambda c=ctx, q=q, k=k, v=v, dim=64, vdim=128, scale=0.1: ops._tc_maps_blocks(  # noqa: E731
        c, q, out, k, v, 2, dim, vdim, 2, scale)
    assert takes() == 0  # 32 tokens a sequence on average, padded
    long, q2, k2, v2, _ = make([100], [0], 4, 2, 128)
    out = out[:100]
    assert takes(long, q2, k2, v2) == 1
    assert takes(long, q2, k2, v2, scale=-0.1) == 0 and takes(long, q2, k2, v2, dim=32, vdim=32) == 0
    assert takes(long, q2, k2[:, :1].expand(-1, 2, -1, -1), v2) == 0  # heads that lie over one another
    shifted = torch.empty(100 * 520 + 8, dtype=torch.bfloat16, device=DEV)[4:100 * 520 + 4].view(100, 520)[:, :512]
    assert takes(long, shifted, k2, v2) == 0  # rows that are not on 16-byte boundaries
    # the masked form: more than 256 tokens, heads of 64 or 128
    masked = lambda c, q, k, v, dim=128, steep=8.0: ops._tc_mask_blocks(c, q, q, k, v, 2, dim, 0.1, steep)  # noqa: E731
    few, q3, k3, v3, _ = make([200], [0], 4, 2, 128)
    many, q4, k4, v4, _ = make([300], [0], 4, 2, 128)
    assert masked(few, q3, k3, v3) == 0 and masked(many, q4, k4, v4) == 3
    assert masked(many, q4, k4, v4, dim=96) == 0 and masked(many, q4, k4, v4, steep=-1.0) == 0


def exact_masked(q, k, v, table, lens, starts, H, G, D, scale, window, keep, sink, logits, steep):
    outs, sizes, t0 = [], [], 0
    for i, (n, s) in enumerate(zip(lens, starts)):
        j = torch.arange(s + n, device=DEV)
        kk, vv = (c[table[i][j // PAGE].long(), :, j % PAGE].double().repeat_interleave(H // G, 1) for c in (k, v))
        qq = q[t0:t0 + n].double().view(n, H, D)
        t0 += n
        back = (s + torch.arange(n, device=DEV))[:, None] - j[None]
        z = torch.einsum("thd,jhd->htj", qq, kk) * scale
        if steep:
            slope = 2.0 ** (-steep * torch.arange(1, H + 1, device=DEV).double() / H)
            z = z - slope[:, None, None] * back
        seen = back >= 0
        if window:
            seen &= (back < window) | (j[None] < keep)
        z = z.masked_fill(~seen, -float("inf"))
        if sink:
            term = torch.zeros(H, device=DEV).double() if logits is None else logits.double()
            z = torch.cat([z, term[:, None, None].expand(H, n, 1)], -1)
        w = torch.softmax(z, -1)[..., :s + n]
        outs.append(torch.einsum("htj,jhe->the", w, vv).flatten(1))
        sizes.append(torch.einsum("htj,jhe->the", w, vv.abs()).flatten(1))
    return torch.cat(outs), torch.cat(sizes)


@pytest.mark.parametrize("lens,starts", [([390], [0]), ([300, 65, 70], [0, 0, 0]), ([200, 64], [37, 128]),
                                         ([300, 1, 90], [0, 500, 63])])
@pytest.mark.parametrize("H,G,D,window,keep,sink,logits,steep", [
    (4, 2, 64, 0, 0, 0, False, 8.0), (3, 1, 128, 100, 4, 1, False, 8.0), (4, 4, 64, 64, 0, 1, False, 0.0),
    (2, 2, 128, 129, 70, 1, True, 2.0), (4, 2, 64, 1, 0, 0, False, 0.0)])
def test_masked(ops, lens, starts, H, G, D, window, keep, sink, logits, steep):
    ctx, _, _, _, table = make(lens, starts, H, G, 64)
    g = torch.Generator().manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV).bfloat16()  # noqa: E731
    T = sum(lens)
    q, kv = rnd(T, H * D + 8)[:, :H * D], rnd(table.numel(), 2, G, PAGE, D)
    k, v = kv[:, 0], kv[:, 1]
    terms = torch.randn(H, generator=g).to(DEV) if logits else None
    out, old = (torch.full((T, H * D + 8), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    scale = D ** -0.5
    assert ops._tc_mask_blocks(ctx, q, out, k, v, G, D, scale, steep) > 0
    args = dict(window=window, keep_first=keep, sink=bool(sink and not logits), steep=steep, sink_logits=terms)
    ops.attention_sink(ctx, q, out[:, :H * D], table, k, v, H, G, D, D, scale, **args)
    ops.PREFILL_TC, before = False, ops.PREFILL_TC
    try:
        ops.attention_sink(ctx, q, old[:, :H * D], table, k, v, H, G, D, D, scale, **args)
    finally:
        ops.PREFILL_TC = before
    assert bool((out[:, H * D:] == 7).all()) and ops.gemm_tc_status() == 0
    want, size = exact_masked(q, k, v, table, lens, starts, H, G, D, scale, window, keep, sink, terms, steep)
    off, was = (x[:, :H * D].double() - want for x in (out, old))
    # weights and the result rounded to bfloat16: half a place of each, twice for what else is 32-bit
    assert bool((off.abs() <= 2.0 ** -8 * size + 2.0 ** -8 * want.abs()).all())
    assert float(off.norm()) <= 1.05 * float(was.norm()) + 1e-9
