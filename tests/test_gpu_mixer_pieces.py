"""The per-token pieces around the recurrences that read whole 16-byte pieces or take several steps
in one kernel, at the edges of their runs and blocks, against plain statements of the same work."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from foundry_b200.kernels import ops as o
    return o


def step_of(runs, n_slots, decode=False):
    """A context of `runs` = tokens of each sequence, three padding rows behind them."""
    seq, cu = [], [0]
    for i, n in enumerate(runs):
        seq += [i] * n
        cu.append(cu[-1] + n)
    seq += [-1] * 3
    as_int = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    slots = torch.randperm(n_slots, generator=torch.Generator().manual_seed(3))[:len(runs)].tolist()
    return types.SimpleNamespace(is_decode=decode, n_seqs=len(runs), seq_of_token=as_int(seq),
                                 cu_tokens=as_int(cu), slots=as_int(slots)), slots, cu, len(seq)


@pytest.mark.parametrize("runs", [[1, 1, 1, 1, 1], [1], [3, 70, 1, 2], [530, 9]])
@pytest.mark.parametrize("dim,taps", [(64, 2), (64, 4), (128, 3), (128, 4), (96, 4)])
def test_convolution(ops, runs, dim, taps):
    decode = max(runs) == 1
    ctx, slots, cu, T = step_of(runs, 7, decode)
    n_unit, n_scaled, heads, extra = 3, 1, 5, 0.3
    C = heads * dim
    gen = torch.Generator().manual_seed(dim + taps)
    x = torch.randn(T, C + 8, generator=gen).to(DEV)[:, 4:C + 4]
    w, bias = torch.randn(C, taps, generator=gen).to(DEV), torch.randn(C, generator=gen).to(DEV)
    for b, unit in ((None, n_unit), (bias, n_unit), (bias, 0)):
        rows = torch.randn(8, 8 + (taps - 1) * C, generator=torch.Generator().manual_seed(9)).to(DEV)
        before = rows.clone()
        state = ops.StateRows(rows, [("other", 8), ("tail", (taps - 1) * C)])
        out = torch.full((T, C), 9.0, device=DEV)
        moved = ops.conv_silu_unit(ctx, x, w, state, "tail", out, C, n_unit=unit, dim=dim,
                                   n_scaled=n_scaled if unit else 0, extra=extra, unit_eps=1e-6, bias=b)
        assert moved == decode
        for s, slot in enumerate(slots):
            past = before[slot, 8:].view(taps - 1, C).double()
            full = torch.cat([past, x[cu[s]:cu[s + 1]].double()])
            n = cu[s + 1] - cu[s]
            y = sum(full[a:a + n] * w[:, a].double() for a in range(taps)) + (0 if b is None else b.double())
            y = (y * torch.sigmoid(y)).view(n, heads, dim)
            if unit:
                r = 1.0 / torch.sqrt((y[:, :unit] ** 2).sum(-1, keepdim=True) + 1e-6)
                r[:, :n_scaled] *= extra
                y[:, :unit] *= r
            # four products, an exponential and a root: a few 2^-23 of values of up to ten
            assert float((out[cu[s]:cu[s + 1]].double() - y.view(n, C)).abs().max()) < 2e-5
            want = full[-(taps - 1):] if decode else past
            assert torch.equal(rows[slot, 8:].view(taps - 1, C), want.float())
        assert bool((out[cu[-1]:] == 0).all()) and torch.equal(rows[:, :8], before[:, :8])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("runs", [[1, 1, 1], [5, 1, 3], [517, 2]])
@pytest.mark.parametrize("W", [64, 2056, 100])
def test_token_shift(ops, runs, W, dtype):
    decode = max(runs) == 1
    ctx, slots, cu, T = step_of(runs, 5, decode)
    gen = torch.Generator().manual_seed(W)
    h = torch.randn(T, W, generator=gen).to(dtype).to(DEV)
    mu = torch.rand(5, W, generator=gen).to(DEV)
    rows = torch.randn(6, 4 + W, generator=gen).to(DEV)
    before = rows.clone()
    out = torch.full((5, T, W), 9.0, dtype=dtype, device=DEV)
    ops.token_shift_mix(ctx, h, ops.StateRows(rows, [("other", 4), ("prev", W)]), "prev", mu, out)
    for s, slot in enumerate(slots):
        x = h[cu[s]:cu[s + 1]].float()
        prev = torch.cat([before[slot, 4:][None], x[:-1]])
        want = (x + (prev - x) * mu[:, None]).to(dtype)
        assert float((out[:, cu[s]:cu[s + 1]].float() - want.float()).abs().max()) < \
            (0.04 if dtype == torch.bfloat16 else 1e-6)  # a rounding of values of up to five
        assert torch.equal(rows[slot, 4:], x[-1] if decode else before[slot, 4:])
    assert bool((out[:, cu[-1]:] == 0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T", [1, 7, 8, 9, 16, 17, 50])
@pytest.mark.parametrize("rank,n", [(8, 5), (64, 200), (40, 129)])
def test_low_rank(ops, T, rank, n, dtype):
    gen = torch.Generator().manual_seed(T + rank)
    x = torch.randn(T, rank + 7, generator=gen).to(DEV)[:, 3:3 + rank]
    w = (torch.randn(n, rank, generator=gen) / rank ** 0.5).to(dtype).to(DEV)
    bias = torch.randn(n, generator=gen).to(DEV)
    per_head = 1 if n % 5 else 5
    A = torch.randn(n // per_head, generator=gen).to(DEV)
    for act in ("identity", "tanh"):
        rounded = (torch.tanh(x) if act == "tanh" else x).to(dtype).double()
        z = rounded @ w.double().T
        rate = torch.exp(A.double()).repeat_interleave(per_head)
        y = z + bias.double()
        for kw, want in ((dict(), z), (dict(bias=bias), torch.exp(-torch.exp(y))),
                         (dict(bias=bias, A=A, per_head=per_head),
                          torch.exp(-rate * torch.nn.functional.softplus(y)))):
            got = ops.low_rank(x, w, act, **kw)
            # sums of `rank` products near one; a decay moves by no more than its exponent does
            # (a hyperbolic tangent next to a rounding edge may round the other way)
            bound = 4e-3 if act == "tanh" and dtype == torch.bfloat16 else 2e-5
            assert float((got.double() - want).abs().max()) < bound
    assert ops.low_rank(x[:, :rank - 1], w[:, :rank - 1].contiguous()) is None


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,rank,n", [(300, 512, 130), (700, 48, 200), (1025, 8, 64)])
def test_low_rank_at_its_limits(ops, T, rank, n, dtype):
    gen = torch.Generator().manual_seed(rank)
    x = torch.randn(T, rank, generator=gen).to(DEV)
    w = (torch.randn(n, rank, generator=gen) / rank ** 0.5).to(dtype).to(DEV)
    want = x.to(dtype).double() @ w.double().T
    # 2^-24 * 0.41 * |x||w| in the root mean square for terms added one by one (|w| near one)
    assert float(((ops.low_rank(x, w).double() - want).abs() / x.double().norm(dim=1)[:, None]).max()) \
        < 3 * 2.0 ** -24 * float(w.double().norm(dim=1).max())


@pytest.mark.parametrize("T", [1, 8, 9, 16])
def test_several_products_in_one_launch(ops, T):
    gen = torch.Generator().manual_seed(T)
    sizes = [(128, 40), (128, 16), (256, 7), (64, 300), (128, 33), (72, 64)]
    pairs = [(torch.randn(T, k, generator=gen).to(torch.bfloat16).to(DEV),
              torch.randn(n, k, generator=gen).to(torch.bfloat16).to(DEV)) for k, n in sizes]
    for count in range(1, 7):
        assert ops.skinny_many_fits(pairs[:count])
        for (x, w), out in zip(pairs, ops.gemm_skinny_many(pairs[:count])):
            want = x.double() @ w.double().T
            size = x.double().abs() @ w.double().abs().T
            assert bool(((out.double() - want).abs() <= x.shape[1] * 2.0 ** -23 * size).all())
    assert not ops.skinny_many_fits(pairs + pairs[:1])


def test_zero_rows(ops):
    """Rows of several tensors, types and alignments, more than fit one launch; nothing beside them."""
    held = [torch.ones(3, n, dtype=d, device=DEV) for n, d in
            [(1, torch.float32), (7, torch.bfloat16), (4096, torch.float32), (100001, torch.bfloat16)] * 9]
    ops.zero_rows([t[1] for t in held])
    for t in held:
        assert bool((t[1] == 0).all()) and bool((t[0] == 1).all()) and bool((t[2] == 1).all())


def sigmoid64(x):
    return torch.sigmoid(x.double())


@pytest.mark.parametrize("mode,H,rep,dim,vdim,per_head", [
    ("delta", 4, 2, 64, 64, False), ("delta", 3, 1, 128, 128, False), ("delta", 2, 1, 30, 8, True),
    ("delta", 2, 2, 100, 32, True), ("delta", 2, 1, 61, 256, False), ("wkv", 4, 1, 64, 64, False),
    ("wkv", 2, 1, 128, 128, False), ("wkv", 3, 1, 16, 16, False)])
@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_state_step(ops, mode, H, rep, dim, vdim, per_head, form, dtype):
    """A token's decays, step, norm and gate in one kernel against float64. Every 32-bit sum here has up
    to `dim` terms, each off by at most dim * 2^-24 of the magnitudes; the norm makes them of order one
    and adds a few roundings: 64 + dim of them bound the state and the output (bfloat16: its own half
    place, 2^-9, on top)."""
    n, slots_n, n_decay = 3, 5, H if per_head else H * dim
    rnd = lambda *s, seed: torch.randn(*s, generator=torch.Generator().manual_seed(seed)).to(DEV)  # noqa: E731
    slots = [4, 0, 2]
    q, k = rnd(n, H // rep * dim + 3, seed=1), rnd(n, H // rep * dim, seed=2) * dim ** -0.5
    v, gate = rnd(n, H * vdim, seed=3), rnd(n, H * vdim + 5, seed=4)
    raw, beta = rnd(n, n_decay, seed=5), rnd(n, H, seed=6)
    A, bias = rnd(H, seed=7) * 0.3, rnd(n_decay, seed=8)
    bonus, wide_norm = rnd(H, dim, seed=9), mode == "wkv"
    norm = 1 + 0.1 * rnd(H * vdim if wide_norm else vdim, seed=10)
    g = torch.sigmoid(raw) if form == 0 else raw
    rows = rnd(slots_n, 4 + H * dim * vdim, seed=11)
    before = rows.clone()
    state = ops.StateRows(rows, [("front", 4), ("S", H * dim * vdim)])
    as_int = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    ctx = types.SimpleNamespace(is_decode=True, n_seqs=n, cu_tokens=as_int([0, 1, 2, 3]), slots=as_int(slots))
    which = ops.SCAN_DELTA if mode == "delta" else ops.SCAN_WKV
    assert ops.state_step_fits(ctx, which, state, "S", dim, vdim)
    out = torch.empty(n, H * vdim, dtype=dtype, device=DEV)
    act = "sigmoid" if mode == "delta" else "silu"
    ops.state_step(ctx, which, q, k, v, g, None if form == 0 else (A if form == 1 else None, bias), state,
                   "S", norm, gate, act, 1e-5, out, H, rep, dim, vdim, beta=beta, bonus=bonus,
                   decay_per_head=per_head)
    d64 = g.double()
    if form == 1:
        each = A.double() if per_head else A.double().repeat_interleave(dim)
        d64 = torch.exp(-torch.exp(each) * torch.nn.functional.softplus(d64 + bias.double()))
    if form == 2:
        d64 = torch.exp(-torch.exp(d64 + bias.double()))
    room = (64 + dim) * 2.0 ** -24
    for i in range(n):
        S0 = before[slots[i], 4:].double().view(H, dim, vdim)
        for h in range(H):
            S, a = S0[h], (h // rep) * dim
            qq, kk = q[i, a:a + dim].double(), k[i, a:a + dim].double()
            vv = v[i, h * vdim:(h + 1) * vdim].double()
            gg = d64[i, h] if per_head else d64[i, h * dim:(h + 1) * dim, None]
            if mode == "delta":
                new = gg * S
                new = new + kk[:, None] * (sigmoid64(beta[i, h]) * (vv - kk @ new))
                o, size = qq @ new, qq.abs() @ new.abs()
            else:
                kv = kk[:, None] * vv
                o = qq @ (S + bonus[h].double()[:, None] * kv)
                size = qq.abs() @ (S.abs() + (bonus[h].double()[:, None] * kv).abs())
                new = gg * S + kv
            got = rows[slots[i], 4 + h * dim * vdim:4 + (h + 1) * dim * vdim].double().view(dim, vdim)
            assert float((got - new).abs().max()) <= room * float(S.abs().max() + vv.abs().max()) * 4
            scale = 1 / torch.sqrt((o * o).mean() + 1e-5)
            z = gate[i, h * vdim:(h + 1) * vdim].double()
            z = torch.sigmoid(z) if act == "sigmoid" else z * torch.sigmoid(z)
            w = (norm[h * vdim:(h + 1) * vdim] if wide_norm else norm).double() * z
            want = o * scale * w
            bound = room * (size * scale * w.abs() + want.abs() * (1 + size.max() * scale))
            if dtype == torch.bfloat16:
                bound = bound + want.abs() * 2.0 ** -8
            assert bool(((out[i, h * vdim:(h + 1) * vdim].double() - want).abs() <= bound + 1e-7).all())
    untouched = [s for s in range(slots_n) if s not in slots]
    assert torch.equal(rows[untouched], before[untouched]) and torch.equal(rows[:, :4], before[:, :4])


def test_state_step_with_no_epsilon(ops):
    """What the kernels that it takes the place of took: a norm without a constant in its root."""
    n, H, dim, vdim = 2, 3, 64, 64
    rnd = lambda *s, seed: torch.randn(*s, generator=torch.Generator().manual_seed(seed)).to(DEV)  # noqa: E731
    as_int = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    ctx = types.SimpleNamespace(is_decode=True, n_seqs=n, cu_tokens=as_int([0, 1, 2]), slots=as_int([1, 0]))
    q, k, v, gate, g = (rnd(n, H * dim, seed=s) for s in range(5))
    args = (q, k, v, torch.sigmoid(g), None)
    outs = []
    for eps in (0.0, 1e-12):
        state = ops.StateRows(rnd(2, H * dim * vdim, seed=9), [("S", H * dim * vdim)])
        out = torch.empty(n, H * vdim, device=DEV)
        ops.state_step(ctx, ops.SCAN_WKV, *args, state, "S", torch.ones(vdim, device=DEV), gate, "silu", eps, out,
                       H, 1, dim, vdim, bonus=rnd(H, dim, seed=7))
        outs.append(out)
    assert torch.allclose(*outs, rtol=1e-6) and bool(outs[0].isfinite().all())


@pytest.mark.parametrize("W", [4, 100, 1024, 1028, 2048, 3072, 4100, 8192, 8196])
@pytest.mark.parametrize("has_y,norm_y,has_out", [(1, 1, 1), (1, 0, 1), (0, 0, 1), (1, 1, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_layer_norms_around_a_sum(ops, W, has_y, norm_y, has_out, dtype):
    """Rows at the edges of what a block's threads hold, against float64: sums of W terms in 32 bits
    (W * 2^-24 of them at worst, sqrt(W) of order), 16 roundings besides, and bfloat16's half place."""
    T = 3
    rnd = lambda *s, seed: torch.randn(*s, generator=torch.Generator().manual_seed(seed)).to(DEV)  # noqa: E731
    resid, y = rnd(T, W, seed=1) + 0.5, (rnd(T, W, seed=2) * 3 - 1).to(dtype)
    w1, b1, w2, b2 = (rnd(W, seed=s) for s in (3, 4, 5, 6))
    norm = lambda x, w, b: (x - x.mean(-1, keepdim=True)) / torch.sqrt(  # noqa: E731
        x.var(-1, unbiased=False, keepdim=True) + 1e-5) * w.double() + b.double()
    want = resid.double()
    if has_y:
        want = want + (norm(y.double(), w1, b1) if norm_y else 0.7 * y.double())
    pending = types.SimpleNamespace(values=y, weight=w1 if norm_y else None, bias=b1 if norm_y else None,
                                    eps=1e-5, scale=1.0 if norm_y else 0.7) if has_y else None
    out = torch.empty(T, W, dtype=dtype, device=DEV) if has_out else None
    ops.ln_add_ln(resid, pending, w2 if has_out else None, b2 if has_out else None, 1e-5, out)
    room = (16 + 2 * W ** 0.5) * 2.0 ** -24
    assert float((resid.double() - want).abs().max()) <= room * float(want.abs().max() + 4)
    if has_out:
        end = norm(want, w2, b2)
        slack = 0 if dtype == torch.float32 else 2.0 ** -8
        assert bool(((out.double() - end).abs() <= room * 16 + slack * end.abs() + 16 * room * end.abs()).all())


@pytest.mark.parametrize("W", [2, 250, 2048])
def test_embedding_with_sines_and_cosines(ops, W):
    """Both of a pair from one thread; positions far out keep their 32 bits."""
    table, ids = torch.randn(7, W, generator=torch.Generator().manual_seed(1)).to(DEV), [0, 6, 3, 9, -1]
    positions = [0, 1, 77, 131071, 5]
    freq = torch.pow(10000.0, -2.0 * torch.arange(W // 2, dtype=torch.float64) / W).to(DEV)
    out, copy = (torch.empty(5, W, device=DEV) for _ in range(2))
    as_int = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    ops.embed_sinusoid(table, as_int(ids), as_int(positions), freq, 1.5, out, copy)
    angle = torch.tensor(positions, dtype=torch.float64, device=DEV)[:, None] * freq
    pe = torch.stack([angle.sin(), angle.cos()], -1).flatten(1).float()
    rows = torch.stack([table[i] * 1.5 if 0 <= i < 7 else torch.zeros(W, device=DEV) for i in ids])
    # the sine's own rounding and the sum's: half a place each of numbers up to 1 and 8
    assert float((out - (rows + pe)).abs().max()) <= 2.0 ** -24 + 2.0 ** -21 and torch.equal(out, copy)


@pytest.mark.parametrize("T,n,per_head", [(1, 5, 1), (3, 32, 1), (9, 33, 11), (130, 300, 100), (5, 2048, 64)])
@pytest.mark.parametrize("with_A", [True, False])
def test_decays(ops, T, n, per_head, with_A):
    """Channels and tokens at the edges of a block's, from a wider row and in place, against float64: the
    exponent is off by a few roundings of its own size (up to 30), and so is the decay, relatively."""
    rnd = lambda *s, seed: torch.randn(*s, generator=torch.Generator().manual_seed(seed)).to(DEV)  # noqa: E731
    wide, bias, A = rnd(T, n + 3, seed=1) * 2, rnd(n, seed=2), rnd(-(-n // per_head), seed=3) * 0.5
    z = wide[:, :n].double() + bias.double()
    steps = torch.empty(T, n, device=DEV) if with_A else None
    out = torch.empty(T, n, device=DEV)
    ops.decay_gate(wide[:, :n], per_head, bias, A if with_A else None, out=out, steps=steps)
    if with_A:
        soft = torch.nn.functional.softplus(z)
        want = torch.exp(-torch.exp(A.double()).repeat_interleave(per_head)[:n] * soft)
        assert float((steps.double() - soft).abs().max()) <= 16 * 2.0 ** -24 * float(soft.max() + 1)
    else:
        want = torch.exp(-torch.exp(z))
    room = 16 * 2.0 ** -24 * (1 + want.clamp_min(1e-30).log().abs())
    assert bool(((out.double() - want).abs() <= room * want + 1e-37).all())
    own = wide[:, :n].contiguous()
    ops.decay_gate(own, per_head, bias, A if with_A else None)
    assert torch.equal(own, out)


@pytest.mark.parametrize("H,G,dim,vdim", [(32, 8, 64, 64), (24, 8, 128, 128), (3, 1, 20, 12), (32, 16, 128, 128),
                                          (3, 1, 10, 6), (40, 8, 128, 128)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_query_and_key_norms_into_the_cache(ops, H, G, dim, vdim, dtype):
    """Rows in registers and, for sizes those do not take, by elements; a padding token writes no cache. A
    norm's sum of n squares is off by at most n * 2^-24 of itself, its root by half of that; eight
    roundings besides, and bfloat16's half place."""
    T, nq, nk, nv = 3, H * dim, G * dim, G * vdim
    rnd = lambda *s, seed: torch.randn(*s, generator=torch.Generator().manual_seed(seed)).to(DEV)  # noqa: E731
    qkv = rnd(T, nq + nk + nv + 4, seed=1)
    wq, wk = rnd(nq, seed=2), rnd(nk, seed=3)
    k, v = torch.full((4, G, 64, dim), 7.0, device=DEV, dtype=dtype), torch.full((4, G, 64, vdim), 7.0, device=DEV, dtype=dtype)
    as_int = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    table, seqs, pos = as_int([[2, 0], [3, 1]]), [0, -1, 1], [63, 0, 70]
    q_out = torch.empty(T, nq, device=DEV, dtype=dtype)
    ops.qk_norm_cache_write(qkv, q_out, wq, wk, 1e-5, as_int(pos), as_int(seqs), table, k, v, H, G, dim, vdim)
    norm = lambda x, w: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double()  # noqa: E731
    x = qkv.double()
    room = (8 + nq / 2) * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)

    def close(got, want):
        assert bool(((got.double() - want).abs() <= room * want.abs() + 1e-30).all())
    close(q_out, norm(x[:, :nq], wq))
    keys, values = norm(x[:, nq:nq + nk], wk), x[:, nq + nk:nq + nk + nv]
    seen = torch.zeros(4, 64, dtype=torch.bool, device=DEV)
    for t in (0, 2):
        page, r = int(table[seqs[t], pos[t] // 64]), pos[t] % 64
        close(k[page, :, r].flatten(), keys[t])
        close(v[page, :, r].flatten(), values[t])
        seen[page, r] = True
    assert bool((k.transpose(1, 2)[~seen] == 7).all()) and bool((v.transpose(1, 2)[~seen] == 7).all())
