"""The delta rule in chunks of 32 tokens (csrc/chunk_scan.cu) against the rule token by token in
float64: sizes, decays a head and a channel, sequences that end inside a chunk or lie side by side,
steps worked in parts, states that nobody else may touch."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from foundry_b200.kernels import ops as o
    return o


def plain(q, k, v, g, beta, S):
    """One sequence: q, k [T, H, d]; v [T, H, e]; g [T, H, d or 1]; beta [T, H]; S [H, d, e]."""
    out = []
    for t in range(q.shape[0]):
        S = S * g[t, :, :, None]
        u = torch.sigmoid(beta[t])[:, None] * (v[t] - torch.einsum("hd,hde->he", k[t], S))
        S = S + k[t, :, :, None] * u[:, None]
        out.append(torch.einsum("hd,hde->he", q[t], S))
    return torch.stack(out), S


def run(ops, lens, H, G, d, e, channels, decay, seed=0, nan_at=None, padding=0):
    gen = torch.Generator().manual_seed(seed)
    T, n = sum(lens) + padding, len(lens)
    wide = torch.randn(T, 2 * G * d + H * e, generator=gen).to(DEV)  # q | k | v of one product
    for a in (0, G * d):
        part = wide[:, a:a + G * d].view(T, G, d)
        part /= part.norm(dim=-1, keepdim=True)
    if nan_at is not None:
        wide[nan_at] = float("nan")
    g = decay(torch.rand(T, H * d if channels else H, generator=gen)).to(DEV)
    beta = torch.randn(T, H + 3, generator=gen).to(DEV)[:, 3:]
    slots = torch.randperm(n + 2, generator=gen)[:n]
    rows = (0.3 * torch.randn(n + 3, 4 + H * d * e, generator=gen)).to(DEV)
    before = rows.clone()
    cu = [0]
    for x in lens:
        cu.append(cu[-1] + x)
    ctx = types.SimpleNamespace(
        is_decode=False, n_seqs=n, max_q_len=max(lens), slots=slots.to(torch.int32).to(DEV),
        cu_tokens=torch.tensor(cu, dtype=torch.int32, device=DEV))
    state = ops.StateRows(rows, [("tail", 4), ("S", H * d * e)])
    out = torch.full((T, H * e), 9.0, device=DEV)
    q, k, v = wide, wide[:, G * d:], wide[:, 2 * G * d:]
    assert ops.chunk_scan_unit(ctx, ops.SCAN_DELTA, T, H, d, e, (q, k, out), state, "S") > 0
    ops.state_scan(ctx, ops.SCAN_DELTA, q, k, v, g, state, "S", out, H, H // G, d, e, beta=beta,
                   decay_per_head=not channels)
    heads = [wide[:, a:a + G * d].double().view(T, G, d).repeat_interleave(H // G, 1)
             for a in (0, G * d)]
    values = wide[:, 2 * G * d:].double().view(T, H, e)
    want, states = [], before[:, 4:].double().view(n + 3, H, d, e).clone()
    for s, a, b in zip(slots.tolist(), cu, cu[1:]):
        if a == b:
            continue
        part, states[s] = plain(heads[0][a:b], heads[1][a:b], values[a:b],
                                g[a:b].double().view(b - a, H, -1), beta[a:b].double(), states[s])
        want.append(part)
    assert torch.equal(rows[:, :4], before[:, :4])
    assert bool((out[cu[-1]:] == 9.0).all())  # padding rows stay as they were
    return out[:cu[-1]].double().view(-1, H, e), torch.cat(want), rows[:, 4:].double().view_as(states), states


def near(a, b):
    # sums of up to 128 + 32 products and a substitution of 32 steps, each off by 2^-24 of its
    # terms: about sqrt(32) * 2^-24 = 3.4e-7 in the 2-norm where they are off independently
    assert float((a - b).norm() / b.norm()) < 1e-6


DECAYS = {"slow": lambda x: 1.0 - 0.05 * x, "any": lambda x: torch.exp(-torch.exp(8.0 * x - 5.0)),
          "gone": lambda x: torch.where(x < 0.3, 0.0, x)}


@pytest.mark.parametrize("decay", list(DECAYS))
@pytest.mark.parametrize("channels", [False, True])
@pytest.mark.parametrize("H,G,d,e", [(4, 2, 64, 64), (2, 2, 128, 128), (3, 1, 64, 16), (2, 1, 128, 48)])
def test_chunks_equal_token_by_token(ops, H, G, d, e, channels, decay):
    for lens in ([97], [128], [300, 96, 161]):
        out, want, rows, states = run(ops, lens, H, G, d, e, channels, DECAYS[decay], seed=d + e)
        near(out, want)
        near(rows, states)  # every slot's: the sequences' moved on, the others as they were


@pytest.mark.parametrize("H,G,d,e", [(24, 24, 128, 128), (60, 30, 128, 48), (28, 28, 128, 112), (40, 20, 64, 64)])
def test_blocks_of_24_columns(ops, H, G, d, e):
    """Heads whose blocks of 16 columns are more than the SMs, those of 24 are not; the last block of a
    head has 8, 24 or 16 columns."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if not H * (e // 16) > sms >= H * -(-e // 24):
        pytest.skip("another number of SMs")
    out, want, rows, states = run(ops, [131], H, G, d, e, True, DECAYS["slow"], seed=e)
    near(out, want)
    near(rows, states)


@pytest.mark.parametrize("room", [1, 2, 5])
def test_steps_in_parts(ops, room, monkeypatch):
    """A workspace of so many chunks: parts that begin and end inside sequences."""
    unit = ops._fn("fb_chunk_scan_unit")(2, 64, 32)
    monkeypatch.setattr(ops, "CHUNK_SCAN_ROOM", room * unit)
    out, want, rows, states = run(ops, [200, 96, 130], 2, 1, 64, 32, True, DECAYS["any"])
    near(out, want)
    near(rows, states)


def test_parts_do_not_change_the_numbers(ops, monkeypatch):
    whole, _, moved, _ = run(ops, [200, 96, 130], 2, 1, 64, 32, True, DECAYS["any"])
    monkeypatch.setattr(ops, "CHUNK_SCAN_ROOM", 3 * ops._fn("fb_chunk_scan_unit")(2, 64, 32))
    out, _, rows, _ = run(ops, [200, 96, 130], 2, 1, 64, 32, True, DECAYS["any"])
    assert torch.equal(out, whole) and torch.equal(rows, moved)


def test_no_memory_for_the_chunks(ops, monkeypatch):
    """Token by token, then."""
    monkeypatch.setattr(ops, "_chunk_workspace", lambda *a: None)
    out, want, rows, states = run(ops, [200, 96], 2, 1, 64, 32, True, DECAYS["any"])
    near(out, want)
    near(rows, states)


def test_a_later_token_that_is_no_number_does_not_reach_earlier_ones(ops):
    out, want, _, _ = run(ops, [128], 2, 2, 64, 64, True, DECAYS["slow"], nan_at=70)
    assert bool(torch.isfinite(out[:70]).all()) and bool(torch.isnan(out[70:]).all())
    near(out[:70], want[:70])


def test_what_the_delta_rule_does_not_take_is_refused(ops):
    """A constant on the outputs, or no step sizes: the same for chunks as token by token."""
    H, d, T = 2, 64, 128
    x, g = torch.randn(T, H * d, device=DEV), torch.rand(T, H * d, device=DEV)
    beta, out = torch.randn(T, H, device=DEV), torch.empty(T, H * d, device=DEV)
    state = ops.StateRows(torch.zeros(1, H * d * d, device=DEV), [("S", H * d * d)])
    ctx = types.SimpleNamespace(is_decode=False, n_seqs=1, max_q_len=T,
                                slots=torch.zeros(1, dtype=torch.int32, device=DEV),
                                cu_tokens=torch.tensor([0, T], dtype=torch.int32, device=DEV))
    for more in (dict(beta=beta, out_scale=2.0), dict(beta=None)):
        with pytest.raises(ops.KernelError, match="state_scan"):
            ops.state_scan(ctx, ops.SCAN_DELTA, x, x, x, g, state, "S", out, H, 1, d, d, **more)


def test_many_sequences_in_parts(ops, monkeypatch):
    """More than a warp's lanes of sequences: the search for a chunk's sequence and the count of the
    chunks in front of one go on for a second round."""
    gen = torch.Generator().manual_seed(4)
    lens = torch.randint(100, 220, (40,), generator=gen).tolist()
    monkeypatch.setattr(ops, "CHUNK_SCAN_ROOM", 37 * ops._fn("fb_chunk_scan_unit")(2, 64, 16))
    out, want, rows, states = run(ops, lens, 2, 1, 64, 16, True, DECAYS["any"])
    near(out, want)
    near(rows, states)


@pytest.mark.parametrize("lens,padding", [([300, 0, 161, 0], 51), ([0, 0, 400], 1), ([129] + [0] * 3, 255),
                                          ([0] * 33 + [6200] + [0] * 5, 120)])
def test_empty_sequences_and_padding_tokens(ops, lens, padding):
    """A replayed step's form: sequences without tokens, and tokens behind the last sequence."""
    out, want, rows, states = run(ops, lens, 2, 1, 64, 32, False, DECAYS["slow"], padding=padding)
    near(out, want)
    near(rows, states)


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("H,d,e", [(2, 64, 64), (3, 128, 40), (4, 16, 24), (1, 256, 20)])
def test_wkv_over_prompts(ops, H, d, e, per_head):
    """The recurrence with a bonus, its tokens in chunks where the decay is a channel's, token by
    token where it is a head's: o = q . (S + bonus k v), S <- g S + k v."""
    gen = torch.Generator().manual_seed(d + e)
    lens = [300, 7, 129]
    T, n = sum(lens), len(lens)
    q, k, v = (torch.randn(T, H * x, generator=gen).to(DEV) for x in (d, d, e))
    g = torch.exp(-torch.exp(torch.randn(T, H if per_head else H * d, generator=gen) - 3)).to(DEV)
    bonus = torch.randn(H, d, generator=gen).to(DEV)
    rows = (0.3 * torch.randn(n, H * d * e, generator=gen)).to(DEV)
    states = rows.double().view(n, H, d, e).clone()
    cu = [0, 300, 307, 436]
    ctx = types.SimpleNamespace(is_decode=False, n_seqs=n, max_q_len=300,
                                slots=torch.arange(n, dtype=torch.int32, device=DEV),
                                cu_tokens=torch.tensor(cu, dtype=torch.int32, device=DEV))
    out = torch.empty(T, H * e, device=DEV)
    ops.state_scan(ctx, ops.SCAN_WKV, q, k, v, g, ops.StateRows(rows, [("S", H * d * e)]), "S", out, H, 1, d,
                   e, bonus=bonus, decay_per_head=per_head)
    want = []
    for s, a, b in zip(range(n), cu, cu[1:]):
        for t in range(a, b):
            kv = k[t].double().view(H, d, 1) * v[t].double().view(H, 1, e)
            want.append(torch.einsum("hd,hde->he", q[t].double().view(H, d),
                                     states[s] + bonus.double()[:, :, None] * kv).flatten())
            states[s] = states[s] * g[t].double().view(H, -1, 1) + kv
    near(out.double(), torch.stack(want))
    near(rows.double().view_as(states), states)
