"""Which kernel a call goes to: rules that read shapes, strides and counts alone, so that tensors on
the CPU show them."""
import types

import pytest
import torch

from foundry_b200.kernels import ops


def test_router_kernel_takes_rows_of_the_routers_width_only():
    """The kernel walks the rows' width in both operands: another one is the product's to refuse."""
    x = torch.zeros(100, 128, dtype=torch.bfloat16)
    router = torch.zeros(8, 128, dtype=torch.bfloat16)
    assert ops.moe_router_fits(x, router)
    for width in (64, 192, 256):
        other = torch.zeros(8, width, dtype=torch.bfloat16)
        assert not ops.moe_router_fits(x, other)
        chosen, weights = torch.zeros(100, 2, dtype=torch.int32), torch.zeros(100, 2)
        with pytest.raises(ops.KernelError, match="router"):
            ops.moe_router_sorted(x, other, None, 2, chosen, weights, 8)
    with pytest.raises(ops.KernelError, match="choices"):
        ops.moe_router_sorted(x, router, None, 2, torch.zeros(99, 2, dtype=torch.int32),
                              torch.zeros(99, 2), 8)


def rows_of(T, H=3, k1=64, k2=32, e=64):
    bf = dict(dtype=torch.bfloat16)
    return [torch.zeros(T, H * (k1 + k2), **bf), torch.zeros(T, H * e, **bf), torch.zeros(T, H, k1, **bf),
            torch.zeros(T, k2, **bf), torch.zeros(T, H, e, **bf)]


def rows_step(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return types.SimpleNamespace(n_seqs=len(lens), cu_tokens_host=cu)


def test_rows_attention_on_tensor_maps_takes_heads_side_by_side_only():
    T, ctx = 96, rows_step([96])
    q, out, k, shared, v = rows_of(T)
    assert ops._tc_rows_blocks(ctx, q, out, k, shared, v, 64, 32, 64, 0.0) == 1
    for other in (dict(k=k[:, :1].expand(T, 3, 64)), dict(v=v[:, :1].expand(T, 3, 64)),
                  dict(shared=shared[:1].expand(T, 32)), dict(k=k[:1].expand(T, 3, 64)),
                  dict(v=torch.zeros(3, T, 64, dtype=torch.bfloat16).transpose(0, 1)),
                  dict(k=torch.zeros(T, 96, dtype=torch.bfloat16).as_strided((T, 3, 64), (96, 16, 1)))):
        args = dict(dict(k=k, shared=shared, v=v), **other)
        assert ops._tc_rows_blocks(ctx, q, out, args["k"], args["shared"], args["v"], 64, 32, 64, 0.0) == 0


@pytest.mark.parametrize("lens,k64,k128", [
    ([64], 1, 1), ([63], 0, 0), ([129, 1, 63], 4, 4), ([70] * 8, 8, 8), ([64] * 16, 16, 16),
    ([64] * 64, 0, 64), ([64] + [8] * 31, 0, 0), ([64] + [16] * 15, 0, 16), ([200] + [5] * 7, 0, 9),
    ([1000] + [5] * 15, 23, 23)])
def test_rows_attention_on_tensor_maps_by_tokens_a_sequence(lens, k64, k128):
    """The same for a plain step and for the padded one that replays it."""
    from foundry_b200.engine.decode import bucket_of
    from foundry_b200.engine.prompt import token_bucket
    T = sum(lens)
    for k1, want in ((64, k64), (128, k128)):
        args = (k1, 32, 64, 0.0)
        assert ops._tc_rows_blocks(rows_step(lens), *rows_of(T, k1=k1), *args) == want
        t, n = token_bucket(T), bucket_of(len(lens))
        replay = types.SimpleNamespace(n_seqs=n, cu_tokens_host=None, query_blocks_bound=(t + 63) // 64 + n,
                                       long_queries=max(lens) >= 64)
        assert (ops._tc_rows_blocks(replay, *rows_of(t, k1=k1), *args) > 0) == (want > 0)


@pytest.mark.parametrize("H,dim,vdim,lens,chunks", [
    (32, 64, 64, [128], True), (32, 64, 64, [95], True), (32, 64, 64, [64], False), (32, 64, 64, [200] * 4, True),
    (32, 64, 64, [200] * 5, False), (4, 64, 64, [200] * 32, True), (4, 64, 64, [200] * 33, False),
    (32, 64, 128, [200] * 16, True), (24, 128, 128, [100] * 16, True), (24, 128, 48, [100] * 16, False)])
def test_delta_rule_in_chunks_by_tokens_and_heads(H, dim, vdim, lens, chunks, monkeypatch):
    """The same for a plain step and for the padded one that replays it."""
    from foundry_b200.engine.decode import bucket_of
    from foundry_b200.engine.prompt import token_bucket
    monkeypatch.setattr(ops, "_fn", lambda name: lambda h, d, e: 1)
    for T, n in ((sum(lens), len(lens)), (token_bucket(sum(lens)), bucket_of(len(lens)))):
        state = ops.StateRows(torch.zeros(1, 4), [("S", 4)])
        ctx = types.SimpleNamespace(is_decode=False, n_seqs=n)
        rows = [torch.zeros(1, 4)]
        assert bool(ops.chunk_scan_unit(ctx, ops.SCAN_DELTA, T, H, dim, vdim, rows, state, "S")) == chunks


@pytest.mark.parametrize("free,room", [(10 ** 9, 5), (45, 3), (25, 2), (15, 1), (5, None)])
def test_workspace_of_the_chunks_fits_the_memory_there_is(free, room, monkeypatch):
    """Fewer chunks at a time where memory is short; token by token where there is none for one."""
    asked = []

    def empty(count, **kw):
        asked.append(count)
        if count > free:
            raise torch.cuda.OutOfMemoryError("no room")
        return [0.0] * count

    monkeypatch.setattr(ops.torch, "empty", empty)
    got = ops._chunk_workspace(10, 5, "cuda")
    assert got is None if room is None else (len(got[0]), got[1]) == (10 * room, room)
    assert asked == sorted(asked, reverse=True)


@pytest.mark.parametrize("more", [dict(A=torch.zeros(3), per_head=4), dict(A=torch.zeros(16), per_head=0),
                                  dict(bias=torch.zeros(15)), dict(A=torch.zeros(16), bias=None)])
def test_decays_that_do_not_cover_the_channels_are_refused(more):
    args = dict(dict(bias=torch.zeros(16)), **more)
    with pytest.raises(ops.KernelError, match="low_rank"):
        ops.low_rank(torch.zeros(5, 8), torch.zeros(16, 8), **args)


def test_low_rank_kernel_by_rank_tokens_and_type():
    """The same for a plain step and for the padded one that replays it."""
    from foundry_b200.engine.prompt import token_bucket
    for dtype, ranks, most in ((torch.bfloat16, (32, 48), 5000), (torch.bfloat16, (64,), 0),
                               (torch.bfloat16, (8, 512), 0), (torch.float32, (24, 8), 5000),
                               (torch.float32, (40,), 128), (torch.float32, (48,), 0)):
        for T in (1, 8, 100, 128, 129, 5000):
            assert ops.low_rank_pays(T, dtype, *ranks) == (T <= most)
            assert ops.low_rank_pays(token_bucket(T), dtype, *ranks) == (T <= most)


@pytest.mark.parametrize("rows,K,gated,form", [
    (127, 3072, True, 1), (128, 3072, True, 2), (128, 14336, True, 2), (199, 2048, False, 1),
    (200, 2048, False, 2), (500, 8192, False, 1), (600, 8192, False, 2)])
def test_form_of_the_experts_products_by_rows_an_expert(rows, K, gated, form):
    assert ops.grouped_form(16 * rows, 16, K, gated) == form
