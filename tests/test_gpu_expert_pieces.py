"""The pieces around the routed experts' products: the router with its choice, the sort of the pairs,
gather and combine, at the edges of their warps' runs and blocks, against plain statements."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from foundry_b200.kernels import ops as o
    return o


@pytest.mark.parametrize("pairs", [1, 31, 32, 33, 1024, 1025, 5003])
@pytest.mark.parametrize("E,experts", [(1, 1), (16, 16), (20, 16), (256, 256)])
def test_sort_of_the_pairs(ops, pairs, E, experts):
    chosen = torch.randint(0, E, (pairs, 1), generator=torch.Generator().manual_seed(pairs),
                           dtype=torch.int32).to(DEV)
    order = ops.ExpertOrder(chosen, experts)
    flat = chosen.flatten().long().cpu()
    counts = torch.bincount(flat, minlength=E)[:experts]
    assert order.counts.cpu().tolist() == counts.tolist()
    assert order.starts.cpu().tolist() == [0] + counts.cumsum(0).tolist()
    listed = torch.argsort(flat, stable=True)
    listed = listed[flat[listed] < experts]
    assert order.pair_at.cpu()[:len(listed)].tolist() == listed.tolist()
    place = torch.full((pairs,), -1)
    place[listed] = torch.arange(len(listed))
    assert order.place.flatten().cpu().tolist() == place.tolist()


def test_choices_that_name_no_expert_have_no_place(ops):
    """Any number outside the experts, on either side of the table."""
    chosen = torch.tensor([[-2, 0], [-1, 3], [4, -2], [2, -2 ** 31], [3, 2 ** 31 - 1]],
                          dtype=torch.int32).to(DEV)
    order = ops.ExpertOrder(chosen, 4, sort=False)
    order.place.fill_(7)  # a place that would be read as a row
    ops._call("fb_moe_sort", chosen.data_ptr(), 10, 4, order.counts.data_ptr(), order.starts.data_ptr(),
              order.place.data_ptr(), order.pair_at.data_ptr(), ops._stream())
    assert order.place.cpu().tolist() == [[-1, 0], [-1, 2], [-1, -1], [1, -1], [3, -1]]
    assert order.pair_at.cpu().tolist()[:4] == [1, 6, 3, 8] and order.counts.cpu().tolist() == [1, 0, 1, 2]


@pytest.mark.parametrize("T", [1, 65, 70])
@pytest.mark.parametrize("W", [64, 1028, 70, 4120])
def test_gather_and_combine(ops, T, W):
    gen = torch.Generator().manual_seed(T + W)
    chosen = torch.randint(0, 6, (T, 3), generator=gen, dtype=torch.int32).to(DEV)
    order = ops.ExpertOrder(chosen, 4)  # experts 4 and 5: identities
    x = torch.randn(T, W, generator=gen).to(torch.bfloat16).to(DEV)
    n = int(order.starts[-1])
    rows = ops.moe_gather(x, order)
    assert torch.equal(rows[:n], x[order.pair_at[:n].long() // 3])
    y = torch.randn(T * 3, W, generator=gen).to(DEV)
    weights = torch.rand(T, 3, generator=gen).to(DEV)
    addend = torch.randn(T, W, generator=gen).to(DEV)
    for add, own in ((None, None), (addend, None), (addend, x)):
        out = torch.empty(T, W, device=DEV)
        ops.moe_combine(y, order, weights, out, addend=add, identity=own)
        place = order.place.long()
        none = torch.zeros(T, 1, W, dtype=torch.float64, device=DEV)
        picked = torch.where((place >= 0)[..., None], y.double()[place.clamp(min=0)],
                             none if own is None else own.double()[:, None])
        want = (weights.double()[..., None] * picked).sum(1) + (0 if add is None else add.double())
        assert float((out.double() - want).abs().max()) < 1e-5  # four terms of up to five


@pytest.mark.parametrize("T", [65, 80, 81])
@pytest.mark.parametrize("E,K", [(5, 64), (16, 1088), (32, 128), (64, 512)])
def test_router_with_its_choice(ops, T, E, K):
    gen = torch.Generator().manual_seed(E)
    x = torch.randn(T, K + 8, generator=gen).to(torch.bfloat16).to(DEV)[:, :K]
    router = (torch.randn(E, K, generator=gen) / K ** 0.5).to(torch.bfloat16).to(DEV)
    bias, correction = torch.randn(E, generator=gen).to(DEV), torch.randn(E, generator=gen).to(DEV)
    rules = [dict(score="softmax_chosen"), dict(score="sigmoid", correction=correction, normalise=True)]
    if E % 4 == 0:
        rules.append(dict(score="softmax", groups=4, keep=2, group_best=1, weight_scale=2.0))
    z = (x.double() @ router.double().T).float()
    assert ops.moe_router_fits(x, router)
    for rule in rules:
        got = [torch.empty((T, 2), dtype=d, device=DEV) for d in (torch.int32, torch.float32)]
        want = [torch.empty_like(t) for t in got]
        order = ops.moe_router_sorted(x, router, bias, 2, *got, E, **rule)
        ops.moe_route(z, bias, 2, *want, **rule)
        # logits of about one, sums of K products off by some 2^-24 of sqrt(K) of them: weights move
        # by as much, and two choices trade places only where they are that close
        same = (got[0] == want[0]).all(1)
        assert int((~same).sum()) <= 1
        assert float((got[1][same] - want[1][same]).abs().max()) < 1e-4
        assert int(order.counts.sum()) == 2 * T
