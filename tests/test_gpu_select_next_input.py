"""Token selection that also leaves the tokens as the next step's input: the row's last block
merges, against the two-kernel form."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [100, 16383, 16384, 40001, 131072])
@pytest.mark.parametrize("n", [1, 7, 48])
def test_same_tokens_in_both_places(n, V):
    from foundry_b200.kernels import ops
    gen = torch.Generator().manual_seed(n + V)
    logits = torch.randn(n, V, generator=gen).cuda()
    logits[0, V // 2:] = 9.0                     # ties: the first of them
    logits[n - 1] = float("nan") if n > 1 else logits[n - 1]
    heat = torch.tensor([0.7 * (i % 3 == 1) for i in range(n)], device="cuda")
    streams = torch.arange(n, device="cuda") * 7919
    steps = torch.arange(n, device="cuda")
    new = lambda: torch.full((n,), -1, dtype=torch.int32, device="cuda")  # noqa: E731
    want = ops.select_tokens(logits, new(), heat, streams, steps)
    with ops.scratch_owner(("test", n, V)):
        for _ in range(3):  # the rows' counters are left as they were found
            also = new()
            got = ops.select_tokens(logits, new(), heat, streams, steps, also=also)
            assert torch.equal(got, want) and torch.equal(also, want)
    ops.release_scratch(("test", n, V))
