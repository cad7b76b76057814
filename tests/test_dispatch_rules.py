"""Which kernel a call goes to: rules that read shapes, strides and counts alone, so that tensors on
the CPU show them."""
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
