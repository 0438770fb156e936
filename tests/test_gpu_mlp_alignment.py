"""Weights that do not start on a 16-byte boundary: the forward pass and the grid give the bits of aligned ones."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 70000])
def test_forward_and_grid_with_weights_off_a_16_byte_boundary(n):
    from kups_gb300.mlp import LearnedInsertionProposal

    net = LearnedInsertionProposal(seed=7, grid=16)
    x = torch.rand((n, 3), generator=torch.Generator("cuda").manual_seed(n), dtype=torch.float64, device="cuda")
    want = [net.forward(x)] + [t.clone() for t in net.build_grid()]
    for offset in (1, 4):
        moved = torch.empty(net.param_bf16.numel() + offset, dtype=torch.bfloat16, device="cuda")[offset:]
        moved.copy_(net.param_bf16)
        net.net.param_bf16 = moved.data_ptr()
        for got, ref in zip([net.forward(x)] + list(net.build_grid()), want):
            assert torch.equal(got, ref)
