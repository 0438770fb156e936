"""Loss and gradients of the proposal's training step at the edges of its tiles: 128-point tiles of the
layers (one per CTA, 152 CTAs, then a second tile), 64-point chunks of the weight gradients and their
shares, zero rows past a ragged end, and weights that do not start on a 16-byte boundary.

Bars, against the float64 oracle that rounds the same operands to bfloat16: the loss within 1e-5 (float32
sums of values near 1), each gradient block within relative 2e-3 (a bfloat16 operand is half an ulp, 2^-9 of
one element, off when float32 and float64 round to different sides; under 1 in 100 elements do).
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(net, n, seed):
    from oracle import mlp as om

    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 2, (n, 3))
    y = (rng.uniform(size=n) < 0.5).astype(np.float32)
    net.grad.zero_()
    loss = torch.zeros(1, device="cuda")
    net.backward(torch.as_tensor(x, device="cuda"), torch.as_tensor(y, device="cuda"), loss)
    assert int(net.status.cpu()[0]) == 0
    grad = om.unflatten(net.grad.cpu().numpy())
    ref_loss, ref = om.loss_and_grad(net.params(), x, y, net.freq.cpu().numpy())
    assert abs(loss.item() - ref_loss) < 1e-5 * max(1.0, ref_loss)
    for k in ref:
        assert np.linalg.norm(grad[k] - ref[k]) <= 2e-3 * max(np.linalg.norm(ref[k]), 1e-30), k


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 191, 2047, 152 * 128 + 1, 65536])
def test_training_rows_match_oracle(n):
    from kups_gb300.mlp import LearnedInsertionProposal

    _check(LearnedInsertionProposal(seed=6, grid=16), n, n)


def test_training_rows_with_weights_off_a_16_byte_boundary():
    from kups_gb300.mlp import LearnedInsertionProposal

    net = LearnedInsertionProposal(seed=7, grid=16)
    for name, field in (("param_bf16", "param_bf16"), ("param_bf16_t", "param_bf16_t"), ("grad", "grad")):
        old = getattr(net, name)
        moved = torch.empty(old.numel() + 1, dtype=old.dtype, device="cuda")[1:]
        moved.copy_(old)
        setattr(net, name, moved)
        setattr(net.net, field, moved.data_ptr())
    _check(net, 777, 8)
