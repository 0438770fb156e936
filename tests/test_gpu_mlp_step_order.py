"""A training step's kernels start while their predecessors still run: an update and the gradients behind it,
launched without a synchronisation between them (on the default stream, on another one, and captured), against
the oracle on the updated parameters."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["default", "stream", "graph"])
@pytest.mark.parametrize("n", [1, 129, 152 * 128 + 1])
def test_update_and_gradients_back_to_back(how, n):
    from kups_gb300.mlp import LearnedInsertionProposal
    from oracle import mlp as om

    net = LearnedInsertionProposal(seed=9, grid=16)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 2, (n, 3))
    y = (rng.uniform(size=n) < 0.5).astype(np.float32)
    dx, dy = torch.as_tensor(x, device="cuda"), torch.as_tensor(y, device="cuda")
    net.backward(dx, dy)  # the workspace
    net.grad.zero_()
    before = net.param.clone()
    loss = torch.zeros(1, device="cuda")

    def step():
        net.backward(dx, dy)
        net.adam(0.02)
        net.backward(dx, dy, loss)
        net.backward(dx, dy)

    torch.cuda.synchronize()
    if how == "default":
        step()
    elif how == "stream":
        with torch.cuda.stream(torch.cuda.Stream()):
            step()
    else:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        graph.replay()
    torch.cuda.synchronize()
    assert int(net.status.cpu()[0]) == 0
    assert (net.param - before).abs().max().item() > 0.01
    grad = om.unflatten(net.grad.cpu().numpy())
    ref_loss, ref = om.loss_and_grad(net.params(), x, y, net.freq.cpu().numpy())
    assert abs(loss.item() - ref_loss) < 1e-5 * max(1.0, ref_loss)
    for k in ref:  # two gradients of the same parameters, each as close as a single one's test asks
        assert np.linalg.norm(grad[k] - 2 * ref[k]) <= 2 * 2e-3 * max(np.linalg.norm(ref[k]), 1e-30), k
