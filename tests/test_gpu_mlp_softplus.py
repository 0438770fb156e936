"""softplus and its derivative as the network's kernels form them, against float64 over the whole range of a
float32 activation.  With W1, W2, W3 at zero the third layer's activations are softplus(b3); with one point,
a label of 1 and b4 far below zero, dL/dg is exactly -1, so the gradients of the head are -h3 and those of b3
the gates -(1 - e^-h3), each from one call and unrounded.  Bounds from the instructions' documented errors:
4e-7 + 2^-24 |x| for softplus, 4e-7 for the gate."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def network():
    from kups_gb300 import mlp

    net = mlp.LearnedInsertionProposal(seed=1, grid=2)
    for x in (net.param, net.param_bf16, net.param_bf16_t, net.grad):
        x.zero_()
    return net, lambda flat, name: flat[mlp.OFFSETS[name][0]:][:int(np.prod(mlp.OFFSETS[name][1]))]


def activations():
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-1, 1, 3000), rng.uniform(-20, 20, 3000), rng.uniform(-110, 110, 1500),
                        rng.choice([-1, 1], 1500) * 10.0 ** rng.uniform(-40, 4, 1500),
                        [0.0, -0.0, 1e4, -1e4, 87.3, -87.4, 88.8, -103.9, -104.1, 1e-45, -1e-45, 16.6, 17.4]])
    return np.resize(x, -(-len(x) // 256) * 256).astype(np.float32).reshape(-1, 256)


def test_softplus_and_its_gate():
    net, part = network()
    part(net.param, "w4").fill_(1.0)
    part(net.param, "b4").fill_(-1e30)
    point, label = torch.zeros((1, 3), dtype=torch.float64, device="cuda"), torch.ones(1, device="cuda")
    for x in activations():
        part(net.param, "b3").copy_(torch.as_tensor(x))
        net.grad.zero_()
        net.backward(point, label)
        h = -part(net.grad, "w4").cpu().numpy().astype(float)
        gate = -part(net.grad, "b3").cpu().numpy().astype(float)
        want = np.logaddexp(0.0, x.astype(float))
        assert (np.abs(h - want) <= 4e-7 + 2.0**-24 * np.abs(x)).all()
        assert (np.abs(gate + np.expm1(-h)) <= 4e-7).all()
    net.check()


def test_softplus_of_the_forward_pass():
    net, part = network()
    x = activations()[::8, :16]
    points = torch.zeros((1, 3), dtype=torch.float64, device="cuda")
    for row in x:
        part(net.param, "b3")[:16].copy_(torch.as_tensor(row))
        for k, v in enumerate(row):
            part(net.param, "w4").zero_()
            part(net.param, "w4")[k] = 1.0
            got = float(net.forward(points)[0])
            assert abs(got - np.logaddexp(0.0, float(v))) <= 4e-7 + 2.0**-24 * abs(float(v))
    net.check()
