"""The window network repeats itself: the same rows give the same bits on every
call, whatever the timing between the CTAs of a cluster.  (The order that this
rests on is checked on the CPU, tests/test_network_order.py.)"""
from __future__ import annotations

import numpy as np
import pytest

import window

pytestmark = pytest.mark.gpu


def weights_of(g):
    """The weight gradients; the biases' are sums of atomic additions."""
    return np.concatenate([a.reshape(-1) for a in window.split_params(g) if a.ndim == 2])


@pytest.mark.parametrize("n", [1, 129, 2664])
def test_forward_and_gradient_repeat(n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    x = torch.from_numpy(rng.normal(size=(n, window.N_IN)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.normal(size=(n, window.N_OUT)).astype(np.float32)).cuda()
    net = window.Network(0, max_batch=n)
    try:
        net.set_params(window.init_params(n))
        y = net.forward(x).clone()
        g = weights_of(net.gradient(x, t)[1])
        for _ in range(200):
            assert torch.equal(net.forward(x), y)
            assert np.array_equal(weights_of(net.gradient(x, t)[1]).view(np.uint32), g.view(np.uint32))
    finally:
        net.close()
