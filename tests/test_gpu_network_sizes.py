"""The window network's kernels (csrc/mlp.cu) at the sizes where a tile or a
ring can go wrong: batches around a 128-row tile, one tile and several, a
network larger than its batch, and the optimiser's update."""
from __future__ import annotations

import numpy as np
import pytest

import mlp_oracle
import window

pytestmark = pytest.mark.gpu

SIZES = [1, 127, 128, 129, 640, 1024]


@pytest.fixture(scope="module")
def net():
    pytest.importorskip("torch")
    n = window.Network(0, max_batch=1024)
    yield n
    n.close()


def batch(n, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 1, (n, window.N_IN)).astype(np.float32), rng.normal(0, 1, (n, 2)).astype(np.float32)


@pytest.mark.parametrize("n", SIZES)
def test_forward(net, n):
    import torch
    p = window.init_params(n)
    net.set_params(p)
    x, _ = batch(n, n)
    y = net.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    want, _ = mlp_oracle.forward(p, x.astype(np.float64))
    assert np.linalg.norm(y - want) <= 1e-2 * np.linalg.norm(want)
    # a row's result does not depend on the rows beside it
    k = n // 2
    one = net.forward(torch.from_numpy(x[k:k + 1]).cuda()).cpu().numpy()
    assert np.array_equal(one.view(np.uint32), y[k:k + 1].view(np.uint32))


@pytest.mark.parametrize("n", SIZES)
def test_gradient_and_update(net, n):
    import torch
    p = window.init_params(n + 1)
    net.set_params(p)
    x, t = batch(n, n + 1)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    loss, g = net.gradient(xd, td)
    assert np.array_equal(net.get_params(), p)                    # no update
    want_loss, want = mlp_oracle.gradient(p, x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - want_loss) <= 1e-2 * abs(want_loss)
    for a, b in zip(window.split_params(g), window.split_params(np.asarray(want))):
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b)
    # AdamW's first step from that gradient, in 64 bits
    net.train_step(xd, td, lr=1e-3, weight_decay=1e-2)
    after = net.get_params().astype(np.float64)
    g64 = g.astype(np.float64)
    m, v = 0.1 * g64, 0.001 * g64 * g64
    step = (m / (1 - 0.9)) / (np.sqrt(v / (1 - 0.999)) + 1e-8)
    decay = np.concatenate([np.full(a.size, 1e-2 if a.ndim == 2 else 0.0) for a in window.split_params(p)])
    want = p.astype(np.float64) - 1e-3 * (step + decay * p)
    # |step| <= 1 wherever the gradient is above AdamW's eps; a bias gradient's own sum order
    # moves only entries near it
    big = np.abs(g64) > 1e-6 * np.abs(g64).max()
    assert np.all(np.abs(after - want)[big] <= 1e-3 * 1e-3 + 2e-7 * np.abs(want)[big])
    # the BF16 copies follow the weights: the next forward uses them
    y = net.forward(xd).cpu().numpy()
    ref, _ = mlp_oracle.forward(net.get_params(), x.astype(np.float64))
    assert np.linalg.norm(y - ref) <= 1e-2 * np.linalg.norm(ref)
