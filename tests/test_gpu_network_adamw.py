"""Several AdamW steps of the window network, replayed in 64 bits from the
gradients that each step exports: the moments are carried from step to step
where they belong, with the corrections of their step, and the BF16 copies that
the products read (both ways round) follow the weights."""
from __future__ import annotations

import numpy as np
import pytest

import mlp_oracle
import window

pytestmark = pytest.mark.gpu

# large enough that a step moves a weight by half of its initial spread: a product
# with the weights of the step before would be off by that much
LR, DECAY, STEPS = 0.02, 1e-2, 4


@pytest.mark.parametrize("n", [100, 384])
def test_steps_replayed(n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    net = window.Network(0, max_batch=n)
    try:
        p = window.init_params(n)
        net.set_params(p)
        decay = np.concatenate([np.full(a.size, DECAY if a.ndim == 2 else 0.0) for a in window.split_params(p)])
        m = v = np.zeros(window.N_PARAMS)
        grads = torch.zeros(window.N_PARAMS, dtype=torch.float32, device="cuda")
        for k in range(1, STEPS + 1):
            x = rng.normal(size=(n, window.N_IN)).astype(np.float32)
            t = rng.normal(size=(n, window.N_OUT)).astype(np.float32)
            xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
            net._check(net.lib.cor_mlp_train_step(net.h, xd.data_ptr(), td.data_ptr(), n, LR, DECAY,
                                                  net.loss.data_ptr(), grads.data_ptr(), net._stream()), "train_step")
            g = grads.cpu().numpy().astype(np.float64)
            _, want = mlp_oracle.gradient(p, x.astype(np.float64), t.astype(np.float64))
            for a, b in zip(window.split_params(g), window.split_params(np.asarray(want))):
                assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b), k
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            step = (m / (1 - 0.9 ** k)) / (np.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
            want = p - LR * (step + decay * p)
            after = net.get_params().astype(np.float64)
            # 32 bits: 1 - 0.999^k holds 6e-8 / 1e-3 of itself, its root half of that; the moment's
            # terms may cancel to 1e-5 of their size; the new weight is rounded once
            clear = np.sqrt(v) > 1e-12
            tol = LR * (1e-4 * np.abs(step) + 1e-5) + 2e-7 * np.abs(p) + 2e-7 * np.abs(want)
            assert np.all(np.abs(after - want)[clear] <= tol[clear]), k
            assert np.abs(after - p).max() > 0.5 * LR
            p = after.astype(np.float32)
            y = net.forward(xd).cpu().numpy()
            ref, _ = mlp_oracle.forward(p, x.astype(np.float64))
            assert np.linalg.norm(y - ref) <= 1e-2 * np.linalg.norm(ref), k
    finally:
        net.close()
