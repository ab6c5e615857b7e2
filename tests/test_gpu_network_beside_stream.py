"""The window network on a device that a scan stream holds but for its
reserved SMs: calls finish before the stream is drained, with the bits they
have on a free device; the stream server predicts windows for requests that
arrive while others are being traced."""
from __future__ import annotations

import os
import time

import numpy as np
import pytest

import cortrace as ct
import serve
import window
from conftest import ROOT
from test_gpu_network_repeats import weights_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reserve", [1, 2])
@pytest.mark.parametrize("n", [1, 128, 129, 2664])
def test_same_bits_beside_a_stream(ctx, n, reserve):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    x = torch.from_numpy(rng.normal(size=(n, window.N_IN)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.normal(size=(n, window.N_OUT)).astype(np.float32)).cuda()
    p = ct.internal_setup("igrf14", [2020, 6, 21, 173, 12, 0, 0])
    job = ct.make_job(50.0, 15.0, rig=5.0, rk=9.0, dele=1.0)
    net = window.Network(0, max_batch=n)
    try:
        net.set_params(window.init_params(n))

        def calls():
            loss, g = net.gradient(x, t)
            return net.forward(x).cpu().numpy(), weights_of(g), g, loss
        want = calls()
        # a call that had to wait would end with the stream's idle limit
        with ct.Stream(ctx, ct.model_set(), slots=2, max_jobs=4, max_trajectories=64, reserve_sms=reserve,
                       idle_limit_s=8.0) as st:
            ticket = st.submit(job, p)
            t0 = time.perf_counter()
            got = calls()
            took = time.perf_counter() - t0
            assert st.wait(ticket)[0].sites["n_traj"][0] == 5
            st.drain()
        assert took < 2.0
        assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32))
        assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
        # the biases' and the loss's sums are atomic additions of n terms, in any order
        bias = np.concatenate([a for a in window.split_params(got[2]) if a.ndim == 1])
        bias0 = np.concatenate([a for a in window.split_params(want[2]) if a.ndim == 1])
        assert np.allclose(bias, bias0, rtol=0, atol=n * 6e-8 * np.abs(bias0).max())
        assert abs(got[3] - want[3]) <= n * 6e-8 * want[3]
    finally:
        net.close()


def test_stream_server_with_a_window_model(monkeypatch):
    pytest.importorskip("torch")
    made = ct.Stream
    monkeypatch.setattr(ct, "Stream", lambda *a, **k: made(*a, **{**k, "idle_limit_s": 20.0}))
    # the network trained with T96, for scans in IGRF-14: the windows are wider of the mark,
    # and every result is traced all the same
    wm = window.WindowModel(os.path.join(ROOT, "cor-model_gb300", "window_t96.npz"))
    wm.external = ct.EXTERNAL_NONE

    def requests():
        reqs = serve.poisson_stream(31, 20.0, 4, ct.EXTERNAL_T96, max_box_sites=4)
        for r in reqs:
            r.external = ct.EXTERNAL_NONE
            r.directions = r.directions[:1]
        return reqs

    def run(reqs):
        return serve.run_stream(serve.StreamServer(0, window_model=wm, externals=(ct.EXTERNAL_NONE,)), reqs)
    try:
        mix = requests()
        assert run(mix)["completed"] == 4
        alone = requests()[2:3]
        alone[0].arrival = 0.0
        run(alone)
        assert np.array_equal(alone[0].result.view(np.uint8), mix[2].result.view(np.uint8))
    finally:
        wm.close()
