"""One context per thread (include/cor_trace.h): field batches and scans of
very different sizes from two threads at a time give each thread what it gets
alone."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import cortrace as ct
from test_gpu_team import PARMOD, TIME7, jobs_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("external", [ct.EXTERNAL_NONE, ct.EXTERNAL_T96, ct.EXTERNAL_TS05])
def test_two_threads(external):
    p = ct.internal_setup("igrf14", TIME7, parmod=PARMOD)
    m = ct.model_set(ct.INTERNAL_SH, external)
    rng = np.random.default_rng(5)
    u = rng.normal(size=(5000, 3))
    pts = u / np.linalg.norm(u, axis=1)[:, None] * rng.uniform(1.1, 9.0, 5000)[:, None] * ct.DEF_RE
    jobs = jobs_of(80, 25, 9)
    sizes = [(1, 1), (5000, 80), (300, 3), (2500, 40)]

    def calls(ctx, order):
        out = {}
        for n, j in order:
            r = ctx.trace_batch(jobs[:j], p, m, step_limit=20)
            out[n] = (ctx.field_batch(pts[:n], p, m).tobytes(), r.sites.tobytes(), r.status.tobytes())
        return out

    with ct.Context(0) as a, ct.Context(0) as b:
        want = calls(a, sizes)
        wrong = []

        def loop(ctx, order):
            try:
                for _ in range(25):
                    if calls(ctx, order) != want:
                        wrong.append("another result")
            except Exception as e:  # noqa: BLE001
                wrong.append(repr(e))
        ts = [threading.Thread(target=loop, args=(a, sizes)), threading.Thread(target=loop, args=(b, sizes[::-1]))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert not wrong, wrong[:3]
