"""Calls on the SMs that a scan stream reserves, in a process of its own (which
kernels a process has loaded matters here): a context that has run a set in a
large size goes on beside the stream in every other size.  (A call for which
the context's buffers have to grow waits for the stream: freeing device memory
does.)"""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import sys, time
sys.path.insert(0, sys.argv[1])
import numpy as np
import cortrace as ct
external = int(sys.argv[2])
p = ct.internal_setup("igrf14", [2020, 6, 21, 173, 12, 0, 0], parmod=[3.0, -60.0, 4.0, -7.0, 0.4, 0.8, 0.3, 1.1, 0.6, 0.9])
m = ct.model_set(1, external)
sites = np.concatenate([ct.make_job(-60.0 + 11 * k, 25.0 * k, rig=1.0, rk=20.99, dele=0.01) for k in range(12)])
pts = np.tile([[3.0, 1.0, 2.0]], (40000, 1)) * ct.DEF_RE
idle = 12.0
with ct.Context(0) as a, ct.Context(0) as b:
    b.trace_batch(sites, p, m, step_limit=2)
    b.field_batch(pts, p, m)
    with ct.Stream(a, ct.model_set(), slots=2, max_jobs=4, max_trajectories=64,
                   reserve_sms=2, idle_limit_s=idle) as st:
        t = st.submit(ct.make_job(50.0, 15.0, rig=8.0, rk=9.0, dele=1.0), p)
        st.wait(t)
        t0 = time.perf_counter()
        for n in (1, 12):
            b.trace_batch(sites[:1] if n == 1 else sites, p, m, step_limit=2)
        b.field_batch(pts[:21], p, m)
        b.field_batch(pts, p, m)
        print("took", time.perf_counter() - t0)
        st.drain()      # reports a stream that gave up meanwhile
print("ok")
"""


@pytest.mark.parametrize("external", [0, 1, 2])
def test_calls_of_every_size(external):
    r = subprocess.run([sys.executable, "-c", PROGRAM, os.path.join(ROOT, "cor-model_gb300"), str(external)],
                       capture_output=True, text=True, timeout=180)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout + r.stderr[-2000:]
    took = float(r.stdout.split("took")[1].split()[0])
    assert took < 6.0, took
