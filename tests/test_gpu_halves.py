"""The first generation of a large IGRF-14 scan in blocks of half the threads
(use_halves in csrc/cortrace.cu): from two trajectories a lane on, 77,824 on a
GPU of 152 SMs."""
from __future__ import annotations

import numpy as np
import pytest

import cortrace as ct
from test_gpu_team import TIME7, jobs_of

pytestmark = pytest.mark.gpu


# the last count in whole blocks, the first in halves, and lanes that refill with parked tails
@pytest.mark.parametrize("n_sites,n_rig,limit", [(2594, 30, 40), (2595, 30, 40), (3001, 31, 40), (2600, 30, 400)])
def test_same_bits_as_in_smaller_calls(ctx, n_sites, n_rig, limit):
    jobs = jobs_of(n_sites, n_rig, n_sites)
    p = ct.internal_setup("igrf14", TIME7)
    got = ctx.trace_batch(jobs, p, step_limit=limit, want_records=True)
    half = n_sites // 2
    steps = 0
    for a, b in ((0, half), (half, n_sites)):
        want = ctx.trace_batch(jobs[a:b], p, step_limit=limit, want_records=True)
        s = slice(n_rig * a, n_rig * b)
        assert np.array_equal(got.status[s], want.status)
        assert np.array_equal(got.records[s].view(np.uint8), want.records.view(np.uint8))
        assert np.array_equal(got.sites[a:b].view(np.uint8), want.sites.view(np.uint8))
        steps += want.counters["accepted_steps"]
    assert got.counters["accepted_steps"] == steps
