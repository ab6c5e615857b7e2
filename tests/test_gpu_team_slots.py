"""Team blocks (csrc/team.cuh) of every size: a task kind's chunks hold 32
lanes, so blocks are tried around the slot counts where a kind of task with 2,
3, 5, 6 or 7 per slot takes one more chunk, at the most slots a set has, and
with a second pass over the slots."""
from __future__ import annotations

import numpy as np
import pytest

import cortrace as ct
from test_gpu_team import PARMOD, TIME7, jobs_of
from test_gpu_team import test_field_against_oracle as check_field

pytestmark = pytest.mark.gpu

SMS = 152


# slots per block of the whole batch (IGRF-14: two blocks to an SM share them)
@pytest.mark.parametrize("external", [ct.EXTERNAL_NONE, ct.EXTERNAL_T96, ct.EXTERNAL_TS05])
@pytest.mark.parametrize("slots", [2, 4, 5, 7, 10, 11, 16, 17, 19, 20, 29, 30, 33])
def test_field_same_bits_for_any_block(ctx, external, slots):
    """A point's field does not depend on the slots of its block: the batch against
    its points in calls of at most one slot per block."""
    rng = np.random.default_rng(slots)
    n = min(SMS * slots, {ct.EXTERNAL_NONE: 6485, ct.EXTERNAL_T96: 9728, ct.EXTERNAL_TS05: 29184}[external])
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    pts = u * np.exp(rng.uniform(np.log(1.003), np.log(14.0), n))[:, None] * ct.DEF_RE
    p = ct.internal_setup("igrf14", TIME7, parmod=PARMOD)
    m = ct.model_set(ct.INTERNAL_SH, external)
    got = ctx.field_batch(pts, p, m)
    for a in range(0, min(n, 1500), 150):
        want = ctx.field_batch(pts[a:a + 150], p, m)
        assert np.array_equal(got[a:a + 150].view(np.uint64), want.view(np.uint64)), a
    # the last block's and the last pass's points too
    assert np.array_equal(got[-150:].view(np.uint64), ctx.field_batch(pts[-150:], p, m).view(np.uint64))


@pytest.mark.parametrize("external,n_sites", [(ct.EXTERNAL_NONE, 243), (ct.EXTERNAL_T96, 152), (ct.EXTERNAL_T96, 170),
                                              (ct.EXTERNAL_TS05, 152), (ct.EXTERNAL_TS05, 243), (ct.EXTERNAL_TS05, 260)])
def test_scan_same_bits_for_any_block(ctx, external, n_sites):
    """20 rigidities a site: full blocks, and more trajectories than slots."""
    jobs = jobs_of(n_sites, 20, n_sites)
    p = ct.internal_setup("igrf14", TIME7, parmod=PARMOD)
    m = ct.model_set(ct.INTERNAL_SH, external)
    got = ctx.trace_batch(jobs, p, m, step_limit=60, want_records=True)
    for a in (0, n_sites // 2, n_sites - 7):
        want = ctx.trace_batch(jobs[a:a + 7], p, m, step_limit=60, want_records=True)
        s = slice(20 * a, 20 * (a + 7))
        assert np.array_equal(got.status[s], want.status)
        assert np.array_equal(got.records[s].view(np.uint8), want.records.view(np.uint8))


# the last count that goes by teams and the first that does not
@pytest.mark.parametrize("external,n", [(ct.EXTERNAL_T96, 9728), (ct.EXTERNAL_T96, 9729), (ct.EXTERNAL_TS05, 29184),
                                        (ct.EXTERNAL_TS05, 29185)])
def test_field_at_the_limit(ctx, external, n):
    check_field(ctx, external, n)
