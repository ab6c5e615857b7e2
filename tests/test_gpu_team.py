"""Scans by teams (csrc/team.cuh): small calls, and the tails of large ones,
spread each trajectory over a block.  IGRF-14 is held to the oracle bit for
bit; with an external model a trajectory's results are the same bits whether
it runs by a team (a small call) or by one lane (among many)."""
from __future__ import annotations

import numpy as np
import pytest

import cortrace as ct
import pyoracle

pytestmark = pytest.mark.gpu

TIME7 = [2020, 6, 21, 173, 12, 0, 0]
PARMOD = [3.0, -60.0, 4.0, -7.0, 0.4, 0.8, 0.3, 1.1, 0.6, 0.9]


def jobs_of(n_sites: int, n_rig: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    lat = np.degrees(np.arcsin(rng.uniform(-1, 1, n_sites)))
    lat[:1] = 90.0 if seed % 2 else 0.0                      # the pole's branch; the equator
    lon = rng.uniform(0, 360, n_sites)
    return np.concatenate([ct.make_job(a, b, rig=0.3, rk=0.3 + 0.7 * (n_rig - 1), dele=0.7)
                           for a, b in zip(lat, lon)])


# trajectories: one slot, one block's eight, a block more than resident, and
# one beyond the teams' share (their tails only)
@pytest.mark.parametrize("n_sites,n_rig", [(1, 1), (1, 3), (3, 11), (61, 10), (175, 28), (650, 30)])
def test_igrf_equals_oracle(ctx, n_sites, n_rig):
    jobs = jobs_of(n_sites, n_rig, n_sites)
    p = ct.internal_setup("igrf14", TIME7)
    limit = 120
    gpu = ctx.trace_batch(jobs, p, step_limit=limit, want_records=True)
    cpu = pyoracle.scan_batch(jobs, p, step_limit=limit, threads=8, want_records=True)
    assert np.array_equal(gpu.status, cpu.status)
    assert np.array_equal(gpu.sites.view(np.uint8), cpu.sites.view(np.uint8))
    for k in ("pos", "vel", "v", "time", "length"):
        assert np.array_equal(gpu.records[k].view(np.uint64), cpu.records[k].view(np.uint64)), k
    for k in ("steps", "trials", "status"):
        assert np.array_equal(gpu.records[k], cpu.records[k]), k
    assert gpu.counters["accepted_steps"] == cpu.counters["accepted_steps"]


@pytest.mark.parametrize("tu,nk1", [(0.01, 7), (0.3, 100), (2.0, 33)])
def test_step_settings_equal_oracle(ctx, tu, nk1):
    """Other turn angles (2.0: the test that takes the angle itself) and steps per gyration."""
    jobs = np.concatenate([ct.make_job(a, b, rig=0.5, rk=10.5, dele=2.0, nk1=nk1, zn=z)
                           for a, b, z in ((50.0, 15.0, 1.0), (-20.0, 200.0, 2.0), (0.0, 100.0, -1.0))])
    p = ct.internal_setup("igrf14", TIME7)
    gpu = ctx.trace_batch(jobs, p, step_limit=300, tu_angle=tu, want_records=True)
    cpu = pyoracle.scan_batch(jobs, p, step_limit=300, tu_angle=tu, threads=8, want_records=True)
    assert np.array_equal(gpu.status, cpu.status)
    for k in ("pos", "vel", "time"):
        assert np.array_equal(gpu.records[k].view(np.uint64), cpu.records[k].view(np.uint64)), k
    for k in ("steps", "trials"):
        assert np.array_equal(gpu.records[k], cpu.records[k]), k


@pytest.mark.parametrize("external", [ct.EXTERNAL_T96, ct.EXTERNAL_TS05])
@pytest.mark.parametrize("internal", [ct.INTERNAL_SH, ct.INTERNAL_NONE])
def test_same_bits_among_many_and_alone(ctx, internal, external):
    """20,480 trajectories start one to a lane; the same ones in calls of 7, 640 and
    4,100 run by teams.  Every class, count and final state is the same bits."""
    jobs = jobs_of(640, 32, 5)
    p = ct.internal_setup("igrf14", TIME7, parmod=PARMOD)
    m = ct.model_set(internal, external)
    want = ctx.trace_batch(jobs, p, m, step_limit=70, want_records=True)
    for a, b in ((3, 3 + 1), (100, 120), (500, 628)):
        got = ctx.trace_batch(jobs[a:b], p, m, step_limit=70, want_records=True)
        s = slice(32 * a, 32 * b)
        assert np.array_equal(got.status, want.status[s])
        assert np.array_equal(got.records.view(np.uint8), want.records[s].view(np.uint8))


# points: one, a slot more than a block's eight, the last count that goes by
# teams and the first that does not, and the first sorted four to a thread (152 SMs)
@pytest.mark.parametrize("external,n", [(ct.EXTERNAL_NONE, 1), (ct.EXTERNAL_NONE, 9), (ct.EXTERNAL_NONE, 6485),
                                        (ct.EXTERNAL_NONE, 6486), (ct.EXTERNAL_NONE, 155649), (ct.EXTERNAL_T96, 1), (ct.EXTERNAL_T96, 9),
                                        (ct.EXTERNAL_T96, 6485), (ct.EXTERNAL_T96, 6486), (ct.EXTERNAL_TS05, 1),
                                        (ct.EXTERNAL_TS05, 9), (ct.EXTERNAL_TS05, 19456), (ct.EXTERNAL_TS05, 19457)])
def test_field_against_oracle(ctx, external, n):
    rng = np.random.default_rng(n)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    pts = u * np.exp(rng.uniform(np.log(1.003), np.log(24.0), n))[:, None] * ct.DEF_RE
    p = ct.internal_setup("igrf14", TIME7, parmod=PARMOD)
    m = ct.model_set(ct.INTERNAL_SH, external)
    got = ctx.field_batch(pts, p, m)
    if external == ct.EXTERNAL_NONE:
        # every point, in its own place (large calls evaluate them in another order)
        assert np.array_equal(got.view(np.uint64), pyoracle.calculate_field(pts, p, m).view(np.uint64))
    else:
        want = pyoracle.calculate_field(pts[:200], p, m)
        # within the reference's own spread under one-ulp changes of the C library
        # over storm conditions (T96 8.2e-12; TS05's central differences 2.4e-7) of
        # the sum's largest part (outside the magnetopause the dipole cancels the
        # internal field), or 16 times the point's own
        rel = 8.2e-12 if external == ct.EXTERNAL_T96 else 2.4e-7
        own = pyoracle.calculate_field_nudged(pts[:200], p, m)
        scale = np.linalg.norm(pyoracle.calculate_field(pts[:200], p, ct.model_set(ct.INTERNAL_SH)), axis=1)
        scale = np.maximum(scale, np.linalg.norm(want, axis=1))
        bar = np.maximum(rel * scale, 16.0 * np.linalg.norm(own - want, axis=1))
        assert np.all(np.linalg.norm(got[:200] - want, axis=1) <= bar)
