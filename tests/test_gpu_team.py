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
