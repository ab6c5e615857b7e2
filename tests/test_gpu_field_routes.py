"""The routes of a field batch -- teams, one point to a lane (sorted by band or
not), a warp to a crustal sum -- give a point the same field: with a parameter
block of its own, and at positions where there is nothing ordinary about it.
TS05 by one lane is contracted by the compiler in other places than by a team:
its points are held to the model's own rounding instead of the bits."""
from __future__ import annotations

import numpy as np
import pytest

import cortrace as ct
from test_gpu_team import PARMOD, TIME7

pytestmark = pytest.mark.gpu

# of a calculate_field evaluation: some 10^4 terms of 1e-16 each, added with cancellation
TS05_TOL = 1e-12
# model set, calls by teams, by one lane to a point, by four points to a thread
ROUTES = [((1, 0, 0), (5, 6000), (7000, 320000)), ((1, 1, 0), (5, 9000), (10000, 25000)),
          ((0, 1, 0), (5, 9000), (10000, 25000)), ((1, 2, 0), (5, 29000), (30000, 60000)),
          ((0, 2, 0), (5, 29000), (30000, 60000)), ((1, 0, 1), (5, 33), (1300, 2600)), ((1, 1, 1), (5, 33), (1300, 2600))]


def positions(n, seed, hi=12.0):
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(n, 3))
    return u / np.linalg.norm(u, axis=1)[:, None] * np.exp(rng.uniform(0.003, np.log(hi), n))[:, None] * ct.DEF_RE


def params():
    return np.concatenate([ct.internal_setup("igrf14", [2015 + 3 * k, 1 + k, 1, 1 + 30 * k, 6 * k, 0, 0],
                                             parmod=np.array(PARMOD) * (1 + 0.2 * k)) for k in range(3)])


def same(models, a, b):
    if models[1] != ct.EXTERNAL_TS05:
        return np.array_equal(a, b, equal_nan=True)
    return np.array_equal(np.isfinite(a), np.isfinite(b)) and \
        np.all(np.linalg.norm(a - b, axis=1)[np.isfinite(a).all(1)] <=
               TS05_TOL * np.linalg.norm(b, axis=1)[np.isfinite(a).all(1)])


@pytest.mark.parametrize("models,team,lane", ROUTES)
def test_parameter_block_of_each_point(ctx, models, team, lane):
    p, m = params(), ct.model_set(*models)
    for n in team + lane:
        pts = positions(n, n, 1.5 if models[2] else 12.0)
        idx = np.random.default_rng(n + 1).integers(0, 3, n).astype(np.int32)
        got = ctx.field_batch(pts, p, m, param_index=idx)
        for k in range(3):
            at = np.nonzero(idx == k)[0]
            # the same points in calls of a block's own, of another size
            if len(at):
                assert same(models, got[at], ctx.field_batch(pts[at], p[k:k + 1], m)), (n, k)
                assert same(models, got[at[:3]], ctx.field_batch(pts[at[:3]], p[k:k + 1], m)), (n, k)


@pytest.mark.parametrize("models,team,lane", [r for r in ROUTES if not r[0][2]])
def test_unusual_positions(ctx, models, team, lane):
    """The origin, the axis, infinities and NaN, among ordinary points and alone."""
    inf, nan, re = np.inf, np.nan, ct.DEF_RE
    odd = np.array([[0, 0, 0], [0, 0, 3 * re], [0, 0, -3 * re], [3 * re, 0, 0], [0, 3 * re, 0], [-60 * re, 0, 0],
                    [1e-300, 0, 0], [1e30, 1e30, 1e30], [1e200, 0, 0], [inf, 0, 0], [-inf, inf, 0], [0, 0, inf],
                    [nan, 0, 0], [0, nan, re], [nan, nan, nan], [-0.0, -0.0, 2 * re]], np.float64)
    p, m = params()[:1], ct.model_set(*models)
    alone = ctx.field_batch(odd, p, m)
    for n in team[1:] + lane:
        pts = positions(n, n)
        at = np.random.default_rng(n).choice(n, len(odd), replace=False)
        pts[at] = odd
        got = ctx.field_batch(pts, p, m)
        assert same(models, got[at], alone), n
        # and the points beside them are as they are without them
        rest = np.setdiff1d(np.arange(n), at)[:200]
        assert same(models, got[rest], ctx.field_batch(pts[rest], p, m)) and np.isfinite(got[rest]).all()
