"""The crustal field's split of points over warps (field_kernel) and of a
lane's columns (chaos_geo_warp): every point equals the oracle to the crustal
sum's own rounding, for any count of points and any table size."""
from __future__ import annotations

import numpy as np
import pytest

import cortrace as ct
import pyoracle

pytestmark = pytest.mark.gpu

TIME7 = [2020, 6, 21, 173, 12, 0, 0]


def points(n, seed):
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    return u * rng.uniform(1.01, 1.5, n)[:, None] * ct.DEF_RE


# one point, a warp's 32 and one more, one point a warp, and two a warp for some
@pytest.mark.parametrize("n", [1, 32, 33, 1216, 1217, 2500])
def test_split_keeps_every_point(ctx, n):
    pts = points(n, 7)
    p = ct.internal_setup("igrf14", TIME7)
    m = ct.model_set(ct.INTERNAL_SH, ct.EXTERNAL_NONE, ct.CRUSTAL_CHAOS)
    got = ctx.field_batch(pts, p, m)
    # the same points one call each give the same bits
    for i in {0, n // 2, n - 1}:
        assert np.array_equal(ctx.field_batch(pts[i:i + 1], p, m).view(np.uint64), got[i:i + 1].view(np.uint64))
    k = [i for i in range(0, n, max(1, n // 6))]
    want = pyoracle.calculate_field(pts[k], p, m)
    # 17,391 terms of at most 1e-16 each, the sums in another order
    assert np.all(np.linalg.norm(got[k] - want, axis=1) <= 17391 * 1.2e-16 * np.linalg.norm(want, axis=1))


# columns: one per lane or fewer, an odd table, the largest accepted
@pytest.mark.parametrize("nmax", [2, 31, 33, 65, 192])
def test_table_sizes(nmax):
    rng = np.random.default_rng(nmax)
    nt = nmax * (nmax + 1) // 2
    g, h = rng.normal(size=nt), rng.normal(size=nt)
    g[0] = h[0] = 0.0
    h[[n * (n + 1) // 2 for n in range(nmax)]] = 0.0
    # one point against a plain sum in 64 bits: the recursion of the normalised functions
    x = np.array([[0.4, -0.7, 0.9]])
    r = float(np.linalg.norm(x))
    th, ph = np.arccos(x[0, 2] / r), np.arctan2(x[0, 1], x[0, 0])
    P = np.zeros((nmax, nmax))
    D = np.zeros((nmax, nmax))
    ct_, st_ = np.cos(th), np.sin(th)
    P[0, 0] = 1.0
    for n in range(1, nmax):
        for m in range(n + 1):
            if n == m:
                k = 1.0 if n == 1 else np.sqrt((2.0 * n - 1) / (2.0 * n))
                P[n, n] = st_ * k * P[n - 1, n - 1]
                D[n, n] = k * (ct_ * P[n - 1, n - 1] + st_ * D[n - 1, n - 1])
            else:
                k1 = (2 * n - 1) / np.sqrt(n * n - m * m)
                k2 = np.sqrt(((n - 1) ** 2 - m * m) / (n * n - m * m))
                a = P[n - 2, m] if n >= 2 else 0.0
                b = D[n - 2, m] if n >= 2 else 0.0
                P[n, m] = k1 * ct_ * P[n - 1, m] - k2 * a
                D[n, m] = k1 * (ct_ * D[n - 1, m] - st_ * P[n - 1, m]) - k2 * b
    br = bt = bp = 0.0
    mag = 0.0
    for n in range(1, nmax):
        f = r ** -(n + 2.0)
        for m in range(n + 1):
            i = n * (n + 1) // 2 + m
            c, s = np.cos(m * ph), np.sin(m * ph)
            t = g[i] * c + h[i] * s
            br += (n + 1) * f * t * P[n, m]
            bt -= f * t * D[n, m]
            bp -= f * m * (-g[i] * s + h[i] * c) * P[n, m] / st_
            mag += (n + 1) * f * (abs(g[i]) + abs(h[i])) * (abs(P[n, m]) + abs(D[n, m]) + n * abs(P[n, m]) / st_)
    er = x[0] / r
    et = np.array([ct_ * np.cos(ph), ct_ * np.sin(ph), -st_])
    ep = np.array([-np.sin(ph), np.cos(ph), 0.0])
    want = br * er + bt * et + bp * ep
    p = ct.internal_setup("igrf14", TIME7)
    p["a1"][0], p["a2"][0], p["a3"][0] = [1, 0, 0], [0, 1, 0], [0, 0, 1]
    with ct.Context(0) as c2:
        c2.upload_crustal(g, h, nmax)
        got = c2.field_batch(x * ct.DEF_RE, p, ct.model_set(ct.INTERNAL_NONE, ct.EXTERNAL_NONE, ct.CRUSTAL_CHAOS))
    # each recursion step adds a rounding or two to what it carries
    assert np.linalg.norm(got[0] - want) <= 8 * nmax * 1.2e-16 * mag
