"""The step of the units without contraction (lane_advance<true>, csrc/trace.cuh)
leaves out operations that cannot change a result: it equals the general form
bit for bit, over ordinary states and over fields, charges and speeds at the
edges of what a double holds -- no field at all, an infinite one, none that is
a number.  On the CPU."""
from __future__ import annotations

import ctypes as C
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT
import cortrace as ct
from test_device_code_on_host import FLAGS

TU = 0.01


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    so = str(tmp_path_factory.mktemp("step_forms") / "step_host.so")
    src = os.path.join(ROOT, "tests", "device_on_host", "step_host.cpp")
    r = subprocess.run(["g++", *FLAGS, src, "-o", so, "-lm"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    lib = C.CDLL(so)
    vp, d = C.c_void_p, C.c_double
    lib.host_step.argtypes = [C.c_int, vp, d, d, d, d, C.c_uint64, vp, C.c_int64, vp]
    return lib


def states(n, b, seed):
    """Positions from 1 to 12 R_E, speeds up to the speed of light, field strengths b [nT]."""
    rng = np.random.default_rng(seed)
    s = np.zeros((n, 16))
    u, w, f = (rng.normal(size=(n, 3)) for _ in range(3))
    for a in (u, w, f):
        a /= np.linalg.norm(a, axis=1)[:, None]
    s[:, 0:3] = u * (np.exp(rng.uniform(0.01, math.log(12), n)) * ct.DEF_RE)[:, None]
    v = 299792458.0 * np.minimum(1.0, 1.0 - 10.0 ** rng.uniform(-17, -0.5, n))
    s[:, 3:6] = w * v[:, None]
    with np.errstate(all="ignore"):
        s[:, 6:9] = f * np.asarray(b)[:, None]
        s[:, 9] = 1e-9 * np.sqrt((s[:, 6:9] ** 2).sum(1))
    s[:, 10] = np.sqrt((s[:, 3:6] ** 2).sum(1))
    s[:, 11] = rng.uniform(0, 1, n)
    s[:, 12] = rng.uniform(0, 1e8, n)
    s[:, 13] = rng.choice([1.0, -1.0, 2.0, 26.0], n)
    s[:, 14] = rng.choice([1, 7, 100, 333], n)
    s[:, 15] = s[:, 14]
    return s


def both(lib, s):
    p = ct.internal_setup("igrf14", [2020, 6, 21, 173, 12, 0, 0])
    gc = math.cos(TU)
    half = 0.5 * (math.nextafter(gc, 2.0) - gc)
    out = []
    for plain in (0, 1):
        o = np.zeros((len(s), 12))
        lib.host_step(plain, p.ctypes.data, TU, gc, half, ct.DEF_HM0_P, 25000, s.ctypes.data, len(s), o.ctypes.data)
        o[np.isnan(o)] = np.nan            # whichever NaN
        out.append(o)
    return out


def equal(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


def test_ordinary_steps(lib):
    n = 20000
    want, got = both(lib, states(n, 10.0 ** np.random.default_rng(1).uniform(0, 5, n), 2))
    assert equal(want, got) and len(set(want[:, 0])) > 1


@pytest.mark.parametrize("b", [0.0, 5e-324, 1e-300, 1e-160, 1e-30, 1e160, 1e300, np.inf, np.nan])
def test_edges_of_the_field(lib, b):
    want, got = both(lib, states(500, np.full(500, b), 3))
    assert equal(want, got)
    if b == 0.0:
        # 2 pi m / (q B): infinite, as the division gives it
        assert np.all(np.isinf(want[want[:, 0] == 0][:, 8]))


def test_particle_at_the_speed_of_light(lib):
    """Rounded to it, far above every rigidity scanned: the mass is infinite."""
    s = states(500, np.full(500, 3e4), 4)
    s[:, 10] = 299792458.0
    want, got = both(lib, s)
    assert equal(want, got)
