"""The host side of libcortrace over a stand-in for the CUDA runtime
(tests/host_runtime/fake_cudart.cpp), on the CPU: what it reports when a
launch or a copy fails, how long it keeps what an asynchronous copy reads, and
what calls of other threads can change.  Kernels do nothing here."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT
import build_lib
import cortrace as ct

SRC = os.path.join(ROOT, "tests", "host_runtime", "fake_cudart.cpp")
ERR_NOMEM, ERR_CUDA = -2, -3
TIME7 = [2020, 6, 21, 173, 12, 0, 0]
PARMOD = [3.0, -40.0, 2.0, -5.0, 0.5, 0.4, 0.3, 0.5, 0.3, 0.6]


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    build_lib.build()
    so = str(tmp_path_factory.mktemp("host_runtime") / "libcortrace_host.so")
    objs = [os.path.join(build_lib.BUILD, s + ".o") for s in build_lib.CU_SOURCES + build_lib.LIB_C_SOURCES]
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build_lib.nvcc()))), "include")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fPIC", "-shared", "-pthread", f"-I{cuda}", SRC, *objs,
                        "-o", so, "-Wl,-Bsymbolic", "-Wl,--wrap=free", "-lm", "-ldl"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    was, ct._lib = ct._lib, None
    lib = ct.load(so)
    lib.fake_fail_launch.argtypes = [C.c_char_p]
    lib.fake_fail_call.argtypes = [C.c_char_p, C.c_int]
    lib.fake_memory.argtypes = [C.c_uint64]
    lib.fake_in_use.restype = C.c_uint64
    lib.fake_limits_set.argtypes = [C.c_char_p]
    lib.fake_launch.argtypes = [C.c_int, C.c_char_p, C.c_int, C.POINTER(C.c_uint), C.POINTER(C.c_uint),
                                C.POINTER(C.c_uint64)]
    yield lib
    lib.fake_reset()
    ct._lib = was


@pytest.fixture()
def host(fake):
    fake.fake_reset()
    yield fake
    fake.fake_reset()


def params(external=ct.EXTERNAL_NONE):
    return ct.internal_setup("igrf14", TIME7, parmod=PARMOD if external else None)


def points(n):
    return np.tile(np.array([[3.0, 1.0, 2.0]]) * ct.DEF_RE, (n, 1))


# a team call and one point to a lane, for every model set
FIELD_CALLS = [(m, n) for m in [(1, 0, 0), (1, 1, 0), (0, 1, 0), (1, 2, 0), (0, 2, 0)] for n in (5, 40000)] + \
    [((1, 1, 1), 5)]


@pytest.mark.parametrize("models,n", FIELD_CALLS)
def test_field_launch_that_fails_is_reported(host, models, n):
    """cor_field_batch keeps its output buffer between calls: a launch that
    fails must not hand out the fields of the call before."""
    with ct.Context(0) as ctx:
        m = ct.model_set(*models)
        ctx.field_batch(points(n), params(1), m)
        host.fake_fail_launch(b"field_kernel")
        with pytest.raises(ct.CorError) as e:
            ctx.field_batch(points(n), params(1), m)
        assert e.value.code == ERR_CUDA
        host.fake_fail_launch(b"")
        ctx.field_batch(points(n), params(1), m)


@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_field_copy_that_fails_is_reported(host, nth):
    """Parameters, positions, parameter indices, fields."""
    with ct.Context(0) as ctx:
        idx = np.zeros(7, np.int32)
        ctx.field_batch(points(7), params(), param_index=idx)
        host.fake_fail_call(b"cudaMemcpyAsync", nth)
        with pytest.raises(ct.CorError) as e:
            ctx.field_batch(points(7), params(), param_index=idx)
        assert e.value.code == ERR_CUDA


def test_error_of_one_call_is_not_the_next_ones(host):
    """A call that found no memory has reported it; the next one is itself again."""
    jobs = ct.make_job(50.0, 15.0, rig=1.0, rk=5.0, dele=1.0)
    with ct.Context(0) as ctx:
        for call in (lambda: ctx.field_batch(points(7), params()), lambda: ctx.trace_batch(jobs, params()),
                     lambda: ctx.upload_crustal(np.ones(6), np.ones(6), 3)):
            host.fake_fail_call(b"cudaMalloc", 1)
            with pytest.raises(ct.CorError) as e:
                call()
            assert e.value.code == ERR_NOMEM
            ctx.field_batch(points(7), params(), ct.model_set(ct.INTERNAL_SH, ct.EXTERNAL_T96))
            call()


@pytest.mark.parametrize("n,n_params", [(1, 1), (7, 3), (40000, 1)])
def test_field_parameters_outlive_their_copy(host, n, n_params):
    """The runtime may read a pageable source at any time before the stream is
    waited for: nothing a queued copy reads is freed before."""
    with ct.Context(0) as ctx:
        for models in [(1, 0, 0), (1, 1, 0), (1, 2, 0), (1, 0, 1)]:
            ctx.field_batch(points(n), np.repeat(params(1), n_params), ct.model_set(*models))
            assert host.fake_freed_pending() == 0 and host.fake_pending() == 0


@pytest.mark.parametrize("call", ["cudaMalloc", "cudaOccupancy", "cudaFuncSetAttribute", "cudaMemcpyAsync"])
@pytest.mark.parametrize("nth", range(1, 5))
@pytest.mark.parametrize("models", [(1, 0, 0), (1, 1, 0), (1, 0, 1)])
def test_field_call_that_fails_leaves_no_copy_behind(host, call, nth, models):
    """Whatever fails, no copy from or to the caller's arrays is pending afterwards."""
    with ct.Context(0) as ctx:
        host.fake_fail_call(call.encode(), nth)
        try:
            ctx.field_batch(points(7), params(1), ct.model_set(*models), param_index=np.zeros(7, np.int32))
        except ct.CorError as e:
            assert e.code in (ERR_CUDA, ERR_NOMEM)
        assert host.fake_pending() == 0 and host.fake_freed_pending() == 0


TEAM_SETS = [(1, 0, 0), (1, 1, 0), (0, 1, 0), (1, 2, 0), (0, 2, 0)]


def scan(ctx, n, models):
    jobs = ct.make_job(50.0, 15.0, rig=1.0, rk=1.0 + 0.01 * (n - 1), dele=0.01)
    return ctx.trace_batch(jobs, params(1), ct.model_set(*models), step_limit=10)


@pytest.mark.parametrize("models", TEAM_SETS)
def test_calls_of_other_threads_do_not_change_a_launch(host, models):
    """The limit of dynamic shared memory belongs to a function on the device,
    and contexts of other threads make calls of other sizes: whatever they set
    between this call's set-up and its launch must leave room for it.  Here the
    other thread's call runs right after each setting, with the least shared
    memory a call can take."""
    with ct.Context(0) as a, ct.Context(0) as b:
        m = ct.model_set(*models)
        for mine in (lambda: a.field_batch(points(2000), params(1), m), lambda: scan(a, 2000, models)):
            inside = []

            def other(_name):
                if not inside:
                    inside.append(1)
                    b.field_batch(points(1), params(1), m)
                    scan(b, 1, models)
                    inside.pop()
            hook = C.CFUNCTYPE(None, C.c_char_p)(other)
            host.fake_after_attribute(hook)
            mine()
            host.fake_after_attribute(None)
    for f in (b"team_trace_kernel", b"team_field_kernel"):
        assert host.fake_limits_set(f) == 1


class Network:
    """A window network over the stand-in runtime; rows: the forms its calls launched."""

    def __init__(self, host, max_batch=512):
        import window
        self.lib, self.host = window._bind(host), host
        self.h = C.c_void_p()
        assert self.lib.cor_mlp_create(0, max_batch, C.byref(self.h)) == 0
        self.x = np.zeros((max_batch, window.N_IN), np.float32)
        self.y = np.zeros((max_batch, window.N_OUT), np.float32)
        self.out = np.zeros(window.N_PARAMS + 1, np.float32)

    def forward(self, n=300):
        return self._form(self.lib.cor_mlp_forward(self.h, self.x.ctypes.data, n, self.y.ctypes.data, None), n)

    def train(self, n=300):
        return self._form(self.lib.cor_mlp_train_step(self.h, self.x.ctypes.data, self.y.ctypes.data, n, 1e-3, 0.0,
                                                      self.out.ctypes.data, None, None), n)

    def _form(self, rc, n):
        assert rc == 0
        name, grid = [(k, g) for k, g in launched(self.host) if "rows_kernel" in k][-1]
        split = 4 if "ILi4E" in name else 1
        assert grid == split * ((n + 127) // 128)
        return split

    def close(self):
        self.lib.cor_mlp_destroy(self.h)


def launched(host):
    name, g, b, m = C.create_string_buffer(512), C.c_uint(), C.c_uint(), C.c_uint64()
    out = []
    for i in range(host.fake_launch_count()):
        host.fake_launch(i, name, 512, C.byref(g), C.byref(b), C.byref(m))
        out.append((name.value.decode(), g.value))
    return out


def small_stream(ctx):
    return ct.Stream(ctx, ct.model_set(), slots=2, max_jobs=4, max_trajectories=64, max_params=1, fixed_params=1,
                     pool_params=8, reserve_sms=2)


@pytest.fixture()
def net(host):
    n = Network(host)
    yield n
    n.close()


JOB = dict(rig=1.0, rk=5.0, dele=1.0)


def test_network_beside_a_stream_needs_no_cluster(host, net):
    """A scan stream leaves a network reserve_sms SMs (include/cor_trace.h): too
    few to place clusters of four CTAs until it is drained."""
    with ct.Context(0) as ctx, small_stream(ctx) as st:
        assert (net.forward(), net.train()) == (4, 4)
        for _ in range(2):
            st.submit(ct.make_job(50.0, 15.0, **JOB), params())
            assert (net.forward(), net.train()) == (1, 1)
            st.drain()
            assert (net.forward(), net.train()) == (4, 4)
        host.fake_fail_launch(b"stream_kernel")
        with pytest.raises(ct.CorError):
            st.submit(ct.make_job(50.0, 15.0, **JOB), params())
        assert net.forward() == 4
        host.fake_fail_launch(b"")


def test_network_beside_a_batch_scan_needs_no_cluster(host, net):
    """Nor does it wait for four SMs at a time behind the blocks of another thread's scan."""
    forms = []
    busy = []

    def waiting():
        if not busy:
            busy.append(1)
            forms.append(net.forward())
            busy.pop()
    hook = C.CFUNCTYPE(None)(waiting)
    with ct.Context(0) as ctx:
        host.fake_during_wait(hook)
        ctx.trace_batch(ct.make_job(50.0, 15.0, **JOB), params())
        host.fake_during_wait(None)
    assert 1 in forms and net.forward() == 4


@pytest.mark.parametrize("depends", [False, True])
def test_stream_launch_waits_for_clusters(host, net, depends):
    """A stream that starts in another thread while a network call runs in
    clusters lets them finish first; but not for ever, in case the network call
    waits for what the stream is to do."""
    import threading
    seen, started, threads = [], threading.Event(), []
    with ct.Context(0) as ctx, small_stream(ctx) as st:
        def start():
            st.submit(ct.make_job(50.0, 15.0, **JOB), params())
            started.set()

        def waiting():
            if threads:
                return
            threads.append(threading.Thread(target=start))
            threads[0].start()
            started.wait(20.0 if depends else 0.3)
            seen.append(any("stream_kernel" in k for k, _ in launched(host)))
        hook = C.CFUNCTYPE(None)(waiting)
        host.fake_during_wait(hook)
        net.forward()
        threads[0].join()
        host.fake_during_wait(None)
        assert seen == [depends] and started.is_set()
        assert net.forward() == 1


def test_network_where_no_cluster_fits(host):
    """A part of a GPU with fewer than four SMs."""
    host.fake_fail_call(b"cudaOccupancyMaxActiveClusters", 1)
    net = Network(host)
    assert (net.forward(), net.train()) == (1, 1)
    net.close()


@pytest.mark.parametrize("models", TEAM_SETS)
@pytest.mark.parametrize("n", [1, 20, 400])
def test_teams_beside_a_stream_are_full(host, models, n):
    """A free device takes a trajectory or a point to a block while it has room
    for the blocks; on the SMs that a stream reserves they would run one after
    the other."""
    with ct.Context(0) as a, ct.Context(0) as b, small_stream(a) as st:
        def blocks():
            scan(b, n, models)
            b.field_batch(points(n), params(1), ct.model_set(*models))
            return [g for k, g in launched(host) if "team_" in k][-2:]
        free = blocks()
        st.submit(ct.make_job(50.0, 15.0, **JOB), params())
        beside = blocks()
        st.drain()
        assert blocks() == free and min(free) >= min(n, 100)
        assert max(beside) <= (n + 15) // 16        # 16 slots, the fewest of a full block


@pytest.mark.parametrize("models", TEAM_SETS + [(1, 0, 1)])
@pytest.mark.parametrize("first", [lambda c, m: scan(c, 100000, m), lambda c, m: scan(c, 1, m),
                                   lambda c, m: c.field_batch(points(40000), params(1), ct.model_set(*m)),
                                   lambda c, m: c.field_batch(points(1), params(1), ct.model_set(*m)),
                                   lambda c, m: ct.Stream(c, ct.model_set(*m), slots=1, max_jobs=1,
                                                          max_trajectories=8).close()],
                         ids=["large scan", "small scan", "large field", "small field", "stream"])
def test_first_use_of_a_set_loads_its_kernels(host, models, first):
    """Loading a kernel may wait for a scan stream that is running (until it is
    drained), so a set's kernels are all loaded by the first call, whatever the
    sizes of the later ones."""
    with ct.Context(0) as ctx:
        first(ctx, models)
        for n in (1, 20000, 100000):
            scan(ctx, n, models)
        for n in (1, 40000):
            ctx.field_batch(points(n), params(1), ct.model_set(*models))
        own = [k for k, _ in launched(host) if "trace_kernel" in k or "field_kernel" in k]
        assert len(set(own)) >= (2 if models[2] else 4)
        assert host.fake_loaded_by_launch(b"trace_kernel") == host.fake_loaded_by_launch(b"field_kernel") == 0


def test_large_field_batch_takes_what_it_needs_and_gives_it_back(host):
    """Buffers kept between calls are those of small batches: a large one needs
    48 bytes of device memory a point and no more, and leaves none behind."""
    n = 4_000_000
    with ct.Context(0) as ctx:
        ctx.field_batch(points(21), params())
        kept = host.fake_in_use()
        host.fake_memory(kept + 48 * n + 1_000_000)
        ctx.field_batch(points(n), params())
        assert host.fake_in_use() < kept + 48 * n // 100
        ctx.field_batch(points(n), params())
        ctx.field_batch(points(21), params())
