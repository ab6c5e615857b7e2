"""The order of rows_kernel's products (csrc/mlp.cu, csrc/mlp_schedule.h), as a
graph of what happens before what: the waits of the issuing thread, the
epilogue warps, and the copies between the CTAs of a cluster.  Every read of
the accumulator and of an operand block has to come before whatever writes
there next, along waits and not by luck.  On the CPU."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

WARPS = 16


@pytest.fixture(scope="module")
def schedule(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("order") / "print_schedule")
    src = os.path.join(ROOT, "tests", "network_order", "print_schedule.cpp")
    r = subprocess.run(["g++", "-std=c++17", src, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    s = {"product": [], "owner": {}, "waits": {}, "sets": {}}
    for ln in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines():
        k, *v = ln.split()
        v = [int(x) for x in v]
        if k == "products":
            s["fwd"], s["all"] = v
        elif k == "product":
            s["product"].append(tuple(v))
        elif k == "sets":
            s["sets"][v[0]] = v[1]
        elif k == "owner":
            s["owner"][v[0], v[1]] = v[2]
        else:
            s["waits"].setdefault((v[0], v[1], v[2]), []).append(v[3])
    return s


class Order:
    """Events and their edges; before(a, b) along the edges."""

    def __init__(self):
        self.out = {}

    def edge(self, a, b):
        self.out.setdefault(a, set()).add(b)
        self.out.setdefault(b, set())

    def close(self):
        indeg = {n: 0 for n in self.out}
        for n in self.out:
            for m in self.out[n]:
                indeg[m] += 1
        todo, order = [n for n in indeg if indeg[n] == 0], []
        while todo:
            n = todo.pop()
            order.append(n)
            for m in self.out[n]:
                indeg[m] -= 1
                if indeg[m] == 0:
                    todo.append(m)
        assert len(order) == len(self.out), "a wait that never ends"
        self.bit = {n: i for i, n in enumerate(order)}
        self.reach = {}
        for n in reversed(order):
            r = 1 << self.bit[n]
            for m in self.out[n]:
                r |= self.reach[m]
            self.reach[n] = r

    def before(self, a, b):
        return a in self.bit and b in self.bit and (self.reach[a] >> self.bit[b]) & 1 == 1


def conflicts(s, split, train, waits, sets):
    """The pairs (a read, the write that has to wait for it) that no chain of
    waits orders, for one tile of `split` CTAs."""
    last = s["all"] if train else s["fwd"]
    own = {r: [b for b in range(4) if s["owner"][split, b] == r] for r in range(split)}
    o = Order()
    reader = {}                              # exchange -> the product that reads it
    for p in range(last):
        if s["product"][p][1] >= 0:
            reader[s["product"][p][1]] = p
    hidden = [p for p in range(last - 1) if p != 4]
    for c in range(split):
        prev = None
        for p in range(last):
            blocks, x, _ = s["product"][p]
            for kb in range(blocks):
                e = ("issue", c, p, kb)
                if prev:
                    o.edge(prev, e)
                if x < 0:
                    for w in range(WARPS):
                        o.edge(("local", c, p, w), e)
                else:
                    for b in waits(c, kb):
                        o.edge(("ready", c, x, b), e)
                prev = e
            o.edge(prev, ("done", c, p))     # the commit: every issued product is complete
        for w in range(WARPS):
            at = ("local", c, 0, w)          # the input
            for p in range(last):
                o.edge(("done", c, p), ("read", c, p, w, 0))
                if p == 4:                   # the output layer: the loss, dY into the single block
                    o.edge(at, ("read", c, p, w, 0))
                    at = ("read", c, p, w, 0)
                    if train:
                        o.edge(at, ("put1", c, p, w))
                        o.edge(("put1", c, p, w), ("local", c, 5, w))
                        at = ("local", c, 5, w)
                    continue
                for i, b in enumerate(own[c]):
                    o.edge(at, ("read", c, p, w, i))
                    o.edge(("read", c, p, w, i), ("put", c, p, w, b))
                    at = ("put", c, p, w, b)
                    if p in hidden:
                        o.edge(at, ("ready", c, s["product"][p][2], b))
        for p in hidden:
            x = s["product"][p][2]
            for b in own[c]:
                for r in range(split):
                    if r != c:
                        o.edge(("ready", c, x, b), ("send", c, x, b))
                        o.edge(("send", c, x, b), ("ready", r, x, b))
    o.close()
    bad = []

    def need(a, b):
        if a in o.bit and b in o.bit and not o.before(a, b):
            bad.append((a, b))
    for c in range(split):
        for p in range(last):
            for w in range(WARPS):
                for i in range(len(own[c])):
                    # the accumulator: read by product p's epilogue, written by product p + 1
                    need(("read", c, p, w, i), ("issue", c, p + 1, 0))
        for x, p in reader.items():
            for b in range(4):
                # operand block b of exchange x: read by product p, and by the copies out of it
                k = s["owner"][split, b]
                if k == c:
                    writes = [("put", c, q, w, b) for q in range(last) if q != 4 and s["product"][q][2] == x + sets
                              for w in range(WARPS)]
                else:
                    writes = [("send", k, x + sets, b)]
                for wr in writes:
                    need(("done", c, p), wr)
                    if k == c:
                        for r in range(split):
                            if r != c:
                                need(("ready", r, x, b), wr)
                # a barrier's phase is taken before the next one ends
                need(("issue", c, p, b), ("ready", c, x + sets, b))
        for w in range(WARPS):
            need(("done", c, 0), ("put1", c, 4, w))
    return bad


@pytest.mark.parametrize("split", [1, 4])   # CTAs of a cluster
@pytest.mark.parametrize("train", [False, True])
def test_every_read_comes_before_the_next_write(schedule, split, train):
    assert conflicts(schedule, split, train, lambda c, kb: schedule["waits"][split, c, kb], schedule["sets"][split]) == []


@pytest.mark.parametrize("train", [False, True])
def test_the_model_finds_a_missing_wait(schedule, train):
    """With only the block that the product reads waited for, a CTA of rank 1 to
    3 overwrites the accumulator that its own warps may still read; with room for
    one exchange, a peer's copy lands on an operand in use."""
    bad = conflicts(schedule, 4, train, lambda c, kb: [kb], 2)
    assert {a[1] for a, _ in bad if a[0] == "read"} == {1, 2, 3}
    bad = conflicts(schedule, 4, train, lambda c, kb: schedule["waits"][4, c, kb], 1)
    assert any(a[0] == "done" and b[0] == "send" for a, b in bad)
    # a CTA alone, too, waits for all of its blocks before the first product
    assert conflicts(schedule, 1, train, lambda c, kb: [kb], 1)


def test_weight_gradient_epilogue_decides_as_one():
    """grad_kernel's epilogue warps wait with a limit each and meet at a barrier
    of all 256 threads: whether to go on has to be one decision, taken by a
    barrier of the same threads, or warps whose wait ran out would leave the
    others at theirs."""
    with open(os.path.join(ROOT, "cor-model_gb300", "csrc", "mlp.cu")) as f:
        src = f.read()
    kernel = src[src.index("grad_kernel(const GradArgs g) {"):src.index("// Every weight into its BF16 copies")]
    waits = kernel.index("mbar_wait(&accb")
    assert 0 <= kernel.rindex("epilogue_agrees(", 0, waits + 1) < waits < kernel.index("bar.sync 1")
    helper = src[src.index("bool epilogue_agrees"):src.index("// One tile of a weight gradient")]
    assert "bar.red.and.pred q, 1, 256, p" in helper and "kGradThreads = 32 * 10" in src
    # the row kernel's warps share no barrier between their waits
    rows = src[src.index("rows_kernel(const RowsArgs g) {"):src.index("// ---- weight gradients and AdamW")]
    assert "bar.sync" not in rows and "bar.red" not in rows


def test_a_tile_that_gave_up_waits_out_what_it_issued():
    """Where a wait ran out, copies to and from the peers and products into the
    accumulator may be in flight that nobody waits for any more: every CTA of the
    tile hears of it before it leaves, lets them end, and frees its tensor
    memory after that."""
    with open(os.path.join(ROOT, "cor-model_gb300", "csrc", "mlp.cu")) as f:
        src = f.read()
    rows = src[src.index("rows_kernel(const RowsArgs g) {"):src.index("// ---- weight gradients and AdamW")]
    steps = ["sh.failed = 0;", "tile_sync<SPLIT>();", "__syncthreads_or(!ok)", "st.shared::cluster.u32", "tile_sync<SPLIT>();",
             "sh.failed)", "settle();", "tile_sync<SPLIT>();", "tcgen05.dealloc"]
    at = 0
    for k in steps:
        at = rows.index(k, at) + len(k)
    assert "tile_sync" not in rows[at:]
    grad = src[src.index("grad_kernel(const GradArgs g) {"):src.index("// Every weight into its BF16 copies")]
    assert grad.index("__syncthreads_or(!ok)") < grad.index("settle();") < grad.index("tcgen05.dealloc")
