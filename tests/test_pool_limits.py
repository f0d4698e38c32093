"""Calls that run out of device memory, in a child process whose device pool has a size limit:
each says so, leaves the handle usable, and answers right when called again with and
without room.  Answers are compared with the oracle's."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
LIMIT = 256 << 20

class Loc(C.Structure):
    _fields_ = [("type", C.c_int), ("id", C.c_int)]

class Props(C.Structure):
    _fields_ = [("alloc", C.c_int), ("handles", C.c_int), ("loc", Loc), ("sec", C.c_void_p), ("max_size", C.c_size_t),
                ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]

cu = C.CDLL("libcuda.so.1")
def ok(r):
    assert r == 0, r
dev, ctx, pool = C.c_int(), C.c_void_p(), C.c_void_p()
ok(cu.cuInit(0)); ok(cu.cuDeviceGet(C.byref(dev), 0))
ok(cu.cuDevicePrimaryCtxRetain(C.byref(ctx), dev)); ok(cu.cuCtxSetCurrent(ctx))
ok(cu.cuMemPoolCreate(C.byref(pool), C.byref(Props(1, 0, Loc(1, 0), None, LIMIT, 0))))
ok(cu.cuMemPoolSetAttribute(pool, 4, C.byref(C.c_uint64(2 ** 64 - 1))))  # the release threshold
ok(cu.cuDeviceSetMemPool(dev, pool))

def used():
    ok(cu.cuCtxSynchronize())
    v = C.c_uint64()
    ok(cu.cuMemPoolGetAttribute(pool, 7, C.byref(v)))
    return v.value

def take(size):
    p = C.c_uint64()
    r = cu.cuMemAllocFromPoolAsync(C.byref(p), C.c_size_t(size), pool, None)
    ok(cu.cuCtxSynchronize())
    return p if r == 0 else None

def leave(room):
    "Takes blocks until about `room` bytes of the pool are free."
    held, size = [], LIMIT
    while size >= 1 << 16:
        free = LIMIT - used() - room
        p = take(size) if free >= size else None
        if p:
            held.append(p)
        else:
            size //= 2
    return held

def give(held):
    for p in held:
        ok(cu.cuMemFreeAsync(p, None))
    ok(cu.cuCtxSynchronize())

from acctricnt_gb300 import accx
from oracle import oracle

def sweep(prep, op, check, rooms):
    "Calls op with less and less taken: right or out of memory, twice, then right with all the room."
    seen = set()
    base = used()
    for room in rooms:
        g = prep()
        held = leave(room)
        for _ in range(2):
            try:
                check(op(g))
                seen.add("right")
            except accx.AccxError as e:
                assert e.status == accx.ERR_OOM, (room, e)
                seen.add("oom")
        give(held)
        check(op(g))
        g.free()
        assert used() == base, (room, used(), base)
    assert seen == {"right", "oom"}, seen
    print(sorted(seen))

off, dst = accx.generate_host(accx.rmat_params(14, 16, seed=3))
assert len(dst) > 1 << 17
ref = oracle.scan(off, dst, 0.3, 3)

def graph(**count):
    g = accx.Graph.from_csr(off, dst)
    if count:
        g.count(out=None, **count)
    return g

def same_scan(r):
    for k in ("sim", "label", "cluster"):
        assert np.array_equal(r[k], ref[k]), k

def same_counts(c):
    assert np.array_equal(c, ref["cnn"])

ROOMS = [k << 18 for k in range(0, 100, 3)]
"""


def _child(code):
    r = subprocess.run([sys.executable, "-c", CHILD + code, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_query_keys():
    _child("sweep(lambda: graph(policy='gallop', bias=2), lambda g: g.scan(0.3, 3), same_scan, ROOMS)\n")


@pytest.mark.parametrize("kw", ["dict()", "dict(policy='bitmap')", "dict(policy='merge')",
                                "dict(policy='bitmap', orient=True)", "dict(policy='merge', orient=True)"])
def test_counts(kw):
    _child("sweep(graph, lambda g: g.count(bias=2, **%s), same_counts, ROOMS)\n" % kw)


def test_relabel_and_count():
    _child("""
def op(g):
    g.relabel()
    return g.count(policy='bitmap', bias=2, orient=True)
sweep(graph, op, same_counts, ROOMS)
""")


# the default policy's count of a larger graph keeps lists for the next one: what a query, an
# oriented count or a relabel of the same graph needs after it may take their place
@pytest.mark.parametrize("op,check", [
    ("lambda g: g.scan(0.3, 3)", "same_scan"),
    ("lambda g: g.count(policy='merge', bias=2, orient=True)", "same_counts"),
    ("lambda g: (g.relabel(), g.count(policy='bitmap', bias=2, orient=True))[1]", "same_counts")])
def test_lists_of_the_default_count_are_given_back(op, check):
    _child("""
op, check = %s, %s
STEP = 1 << 18
def least(**kw):
    "after a count: what it took, and the smallest room (in steps) beside it at which op answers"
    base = used()
    for k in range(400):
        g = graph()
        b = used()
        g.count(out=None, bias=2, **kw)
        took = used() - b
        held = leave(k * STEP)
        try:
            check(op(g))
            done = True
        except accx.AccxError as e:
            assert e.status == accx.ERR_OOM
            done = False
        give(held)
        check(op(g))
        same_counts(g.count(bias=2))
        g.free()
        assert used() == base
        if done:
            return took, k
    assert False
took, room = least(policy='gallop')
took2, room2 = least()
lists = (took2 - took) // STEP
print(room, room2, lists)
assert lists * STEP > 7 * len(dst)  # two words an entry and more
assert room2 <= max(0, room - lists) + 2, (room, room2, lists)
""" % (op, check))


def test_captured_lists_stay():
    _child("""
import torch
g = graph(bias=2)
before = used()
s = torch.cuda.Stream()
torch.cuda.synchronize()
cg = torch.cuda.CUDAGraph()
with torch.cuda.graph(cg, stream=s):
    g.count(bias=2, out=None, stream=s.cuda_stream)
held = leave(1 << 16)
for op in (lambda: g.scan(0.3, 3), lambda: g.count(policy='merge', bias=2, orient=True), lambda: g.relabel()):
    try:
        op()
        assert False
    except accx.AccxError as e:
        assert e.status == accx.ERR_OOM
g2 = g.count(policy='gallop', bias=9)
assert np.array_equal(g2, ref["cnn"] + 7)
cg.replay()
torch.cuda.synchronize()
same_counts(g.read_counts())
give(held)
g.count(bias=2, out=None)  # the handle's bias is the last count's, not the replay's
same_scan(g.scan(0.3, 3))
""")


def test_query_and_pairs():
    _child("""
def op(g):
    r = g.scan(0.3, 3)
    r["pairs"] = g.pairs()
    return r
want = graph(bias=2)
want.scan(0.3, 3)
pairs = want.pairs()
def check(r):
    same_scan(r)
    assert np.array_equal(r["pairs"], pairs)
sweep(lambda: graph(policy='gallop', bias=2), op, check, ROOMS)
""")


def test_edge_lists_with_an_id_out_of_range():
    """Named as such wherever the keys themselves fit, also where their sort does not."""
    _child("""
n = len(off) - 1
src = np.repeat(np.arange(n), np.diff(off)).astype(np.uint32)
bad = dst.astype(np.uint32).copy()
bad[len(bad) // 3] = n
block = 4 * 2 * len(src) + 2 * 4 * len(src)  # 32-bit keys of both directions, the two lists
base = used()
good = {}
for room in [k << 18 for k in range(0, 120, 2)]:
    held = leave(room)
    for what, d in (("good", dst.astype(np.uint32)), ("bad", bad)):
        try:
            g = accx.Graph.from_edges(src, d, n)
            assert what == "good"
            o, a = g.download()
            assert np.array_equal(o, off) and np.array_equal(a, dst)
            g.free()
            good[room] = True
        except accx.AccxError as e:
            assert e.status in ((accx.ERR_OOM,) if what == "good" else (accx.ERR_OOM, accx.ERR_RANGE)), (room, e)
            if what == "good":
                good[room] = False
            elif room > block + (2 << 20):
                assert e.status == accx.ERR_RANGE, (room, block)
    give(held)
    assert used() == base
assert any(not v and r > block + (2 << 20) for r, v in good.items())  # rooms where only the sort does not fit
assert good[max(good)]
""")
