"""Relabeled rows at the lengths where their sort changes, with ids of few and of many
bits (a word of neighbour and place, or a pair), against numpy."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle


@pytest.mark.parametrize("spare", [0, 1 << 20, (1 << 24) - 30000, 1 << 25])
def test_row_lengths(spare):
    rng = np.random.default_rng(spare + 1)
    us, vs, c = [], [], 0
    pool = 9000
    lens = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 4095, 4096, 4097, 8999]
    for d in lens * 2:  # centres of that many neighbours in a common pool
        us.append(np.full(d, c))
        vs.append(len(lens) * 2 + rng.permutation(pool)[:d])
        c += 1
    n = len(lens) * 2 + pool + spare  # the rest are isolated: they only widen the ids
    u, v = np.concatenate(us), np.concatenate(vs)
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    off = np.searchsorted(k, np.arange(n + 1, dtype=np.int64) * n).astype(np.uint32)
    dst = (k % n).astype(np.int32)
    G = accx.Graph.from_csr(off, dst)
    G.relabel()
    roff, rdst, rmap, oldid = (x.astype(np.int64) for x in G.relabeled_csr())
    deg = np.diff(off.astype(np.int64))
    assert np.array_equal(oldid, np.lexsort((np.arange(n), -deg)))
    newid = np.empty(n, np.int64)
    newid[oldid] = np.arange(n)
    src = np.repeat(np.arange(n), deg)
    order = np.lexsort((newid[dst], newid[src]))
    assert np.array_equal(roff, np.concatenate([[0], np.cumsum(deg[oldid])]))
    assert np.array_equal(rdst, newid[dst][order])
    ref = np.empty(len(dst), np.int64)
    ref[order] = np.arange(len(dst))
    assert np.array_equal(rmap, ref)


# the reverse index of suffix entries: tiles of 256 entries with one row, many rows and
# runs of empty rows, ids that are not relabeled (prefixes of every length)
@pytest.mark.parametrize("n,k,spread", [(2, 1, 1), (3, 3, 1), (40, 300, 1), (256, 9000, 1), (257, 257, 1), (5000, 700, 1),
                                        (600, 900, 1000), (3000, 40000, 7)])
@pytest.mark.parametrize("relabel", [False, True])
def test_reverse_of_suffix_entries(n, k, spread, relabel):
    rng = np.random.default_rng(n + k)
    u, v = rng.integers(0, n, k), rng.integers(0, n, k)
    u[0], v[0] = 0, n - 1
    u, v = u[u != v] * spread, v[u != v] * spread
    N = n * spread
    key = np.unique(np.concatenate([u * N + v, v * N + u]))
    off, dst = np.searchsorted(key, np.arange(N + 1) * N).astype(np.uint32), (key % N).astype(np.int32)
    ref = oracle.cn_count(off, dst, nthreads=4)
    G = accx.Graph.from_csr(off, dst)
    if relabel:
        G.relabel()
    for policy in ("merge", "gallop", "bitmap"):
        assert np.array_equal(G.count(policy=policy, bias=2, orient=True), ref), policy
