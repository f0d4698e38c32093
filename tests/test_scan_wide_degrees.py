"""Similarity of entries whose degrees and common neighbours need more than a float's 24 bits:
two hubs joined to 2^24 and more common leaves, at thresholds next to the entries' own
ratios, against the predicate's exact form."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle

N = 1 << 24  # common leaves


@pytest.fixture(scope="module")
def graph():
    own = 5001  # leaves of the second hub alone
    n = 2 + N + own
    common = np.arange(2, 2 + N, dtype=np.int32)
    row0 = np.concatenate([[1], common])
    row1 = np.concatenate([[0], common, np.arange(2 + N, n)])
    dst = np.concatenate([row0, row1, np.tile([0, 1], N), np.ones(own)]).astype(np.int32)
    deg = np.concatenate([[len(row0), len(row1)], np.full(N, 2), np.ones(own)]).astype(np.int64)
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    G = accx.Graph.from_csr(off, dst)
    cnt = G.count(bias=2)
    # one entry of every kind: hub-hub, hub-leaf of either hub, both ways, hub-own leaf
    e = np.array([0, 1, len(row0), len(row0) + 1, len(row0) + len(row1), len(row0) + len(row1) + 1, len(row0) + len(row1) - 1,
                  len(dst) - 1])
    src = np.array([0, 0, 1, 1, 2, 2, 1, n - 1])
    want = np.array([N, 1, N, 1, 1, 1, 0, 0]) + 2
    assert np.array_equal(cnt[e], want)
    kind = np.concatenate([[0], np.full(N, 1), [2], np.full(N, 3), np.full(own, 6), np.tile([4, 5], N), np.full(own, 7)]).astype(np.uint8)
    return G, kind, want, deg[src] + 1, deg[dst[e]] + 1


def test_thresholds(graph):
    G, kind, c, du, dv = graph
    x = c / np.sqrt(du.astype(np.float64) * dv)
    assert (du.max() >= N) and (c.max() > N)
    eps = set()
    for r in np.unique(x):
        for rel in (1e-3, 1e-5, 1e-6, 3e-7, 1e-7, 1e-8, 1e-12, 0.0):
            eps.update((float(r * (1 + rel)), float(r * (1 - rel))))
        eps.update((float(np.nextafter(r, 0)), float(np.nextafter(r, 2))))
    for e in sorted(eps):
        ref = oracle.sim_batch(c, du, dv, e)
        assert np.array_equal(ref, accx.similar_exact_batch(c, du, dv, e))
        r = G.scan(e, 2, want_label=False, want_cluster=False)
        assert np.array_equal(r["sim"].astype(bool), np.asarray(ref, bool)[kind]), e
