"""The SCAN query's kernels where their work changes hands, against the oracle: entry
counts around whole words, rows around the CTA's and the push slices' lengths, several
clusters with hubs between them, thresholds on and next to entries' own ratios, and
similarity bytes into device memory of any alignment."""
import ctypes

import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    import torch
    from acctricnt_gb300 import accx
    from oracle import oracle


def _csr(n, u, v):
    keep = u != v
    u, v = u[keep].astype(np.int64), v[keep].astype(np.int64)
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    return np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)


def _check(off, dst, queries):
    G = accx.Graph.from_csr(off, dst)
    G.count(bias=2)
    for eps, mu in queries:
        ref = oracle.scan(off, dst, eps, mu, nthreads=8)
        r = G.scan(eps, mu)
        for k in ("sim", "label", "cluster"):
            assert np.array_equal(r[k], ref[k]), (k, eps, mu)
        assert r["summary"]["similar_entries"] == int(ref["sim"].sum())
        for shift in (0, 1, 4):  # device outputs; only the first allows 8-byte stores
            sim = torch.full((G.m + 16,), 7, dtype=torch.uint8, device="cuda")
            cl = torch.empty(max(G.n, 1), dtype=torch.int32, device="cuda")
            st = accx.lib.accx_scan_query(G._h, eps, mu, ctypes.c_void_p(sim.data_ptr() + shift), None,
                                          ctypes.c_void_p(cl.data_ptr()), None, None)
            assert st == accx.OK
            got = sim.cpu().numpy()
            assert np.array_equal(got[shift:shift + G.m], ref["sim"])
            assert (got[:shift] == 7).all() and (got[shift + G.m:] == 7).all()
            assert np.array_equal(cl.cpu().numpy()[:G.n], ref["cluster"])


@pytest.mark.parametrize("edges", [1, 2, 3, 4, 5, 15, 16, 17, 127, 128, 129, 1024])
def test_word_edges(edges):
    rng = np.random.default_rng(edges)
    n = 64
    a, b = np.triu_indices(n, 1)
    p = rng.permutation(len(a))[:edges]
    _check(*_csr(n, a[p], b[p]), [(0.2, 1), (0.5, 2), (0.9, 3)])


@pytest.mark.parametrize("leaves", [254, 256, 257, 511, 513, 1025, 4094, 4096, 4098])
def test_row_lengths(leaves):
    """Two joined hubs whose rows have about `leaves` entries, cores at a low threshold."""
    n = leaves + 3
    hubs = np.array([0, 1])
    u = np.concatenate([np.repeat(hubs, leaves), [0]])
    v = np.concatenate([np.tile(np.arange(3, leaves + 3), 2), [1]])
    _check(*_csr(n, u, v), [(0.01, 1), (0.01, 100), (0.02, 3), (0.5, 2)])


@pytest.mark.parametrize("cliques,size", [(3, 40), (40, 9), (2, 700)])
def test_clusters_and_hubs(cliques, size):
    rng = np.random.default_rng(size)
    us, vs = [], []
    for c in range(cliques):
        a, b = np.triu_indices(size, 1)
        us.append(a + c * size)
        vs.append(b + c * size)
    n0 = cliques * size
    n = n0 + 50  # outsiders: joined to one clique, or to two (hubs)
    for i in range(50):
        k = 1 + i % 2
        t = rng.choice(cliques, size=min(k, cliques), replace=False) * size
        us.append(np.full(len(t), n0 + i))
        vs.append(t + rng.integers(0, size, len(t)))
    p = rng.permutation(n)
    _check(*_csr(n, p[np.concatenate(us)], p[np.concatenate(vs)]), [(0.3, 3), (0.7, 2), (0.95, 5), (0.05, 2)])


def test_thresholds_at_ratios():
    """eps equal to entries' own ratios and their neighbouring doubles: the keys' band."""
    G = accx.Graph.generate(accx.rmat_params(11, 16, seed=3))
    off, dst = G.download()
    cnn = oracle.cn_count(off, dst, nthreads=8)
    deg = np.diff(off).astype(np.int64) + 1
    src = np.repeat(np.arange(len(deg)), np.diff(off))
    x = (cnn / np.sqrt((deg[src] * deg[dst]).astype(np.longdouble))).astype(np.float64)
    rng = np.random.default_rng(1)
    eps = [e for t in rng.choice(np.unique(x[x < 1]), 12) for e in (np.nextafter(t, 0), t, np.nextafter(t, 1))]
    _check(off, dst, [(float(e), 3) for e in eps])
