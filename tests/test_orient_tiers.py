"""GPU parity of the oriented bitmap kind's tiers at their edges: owners walked by a
warp or by a CTA (prefix lengths around the warp's table, probe work and degree
around its limits), against the oracle's counts.  Counts are whole numbers: equal
or wrong."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle


def _csr(n, u, v):
    keep = u != v
    u, v = u[keep].astype(np.int64), v[keep].astype(np.int64)
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    off = np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32)
    return off, (k % n).astype(np.int32)


def _hubs_and_leaves(hubs, leaf_prefixes, density, seed, satellites=0):
    """`hubs` vertices joined pairwise with probability `density` (each with enough
    satellites to stay ahead of the leaves in degree order), and per entry p of
    leaf_prefixes one vertex joined to p random hubs."""
    rng = np.random.default_rng(seed)
    a, b = np.triu_indices(hubs, 1)
    m = rng.random(len(a)) < density
    us, vs = [a[m]], [b[m]]
    n = hubs
    for p in leaf_prefixes:
        us.append(np.full(p, n))
        vs.append(rng.permutation(hubs)[:p])
        n += 1
    for h in range(hubs):
        us.append(np.full(satellites, h))
        vs.append(np.arange(n, n + satellites))
        n += satellites
    u, v = np.concatenate(us), np.concatenate(vs)
    p = rng.permutation(n)  # the relabel has to find the order
    return _csr(n, p[u], p[v])


def _check(off, dst, **kw):
    ref = oracle.cn_count(off, dst, nthreads=8)
    G = accx.Graph.from_csr(off, dst)
    G.relabel()
    assert np.array_equal(G.count(policy="bitmap", bias=2, orient=True, **kw), ref)
    st = G.last_stats()
    matches, _ = G.last_matches()
    assert sum(matches.values()) == (int(ref.sum()) - 2 * len(ref)) // 6  # every triangle once
    assert sum(s["edges"] for s in st.values()) <= len(dst) // 2


# the warp's table takes 512 prefix ids and 64 to 1024 slots
@pytest.mark.parametrize("p", [1, 2, 15, 16, 17, 31, 32, 33, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513])
def test_prefix_length_edges(p):
    _check(*_hubs_and_leaves(540, [p] * 5 + [p - 1 or 1] * 3, 0.1, seed=p, satellites=60))


# probe work around the light limits (a share of all probes, 4096, 8192): a leaf of p hubs probes about
# p * density * hubs / 2 ids
@pytest.mark.parametrize("density", [0.02, 0.05, 0.1, 0.2, 0.5, 1.0])
def test_probe_work_edges(density):
    _check(*_hubs_and_leaves(256, list(range(1, 257, 5)) * 2, density, seed=11, satellites=40))


# rows around the light owners' 4096 entries: few prefix ids, long suffixes
@pytest.mark.parametrize("sats", [4000, 4090, 4096, 4100])
def test_row_length_edges(sats):
    rng = np.random.default_rng(sats)
    hubs, n = 6, 6
    us, vs = [], []
    for h in range(hubs):
        us.append(np.full(sats, h))
        vs.append(rng.permutation(sats + 200)[:sats] + hubs)
    a, b = np.triu_indices(hubs, 1)
    us.append(a)
    vs.append(b)
    n = hubs + sats + 200
    _check(*_csr(n, np.concatenate(us), np.concatenate(vs)))


@pytest.mark.parametrize("kw", [{"window_kb": 1, "sparse_kb": 1, "block_warps": 4}, {"window_kb": 8, "block_warps": 16},
                                {"window_kb": 64, "sparse_kb": 16, "block_warps": 32}])
def test_shapes(kw):
    G = accx.Graph.generate(accx.chung_lu_params(60000, 20, 2.1, 6000, seed=5))
    off, dst = G.download()
    _check(off, dst, **kw)


# dense rows (hub ids as bit masks): 1024, 2048 and 4096 bits a row by the graph's
# size, every edge of the bitmap kind or only some (tables, few owner counters), rows
# cut by the window, and graphs too small or flat for any
@pytest.mark.parametrize("scale,ef", [(11, 40), (13, 24), (15, 16), (16, 32), (18, 16), (20, 8)])
def test_dense_rows_rmat(scale, ef):
    G = accx.Graph.generate(accx.rmat_params(scale, ef, seed=scale))
    off, dst = G.download()
    ref = oracle.cn_count(off, dst, nthreads=16)
    G.relabel()
    rng = np.random.default_rng(scale)
    for kw in ({"policy": "bitmap"}, {"policy": "bitmap", "sparse_kb": 1}, {"policy": "bitmap", "window_kb": 1},
               {"policy": "table", "table": rng.integers(0, 3, size=(24, 24)).astype(np.uint8)}):
        assert np.array_equal(G.count(bias=2, orient=True, **kw), ref), kw
        matches, _ = G.last_matches()
        assert sum(matches.values()) == (int(ref.sum()) - 2 * len(ref)) // 6, kw


@pytest.mark.parametrize("n,hubs", [(1500, 1023), (1500, 1024), (1500, 1025), (2600, 2049), (5200, 4097)])
def test_dense_rows_around_k(n, hubs):
    """Cliques of hubs around the mask's 1024, 2048 and 4096 ids, with leaves on them:
    counters near their ten bits, rows of every word."""
    rng = np.random.default_rng(hubs)
    a, b = np.triu_indices(hubs, 1)
    m = rng.random(len(a)) < (1.0 if hubs < 1100 else 0.3)
    k = (n - hubs) * 200
    off, dst = _csr(n, np.concatenate([a[m], rng.integers(hubs, n, k)]), np.concatenate([b[m], rng.integers(0, hubs, k)]))
    _check(off, dst)


# galloping edges by lane (partner lists that average up to 24 ids) and by group: sparse
# and dense graphs, partner lists around the lane's 32 ids, owners much longer
@pytest.mark.parametrize("n,mean", [(40, 3), (3000, 6), (3000, 45), (2000, 62), (2000, 66), (1500, 140), (400, 300)])
def test_gallop_random(n, mean):
    rng = np.random.default_rng(n + mean)
    k = n * mean // 2
    off, dst = _csr(n, rng.integers(0, n, k), rng.integers(0, n, k))
    ref = oracle.cn_count(off, dst, nthreads=8)
    for relabel in (False, True):
        G = accx.Graph.from_csr(off, dst)
        if relabel:
            G.relabel()
        assert np.array_equal(G.count(policy="gallop", bias=2, orient=True), ref)
        matches, _ = G.last_matches()
        assert matches["gallop"] == (int(ref.sum()) - 2 * len(ref)) // 6


@pytest.mark.parametrize("p", [1, 3, 8, 31, 32, 33, 40])
def test_gallop_skewed(p):
    """Leaves of p hubs on hubs with long prefixes: the searching side of both kernels."""
    off, dst = _hubs_and_leaves(600, [p] * 900, 0.5, seed=p, satellites=45)
    ref = oracle.cn_count(off, dst, nthreads=8)
    G = accx.Graph.from_csr(off, dst)
    G.relabel()
    assert np.array_equal(G.count(policy="gallop", bias=2, orient=True), ref)


def test_captured_counts_keep_their_indices():
    """A captured count replays with the dense rows it was recorded with whatever windows
    were counted in between; a first oriented count is refused in a capture, and a
    default count that has no room for its lists there falls back."""
    import torch
    G = accx.Graph.generate(accx.rmat_params(16, 32, seed=16))
    B = accx.Batch([G])
    U = B.union
    U.relabel()
    want = U.count(policy="merge", bias=2, orient=True)
    s = torch.cuda.Stream()
    B.capture(policy="bitmap", bias=2, stream=s.cuda_stream, orient=True)
    for kb in (1, 2, 24):
        assert np.array_equal(U.count(policy="bitmap", bias=2, orient=True, window_kb=kb), want)
        U.count(policy="merge", bias=7, out=None)
        torch.cuda.synchronize()
        B.launch(stream=s.cuda_stream)
        s.synchronize()
        assert np.array_equal(U.read_counts(), want)
    for first in ({"policy": "bitmap"}, {"policy": "gallop", "orient": True}):
        H = accx.Graph.generate(accx.rmat_params(16, 32, seed=16))
        off, dst = H.download()
        H = accx.Graph.from_csr(off, dst)
        H.count(bias=2, **first)
        torch.cuda.synchronize()
        cg = torch.cuda.CUDAGraph()
        with torch.cuda.graph(cg, stream=s):
            if "orient" not in first:
                with pytest.raises(accx.AccxError):
                    H.count(policy="bitmap", bias=2, orient=True, out=None, stream=s.cuda_stream)
            H.count(bias=2, out=None, stream=s.cuda_stream)
        cg.replay()
        torch.cuda.synchronize()
        assert np.array_equal(H.read_counts(), want)
        assert np.array_equal(H.count(policy="bitmap", bias=2, orient=True), want)
