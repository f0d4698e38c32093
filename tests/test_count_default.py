"""The default policy on symmetric graphs: the single-kernel count of small graphs and the
degree-ordered count of larger ones, against the oracle's counts and the statistics of
the ratio-50 rule.  Counts are whole numbers: equal or wrong."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle

SMALL_M = 1 << 17  # entries up to which one kernel counts


def _csr(n, u, v):
    keep = u != v
    u, v = u[keep].astype(np.int64), v[keep].astype(np.int64)
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    return np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)


def _rule_stats(off, dst):
    """Edges, probe and owner elements per kind of the ratio-50 rule (owner = larger degree)."""
    deg = np.diff(off).astype(np.int64)
    src = np.repeat(np.arange(len(deg)), deg)
    own = (deg[src] > deg[dst]) | ((deg[src] == deg[dst]) & (src < dst))
    du, dv = deg[src][own], deg[dst][own]
    gal = 50 * dv < du
    return {k: (int(m.sum()), int(dv[m].sum()), int(du[m].sum())) for k, m in (("merge", ~gal), ("gallop", gal))}


def _check(off, dst, relabel=False):
    ref = oracle.cn_count(off, dst, nthreads=16)
    G = accx.Graph.from_csr(off, dst)
    if relabel:
        G.relabel()
    for bias in (2, 0):
        assert np.array_equal(G.count(bias=bias), ref - 2 + bias)
    st, ow = G.last_stats(), G.owner_work()
    for k, (e, w, o) in _rule_stats(off, dst).items():
        assert (st[k]["edges"], st[k]["work"], ow[k]) == (e, w, o), k
    assert st["bitmap"]["edges"] == 0
    # without the symmetry check the kinds' own kernels run
    H = accx.Graph.from_csr(off, dst, validate=False)
    assert np.array_equal(H.count(bias=2), ref)


@pytest.mark.parametrize("n,mean", [(2, 1), (70, 3), (1000, 20), (4000, 30), (8600, 30), (9000, 30), (40000, 12)])
def test_random(n, mean):
    rng = np.random.default_rng(n)
    k = n * mean // 2
    _check(*_csr(n, rng.integers(0, n, k), rng.integers(0, n, k)))


# |F| around the warps' 32 and 128 ids and the CTA's 1024, a graph past
# the single kernel's size
@pytest.mark.parametrize("hubs", [31, 33, 34, 63, 65, 127, 130, 600, 1023, 1025, 2200])
def test_cliques_with_leaves(hubs):
    rng = np.random.default_rng(hubs)
    a, b = np.triu_indices(hubs, 1)
    leaves = 6000
    k = 40 * leaves
    n = hubs + leaves
    off, dst = _csr(n, np.concatenate([a, rng.integers(hubs, n, k)]), np.concatenate([b, rng.integers(0, n, k)]))
    p = rng.permutation(n)
    src = np.repeat(np.arange(n), np.diff(off))
    off, dst = _csr(n, p[src], p[dst])
    assert len(dst) > SMALL_M
    _check(off, dst)


@pytest.mark.parametrize("leaves", [58, 60, 61, 124, 125, 1020, 1025, 70000])
def test_stars(leaves):
    rng = np.random.default_rng(leaves)
    hubs = 5
    u = np.repeat(np.arange(hubs), leaves)
    v = hubs + np.tile(np.arange(leaves), hubs)
    a, b = np.triu_indices(hubs, 1)
    extra = rng.integers(hubs, hubs + leaves, (2, leaves // 2))
    _check(*_csr(hubs + leaves, np.concatenate([u, a, extra[0]]), np.concatenate([v, b, extra[1]])))


@pytest.mark.parametrize("scale", [8, 12, 14, 16])
def test_rmat_relabeled_too(scale):
    G = accx.Graph.generate(accx.rmat_params(scale, 16, seed=scale))
    off, dst = G.download()
    _check(off, dst)
    _check(off, dst, relabel=True)


# graphs whose ids need 25 and 26 bits
@pytest.mark.parametrize("n", [(1 << 24) + 1, (1 << 25) - 1, 1 << 25])
def test_wide_ids(n):
    rng = np.random.default_rng(n)
    us, vs = [], []
    for c in (33, 129, 130):  # cliques of the highest ids and of random ones: |F| up to 32, 128, 129
        for ids in (np.arange(n - c, n), np.sort(rng.choice(n, c, replace=False))):
            a, b = np.triu_indices(c, 1)
            us.append(ids[a])
            vs.append(ids[b])
    pool = np.concatenate([rng.choice(n, 4000, replace=False), np.arange(n - 500, n)])
    us.append(rng.choice(pool, 150000))
    vs.append(rng.choice(pool, 150000))
    off, dst = _csr(n, np.concatenate(us), np.concatenate(vs))
    assert len(dst) > SMALL_M
    _check(off, dst)
