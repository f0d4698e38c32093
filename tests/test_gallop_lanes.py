"""Galloping edges by a lane each (many edges, short partner lists) and by groups (few edges),
around the number of edges where they change hands, with partner lists around the lane's 32
ids and owners much longer, against the oracle's counts."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle

FEW = 196608


def _check(n, u, v):
    keep = u != v
    u, v = u[keep].astype(np.int64), v[keep].astype(np.int64)
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    off, dst = np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)
    ref = oracle.cn_count(off, dst, nthreads=16)
    lanes = 0
    for relabel in (False, True):
        G = accx.Graph.from_csr(off, dst)
        if relabel:
            G.relabel()
        assert np.array_equal(G.count(policy="gallop", bias=2, orient=True), ref)
        matches, _ = G.last_matches()
        assert matches["gallop"] == (int(ref.sum()) - 2 * len(ref)) // 6
        st = G.last_stats()["gallop"]
        lanes += st["edges"] >= FEW and st["work"] <= 24 * st["edges"]
    return lanes


@pytest.mark.parametrize("edges", [150000, 196000, 198000, 205000, 400000])
@pytest.mark.parametrize("n", [20000, 60000])
def test_random(edges, n):
    rng = np.random.default_rng(edges + n)
    lanes = _check(n, rng.integers(0, n, edges), rng.integers(0, n, edges))
    assert lanes == 0 if edges < FEW else edges < 250000 or lanes == 2


# leaves of p hubs among many short rows: the lane's longest lists, the groups' shortest, owners
# more than eight times as long
@pytest.mark.parametrize("p", [2, 8, 31, 32, 33])
def test_skewed(p):
    rng = np.random.default_rng(p)
    hubs, leaves, n = 600, 2500, 60000
    a, b = np.triu_indices(hubs, 1)
    keep = rng.random(len(a)) < 0.5
    lu = np.repeat(hubs + np.arange(leaves), p)
    lv = np.concatenate([rng.permutation(hubs)[:p] for _ in range(leaves)])
    bu, bv = rng.integers(hubs + leaves, n, (2, 420000))
    bv = np.where(rng.random(len(bv)) < 0.3, bu + rng.integers(1, 5, len(bu)), bv).clip(max=n - 1)
    hu, hv = np.repeat(np.arange(hubs), 60), rng.integers(hubs + leaves, n, 60 * hubs)
    u, v = np.concatenate([a[keep], lu, bu, hu]), np.concatenate([b[keep], lv, bv, hv])
    assert _check(n, u, v) >= 1
