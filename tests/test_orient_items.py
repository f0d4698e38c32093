"""The oriented bitmap kind's work items: long lists in short rows, lists concentrated in a
few entries of a row, and every block size, against the oracle's counts."""
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
    return np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)


def _check(off, dst, shapes=({},)):
    ref = oracle.cn_count(off, dst, nthreads=16)
    table = np.random.default_rng(len(dst)).integers(0, 3, size=(24, 24)).astype(np.uint8)
    for relabel in (False, True):
        G = accx.Graph.from_csr(off, dst)
        if relabel:
            G.relabel()
        for kw in shapes:
            assert np.array_equal(G.count(policy="bitmap", bias=2, orient=True, **kw), ref), (relabel, kw)
            matches, _ = G.last_matches()
            assert sum(matches.values()) == (int(ref.sum()) - 2 * len(ref)) // 6, (relabel, kw)
        assert np.array_equal(G.count(policy="table", table=table, bias=2, orient=True), ref), relabel


SHAPES = [{"block_warps": w} for w in (1, 2, 3, 4, 5, 8)] + \
    [{"block_warps": w, "window_kb": 56} for w in (9, 12, 16)] + \
    [{"block_warps": w, "window_kb": 64, "sparse_kb": 16} for w in (17, 24, 32)]


@pytest.mark.parametrize("n,degree", [(300, 250), (1000, 400), (3000, 850), (9000, 250)])
def test_long_lists_in_short_rows(n, degree):
    rng = np.random.default_rng(n)
    k = n * degree // 2
    _check(*_csr(n, rng.integers(0, n, k), rng.integers(0, n, k)), SHAPES)


# every leaf is joined to all hubs and to a few other leaves: only those entries, the last of a
# row, have lists, and they are as long as the row
@pytest.mark.parametrize("hubs", [70, 500, 1990])
@pytest.mark.parametrize("few", [1, 3, 30, 70, 200])
def test_concentrated_lists(hubs, few):
    rng = np.random.default_rng(hubs + few)
    leaves = 700
    u, v = np.repeat(np.arange(hubs), leaves), hubs + np.tile(np.arange(leaves), hubs)
    extra = hubs + rng.integers(0, leaves, (2, few * leaves // 2))
    _check(*_csr(hubs + leaves, np.concatenate([u, extra[0]]), np.concatenate([v, extra[1]])),
           [{}, {"block_warps": 16, "window_kb": 56}, {"block_warps": 32, "window_kb": 64, "sparse_kb": 16}, {"block_warps": 2}])


@pytest.mark.parametrize("size,copies", [(70, 150), (200, 40), (513, 5), (2000, 2)])
def test_cliques(size, copies):
    a, b = np.triu_indices(size, 1)
    base = np.arange(copies)[:, None] * size
    _check(*_csr(size * copies, (base + a).ravel(), (base + b).ravel()), SHAPES[::4])
