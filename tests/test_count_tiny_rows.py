"""The default policy's count of sparse graphs, whose rows a lane walks by itself: F lists and
rows around the lane's limits (4 ids, 16 entries), with and without triangles, against the
oracle's counts."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle


def _check(n, u, v):
    keep = u != v
    u, v = u[keep].astype(np.int64), v[keep].astype(np.int64)
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    off, dst = np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)
    assert len(dst) > 1 << 17  # not the small graphs' kernel
    ref = oracle.cn_count(off, dst, nthreads=16)
    G = accx.Graph.from_csr(off, dst)
    for bias in (2, 0):
        assert np.array_equal(G.count(bias=bias), ref - 2 + bias)


def _copies(u, v, k, n, seed):
    """k disjoint copies of an n-vertex graph, vertices permuted."""
    base = np.arange(k)[:, None] * n
    p = np.random.default_rng(seed).permutation(k * n)
    return k * n, p[(base + u).ravel()], p[(base + v).ravel()]


@pytest.mark.parametrize("size", [3, 4, 5, 6, 7, 16, 17, 18])
def test_cliques(size):
    a, b = np.triu_indices(size, 1)
    _check(*_copies(a, b, 140000 // (size * (size - 1)) + 1, size, size))


# a wheel: one row of `spokes` entries, rim rows of three; a fan with a second hub
@pytest.mark.parametrize("spokes", [3, 4, 14, 15, 16, 17, 18, 40])
@pytest.mark.parametrize("hubs", [1, 2, 3, 5])
def test_wheels(spokes, hubs):
    i = np.arange(spokes)
    u = np.concatenate([hubs + i] + [np.full(spokes, h) for h in range(hubs)])
    v = np.concatenate([hubs + (i + 1) % spokes] + [hubs + i] * hubs)
    _check(*_copies(u, v, 140000 // (2 * len(u)) + 1, hubs + spokes, spokes))


@pytest.mark.parametrize("rows,cols", [(300, 400), (2, 60000)])
@pytest.mark.parametrize("diagonals", [0, 1, 2])
def test_lattices(rows, cols, diagonals):
    i = np.arange(rows * cols).reshape(rows, cols)
    e = [(i[:, :-1], i[:, 1:]), (i[:-1], i[1:]), (i[:-1, :-1], i[1:, 1:]), (i[:-1, 1:], i[1:, :-1])][:2 + diagonals]
    u, v = (np.concatenate([x[k].ravel() for x in e]) for k in (0, 1))
    _check(rows * cols, u, v)
    p = np.random.default_rng(rows).permutation(rows * cols)
    _check(rows * cols, p[u], p[v])


@pytest.mark.parametrize("mean", [2, 3, 5, 8, 12])
def test_random_with_triangles(mean):
    n = 70000
    rng = np.random.default_rng(mean)
    u = rng.integers(0, n, n * mean // 2)
    _check(n, np.concatenate([u, rng.integers(0, n, n)]), np.concatenate([(u + rng.integers(1, 6, len(u))) % n, rng.integers(0, n, n)]))
