"""SCAN queries with many cores, against the oracle: rings and lattices whose ids follow their
layout and permuted ones, similar entries a core around the hooking kernels' limit, more short
core rows than warps, few cores and none."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle


def _csr(n, u, v):
    u, v = u.astype(np.int64), v.astype(np.int64)
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    return np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)


def _ring(n, half, permute, leaves=0):
    """Every vertex joined to the `half` next ones; `leaves` further vertices hang on two random ones each."""
    rng = np.random.default_rng(n + half)
    i = np.arange(n)
    u, v = np.tile(i, half), np.concatenate([(i + d) % n for d in range(1, half + 1)])
    if leaves:
        w = np.repeat(np.arange(n, n + leaves), 2)
        u, v = np.concatenate([u, w]), np.concatenate([v, rng.integers(0, n, 2 * leaves)])
    n += leaves
    if permute:
        p = rng.permutation(n)
        u, v = p[u], p[v]
    return _csr(n, u, v)


def _check(off, dst, queries):
    G = accx.Graph.from_csr(off, dst)
    G.count(bias=2)
    for eps, mu in queries:
        ref = oracle.scan(off, dst, eps, mu, nthreads=16)
        r = G.scan(eps, mu)
        for k in ("sim", "label", "cluster"):
            assert np.array_equal(r[k], ref[k]), (k, eps, mu)


# 2 half similar entries a core, on both sides of the limit of 32
@pytest.mark.parametrize("half", [2, 8, 15, 16, 17, 40])
@pytest.mark.parametrize("permute", [False, True])
def test_rings(half, permute):
    _check(*_ring(20000, half, permute, leaves=3000), [(0.2, 2), (0.3, 2 * half), (0.5, 1), (0.7, 3)])


# short core rows: a few a warp, and more than a warp takes one by one
@pytest.mark.parametrize("n", [5000, 150000, 400000])
def test_many_short_rows(n):
    _check(*_ring(n, 3, False, leaves=n // 4), [(0.2, 2), (0.5, 2)])


@pytest.mark.parametrize("rows,cols", [(1000, 1000), (2, 70000), (70000, 2)])
def test_lattices(rows, cols):
    i = np.arange(rows * cols).reshape(rows, cols)
    u = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    v = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    _check(*_csr(rows * cols, u, v), [(0.2, 2), (0.4, 3), (0.5, 4), (0.9, 2)])


def test_few_cores_and_none():
    rng = np.random.default_rng(9)
    a, b = np.triu_indices(12, 1)
    k = 40000
    off, dst = _csr(20000, np.concatenate([a, rng.integers(0, 20000, k)]), np.concatenate([b, rng.integers(0, 20000, k) // 2]))
    keep = np.repeat(np.arange(20000), np.diff(off)) != dst
    src = np.repeat(np.arange(20000), np.diff(off))[keep]
    off, dst = _csr(20000, src, dst[keep])
    _check(off, dst, [(0.5, mu) for mu in (3, 5, 8, 9, 10, 11, 12, 50)] + [(0.99, 2), (0.05, 0)])
