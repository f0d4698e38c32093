"""The default policy's count of graphs with rows of many tiles of entries, which several CTAs
filter: row lengths and places around the tiles' ends, in every position, against the
oracle's counts and the statistics of the ratio-50 rule."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle

TILE = 8192


def _csr(n, u, v):
    keep = u != v
    u, v = u[keep].astype(np.int64), v[keep].astype(np.int64)
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    return np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)


def _check(off, dst):
    assert len(dst) > 1 << 17
    ref = oracle.cn_count(off, dst, nthreads=16)
    G = accx.Graph.from_csr(off, dst)
    for _ in range(2):
        assert np.array_equal(G.count(bias=2), ref)
    deg = np.diff(off).astype(np.int64)
    src = np.repeat(np.arange(len(deg)), deg)
    own = (deg[src] > deg[dst]) | ((deg[src] == deg[dst]) & (src < dst))
    du, dv = deg[src][own], deg[dst][own]
    gal = 50 * dv < du
    st, ow = G.last_stats(), G.owner_work()
    for k, m in (("merge", ~gal), ("gallop", gal)):
        assert (st[k]["edges"], st[k]["work"], ow[k]) == (int(m.sum()), int(dv[m].sum()), int(du[m].sum())), k


# one hub's row around two tiles and more, at the front, at the back and between other rows
@pytest.mark.parametrize("row", [2 * TILE - 1, 2 * TILE, 2 * TILE + 1, 2 * TILE + 2, 3 * TILE - 1, 3 * TILE, 3 * TILE + 1, 70000])
@pytest.mark.parametrize("hub", ["first", "middle", "last"])
def test_one_hub(row, hub):
    rng = np.random.default_rng(row)
    leaves = max(row, 66000)
    n = leaves + 1
    h = {"first": 0, "middle": leaves // 3, "last": n - 1}[hub]
    others = np.delete(np.arange(n), h)
    v = rng.permutation(others)[:row]
    extra = others[rng.integers(0, leaves, (2, leaves))]
    _check(*_csr(n, np.concatenate([np.full(row, h), extra[0]]), np.concatenate([v, extra[1]])))


# the hub's row begins `shift` entries into a tile
@pytest.mark.parametrize("shift", [0, 1, 255, 256, 4096, TILE - 1])
def test_row_places(shift):
    n, row = 80000, 40000
    h = n // 4
    rng = np.random.default_rng(shift)
    low = rng.integers(0, h, (2, 20000))
    high = rng.integers(h + 1, n, (2, 60000))
    u, v = np.concatenate([np.full(row, h), low[0], high[0]]), np.concatenate([np.arange(n - row, n), low[1], high[1]])
    off, _ = _csr(n, u, v)
    c = np.arange((shift - int(off[h])) % TILE)  # entries of ids below the hub's, to move it
    off, dst = _csr(n, np.concatenate([u, c]), np.concatenate([v, h + 1 + c]))
    assert int(off[h]) % TILE == shift
    _check(off, dst)


# several long rows, next to each other, with long lists of their own
@pytest.mark.parametrize("hubs,leaves", [(2, 50000), (7, 20000), (40, 17000), (140, 16500)])
def test_many_hubs(hubs, leaves):
    rng = np.random.default_rng(hubs)
    a, b = np.triu_indices(hubs, 1)
    u, v = np.repeat(np.arange(hubs), leaves), hubs + np.tile(np.arange(leaves), hubs)
    keep = rng.random(len(u)) < (1.0 if hubs < 100 else 0.999)
    extra = hubs + rng.integers(0, leaves, (2, leaves))
    n = hubs + leaves
    p = rng.permutation(n)
    u, v = np.concatenate([a, u[keep], extra[0]]), np.concatenate([b, v[keep], extra[1]])
    _check(*_csr(n, u, v))
    if hubs <= 40:
        _check(*_csr(n, p[u], p[v]))
