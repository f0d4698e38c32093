"""Relabeled rows above 4096 entries, which share 4096-entry chunks with the next row, against
numpy: one row, many of like lengths, rows that end on a chunk."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx


@pytest.mark.parametrize("lens", [[4097], [8192], [100000], [4097] * 3, [8192, 4097, 4097], [12288, 8192, 8192, 4100],
                                  [60000, 20480, 12289, 12288, 12287, 4098, 4097, 4096, 30],
                                  list(range(4090, 4130)) * 3, [4096 + 64 * i for i in range(70)]])
def test_rows(lens):
    rng = np.random.default_rng(len(lens) + lens[0])
    pool = max(lens) + 500
    n = len(lens) + pool
    p = rng.permutation(n)  # centres anywhere among the ids
    u = p[np.repeat(np.arange(len(lens)), lens)]
    v = p[np.concatenate([len(lens) + rng.permutation(pool)[:d] for d in lens])]
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
