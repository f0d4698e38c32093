"""GPU parity of oriented counts on CSRs that were not relabeled, at entry counts where the
count array ends on an allocation boundary, against the oracle's counts.  Counts are whole
numbers: equal or wrong."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle


def _with_entries(n, m, seed):
    """A random symmetric CSR of exactly m entries (m / 2 edges)."""
    rng = np.random.default_rng(seed)
    a, b = np.triu_indices(n, 1)
    e = rng.permutation(len(a))[:m // 2]
    u, v = a[e].astype(np.int64), b[e].astype(np.int64)
    k = np.sort(np.concatenate([u * n + v, v * n + u]))
    return np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)


@pytest.mark.parametrize("m", [2, 4, 6, 62, 64, 66, 126, 128, 130, 254, 256, 258, 382, 384, 386, 510, 512, 514, 1022,
                               1024, 1026, 2048, 65536, 131072])
@pytest.mark.parametrize("validate", [True, "exact", False])
def test_entry_counts(m, validate):
    rng = np.random.default_rng(m)
    n = max(4, int(2.2 * m ** 0.5))
    off, dst = _with_entries(n, m, m)
    assert len(dst) == m
    ref = oracle.cn_count(off, dst, nthreads=8)
    table = rng.integers(0, 3, size=(24, 24)).astype(np.uint8)
    for kw in ({"policy": "merge"}, {"policy": "table", "table": table}, {"policy": "gallop"}, {"policy": "bitmap"},
               {"policy": "heuristic"}):
        G = accx.Graph.from_csr(off, dst, validate=validate)
        # graphs before and after the count's arrays: nothing of theirs changes
        other = [accx.Graph.from_csr(off, dst) for _ in range(2)]
        kept = [H.count(policy="merge", bias=0) for H in other]
        assert np.array_equal(G.count(bias=2, orient=True, **kw), ref), kw
        for H, c in zip(other, kept):
            o, d = H.download()
            assert np.array_equal(o, off) and np.array_equal(d, dst) and np.array_equal(H.read_counts(), c), kw
        assert np.array_equal(G.count(bias=7, orient=True, **kw), ref + 5), kw
