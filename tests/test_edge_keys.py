"""CSRs built from edge lists at the sizes where the sort keys change width, against
numpy: self loops and repeats dropped, both directions kept."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx


def _ref(u, v, n):
    u, v = u.astype(np.int64), v.astype(np.int64)
    keep = u != v
    u, v = u[keep], v[keep]
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    return np.searchsorted(k, np.arange(n + 1) * n).astype(np.uint32), (k % n).astype(np.int32)


# ids of 1 to 17 bits and of 21: 32-bit keys up to 65536 vertices, 64-bit ones above
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 255, 256, 257, 65535, 65536, 65537, 1 << 17, (1 << 20) + 1])
@pytest.mark.parametrize("k", [0, 1, 7, 50000])
def test_csr_from_edges(n, k):
    rng = np.random.default_rng(n * 31 + k)
    u = rng.integers(0, n, k).astype(np.uint32)
    v = np.where(rng.random(k) < 0.1, u, rng.integers(0, n, k)).astype(np.uint32)
    if k > 3:  # the largest ids, as a self loop and as an edge
        u[:2], v[:2] = n - 1, (n - 1, 0)
        u[2], v[2] = 0, n - 1
    G = accx.Graph.from_edges(u, v, n)
    off, dst = G.download()
    roff, rdst = _ref(u, v, n)
    assert np.array_equal(off, roff) and np.array_equal(dst, rdst)
    if k:
        u[-1] = n
        with pytest.raises(accx.AccxError) as e:
            accx.Graph.from_edges(u, v, n)
        assert e.value.status == accx.ERR_RANGE
