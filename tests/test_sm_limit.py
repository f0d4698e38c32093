"""accx_count_opts.sm_limit with the default policy's one-kernel count of small graphs: same
counts, and the kernel stays within its SMs."""
import ctypes as C

import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if has_gpu():
    from acctricnt_gb300 import accx
    from oracle import oracle


@pytest.mark.parametrize("scale,ef", [(6, 4), (10, 16), (12, 16)])
def test_small_default_count(scale, ef):
    import torch
    G = accx.Graph.generate(accx.rmat_params(scale, ef, seed=scale))
    off, dst = G.download()
    assert len(dst) <= 1 << 17
    ref = oracle.cn_count(off, dst, nthreads=8)

    def run(limit):
        opts, _ = G._opts("heuristic", None, 2, 0, 0)
        opts.sm_limit = limit
        best = float("inf")
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            assert accx.lib.accx_cn_count(G._h, C.byref(opts), None, None) == accx.OK
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        assert np.array_equal(G.read_counts(), ref), limit
        return best

    free = run(0)
    ms = {limit: run(limit) for limit in (1, 2, 7, 100, 10000)}
    if scale == 12:  # 6000 tiles: on one SM they take many times as long
        assert ms[1] > 4 * free, (free, ms)
