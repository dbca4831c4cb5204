"""Calls that clear memory of their own on their first use, while the legacy default
stream is busy: their kernels run on other streams, which wait for nothing that
is queued there."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")

CYCLES = 400_000_000  # about a fifth of a second


@pytest.mark.parametrize("n,m", [(2000, 8000), (20_000, 90_000), (140_000, 500_000)])
def test_first_call_of_many_roots(n, m):
    """Every lane of g5_bfs_run_many clears its level sums before its first search."""
    rng = np.random.default_rng(n)
    ro, col = orc.build_csr(n, rng.integers(0, n, size=(m, 2)))
    roots = rng.integers(0, n, 9)
    want = [orc.bfs(ro, col, int(r))[0] for r in roots]
    g = g5.Graph.from_csr(ro, col)
    for _ in range(3):
        b = g5.CudaBFS(g)
        outs = [torch.empty(n, dtype=torch.int64, pin_memory=True) for _ in roots]
        torch.cuda.synchronize()
        torch.cuda._sleep(CYCLES)
        b.run_many(roots, outs)
        for w, o in zip(want, outs):
            assert np.array_equal(o.numpy(), w)
        torch.cuda.synchronize()
        b.run_many(roots, outs)  # what was queued there has run by now
        for w, o in zip(want, outs):
            assert np.array_equal(o.numpy(), w)
        b.close()
    g.close()
