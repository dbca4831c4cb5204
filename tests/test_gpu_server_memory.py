"""What a server takes of the device stays within its budget: the smallest
budget that admits a number of slots holds the workspaces it pays for, on graphs
of mean size and on dense ones, where work items outgrow the other arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")

SLACK = 4 << 20  # pages that small allocations share


def used():
    free, total = torch.cuda.mem_get_info()
    return total - free


def smallest_budget(g, mode, slots):
    """Least budget (to 64 KB) that gives at least `slots` slots."""
    def given(budget):
        try:
            sv = g5.Server([g], mem_budget=budget, modes=[mode])
        except g5.G5Error as e:
            assert e.code == g5.G5_ERR_OOM
            return 0
        k = sv.slots()[0]
        sv.close()
        return k
    lo, hi = 0, 1 << 24
    while given(hi) < slots:
        hi *= 2
    while hi - lo > 1 << 16:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if given(mid) < slots else (lo, mid)
    return hi


@pytest.mark.parametrize("scale,edgefactor", [(12, 16), (16, 16), (17, 16), (18, 16), (19, 16), (14, 256), (16, 256)])
@pytest.mark.parametrize("mode", [g5.Server.STREAMS, g5.Server.COHORTS])
def test_budget_holds(scale, edgefactor, mode):
    g = g5.Graph.kronecker(scale, edgefactor)
    roots = g5.select_roots(g, 4)
    with_queue = g5.Server([g], mem_budget=1 << 30, modes=[mode])  # (kernels loaded)
    assert with_queue.wait(with_queue.submit(0, int(roots[0])))
    with_queue.close()
    budget = smallest_budget(g, mode, 6)
    torch.cuda.synchronize()
    before = used()
    sv = g5.Server([g], mem_budget=budget, modes=[mode])
    taken = used() - before - 4 * g.n  # (a result's gathering buffer is the server's own)
    assert sv.slots()[0] >= 6
    assert taken <= budget + SLACK, (taken / budget, taken, budget)
    for r in roots:
        t = sv.submit(0, int(r))
        assert sv.wait(t)
        sv.result(t)  # (frees its slot)
    sv.close()
    g.close()
