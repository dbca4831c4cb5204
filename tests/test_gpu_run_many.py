"""g5_bfs_run_many with several searches at a time: every form of the search,
fewer roots than lanes, as many, and more; parents to device, pinned and
pageable memory and nowhere; the workspace refers to the last root afterwards."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")


def outputs(n, k):
    makers = [lambda: torch.empty(n, dtype=torch.int64, device="cuda"), lambda: np.full(n, 7, np.int64),
              lambda: torch.empty(n, dtype=torch.int64, pin_memory=True), lambda: None]
    return [makers[i % 4]() for i in range(k)]


def host(o):
    return o.cpu().numpy() if hasattr(o, "cpu") else o


def check(g, n, want, roots, **kw):
    b, one = g5.CudaBFS(g, **kw), g5.CudaBFS(g, **kw)
    for k in (2, 1, 3, 5, 9, 16):
        rs = np.array([roots[i % len(roots)] for i in range(k)], np.int64)
        outs = outputs(n, k)
        torch.cuda.synchronize()
        ms = b.run_many(rs, outs, device_ms=True)
        assert (ms > 0).all()
        for r, o in zip(rs, outs):
            if o is not None:
                assert np.array_equal(host(o), want(int(r))), (k, int(r))
        assert one.run(int(rs[-1]), None) == 0
        assert np.array_equal(b.level_log(), one.level_log())
        if kw.get("want_levels"):
            lev, lev1 = np.empty(n, np.int32), np.empty(n, np.int32)
            assert b.run(int(rs[0]), None, lev) == 0 and one.run(int(rs[0]), None, lev1) == 0
            assert np.array_equal(lev, lev1)
    assert b.validate() == (True, True)
    b.close()
    one.close()


@pytest.mark.parametrize("n,m", [(1, 0), (700, 2000), (20_000, 90_000), (140_000, 500_000)])
@pytest.mark.parametrize("kw", [{}, {"want_levels": True}, {"codec": 1}])
def test_forms(n, m, kw):
    rng = np.random.default_rng(n)
    ro, col = orc.build_csr(n, rng.integers(0, n, size=(m, 2)))
    roots = rng.integers(0, n, 7)
    parents = {int(r): orc.bfs(ro, col, int(r))[0] for r in roots}
    g = g5.Graph.from_csr(ro, col)
    check(g, n, parents.__getitem__, roots, **kw)
    g.close()


@pytest.mark.parametrize("scale", [18, 21, 22])
def test_large(scale):
    """Against single runs (which equal the oracle's in their own tests)."""
    g = g5.Graph.kronecker(scale)
    roots = g5.select_roots(g, 5)
    s = g5.CudaBFS(g)
    parents = {}
    for r in roots:
        p = torch.empty(g.n, dtype=torch.int64, device="cuda")
        assert s.run(int(r), p) == 0
        parents[int(r)] = p.cpu().numpy()
    check(g, g.n, parents.__getitem__, roots)
    s.close()
    g.close()


def test_level_cap():
    """A search past the level cap fails the call; the others' parents arrive and
    the workspace goes on."""
    n = 300
    ro, col = orc.build_csr(n, np.array([(i, i + 1) for i in range(n - 1)], np.int64))
    g = g5.Graph.from_csr(ro, col)
    b = g5.CudaBFS(g, max_levels=200)
    roots = [150, 0, 140, 160, 299, 150]
    outs = [np.empty(n, np.int64) for _ in roots]
    for _ in range(2):
        with pytest.raises(g5.G5Error) as e:
            b.run_many(np.array(roots, np.int64), outs)
        assert e.value.code == g5.G5_ERR_TIMEOUT
        for r, o in zip(roots, outs):
            if r not in (0, 299):
                assert np.array_equal(o, orc.bfs(ro, col, r)[0])
    with pytest.raises(g5.G5Error):  # (vertex 299 is 199 levels from 100: one too many)
        b.run_many(np.array([100, 120, 130], np.int64), outs[:3])
    assert np.array_equal(outs[1], orc.bfs(ro, col, 120)[0])
    b.run_many(np.array([101, 120, 130], np.int64), outs[:3])
    assert np.array_equal(outs[0], orc.bfs(ro, col, 101)[0])
    b.close()
    g.close()
