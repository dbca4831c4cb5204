"""The one-launch search at the sizes where its forms and paths change: one
block, one cluster, the grid with one and two blocks per SM; claimed and
counted top-down levels; narrow and wide bottom-up steps; rows of many work
items.  Parents and levels equal the oracle's."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")


def check(n, edges, roots, **kw):
    ro, col = orc.build_csr(n, np.asarray(edges, np.int64).reshape(-1, 2))
    g = g5.Graph.from_csr(ro, col)
    b = g5.CudaBFS(g, want_levels=True, **kw)
    for r in roots:
        want_pred, want_level = orc.bfs(ro, col, int(r))
        for _ in range(2):  # the ring of level sums goes on from search to search
            b.runBFS(int(r))
            assert np.array_equal(b.getPredecessor(), want_pred), (n, r)
            assert np.array_equal(b.getLevels(), want_level), (n, r)
        log = b.level_log()
        deg = np.diff(ro)
        for L in range(int(want_level.max()) + 1):
            m = want_level == L
            assert (int(log[L, 1]), int(log[L, 2])) == (int(m.sum()), int(deg[m].sum())), (n, r, L)
    b.close()
    g.close()


@pytest.mark.parametrize("n", [31, 32, 129, 4096, 4097, 32768, 32769, 100003, (1 << 22) - 1, (1 << 22) + 5])
def test_forms(n):
    rng = np.random.default_rng(n)
    check(n, rng.integers(0, n, size=(3 * min(n, 400_000), 2)), [0, n - 1, n // 2])


@pytest.mark.parametrize("n", [3000, 20000, 70000])
@pytest.mark.parametrize("alpha,beta", [(1e12, 1e12), (1e-6, 1e-6), (1.0, 2.0)])
def test_directions(n, alpha, beta):
    rng = np.random.default_rng(n)
    check(n, rng.integers(0, n, size=(5 * n, 2)), [1, n - 2], alpha=alpha, beta=beta)


@pytest.mark.parametrize("tile", [32, 4096])
def test_hub_rows(tile):
    """A hub of 600,000 entries: many items from one row, and a top-down level
    past the claim limit whose next level is built from the bitmap."""
    n = 700_001
    leaves = np.arange(1, 600_001)
    edges = np.concatenate([np.stack([np.zeros_like(leaves), leaves], 1),
                            np.stack([leaves[::3], 600_001 + leaves[::3] % 90_000], 1)])
    check(n, edges, [0, 17, 650_000], tile_edges=tile, alpha=1e-6)
    check(n, edges, [0, 17], tile_edges=tile)


def test_thin_wide_levels():
    """Bottom-up levels with few candidates per word on a graph of over 10 M
    vertices: 128 words per warp step, and steps with more candidates than the
    list holds (a dense range of vertices in a path)."""
    n = 11_000_003
    hub = np.arange(1, n, 64)
    path = 5_000_000 + np.arange(900)
    edges = np.concatenate([np.stack([np.zeros_like(hub), hub], 1), np.stack([path[:-1], path[1:]], 1),
                            np.stack([hub[:-1], hub[1:]], 1)])
    check(n, edges, [0], alpha=1e12, beta=1e12, max_levels=2000)
