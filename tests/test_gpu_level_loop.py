"""The level loop (searches with the codec, with fix-up parents, without the
graph) where its passes change: tiles split over warps, queues with and without
edge offsets, raw copies by one block and by all, levels and no levels; parents and levels equal the oracle's."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")


def hubs_and_paths():
    """Hubs whose rows span many tiles, between chains of vertices of one or two
    entries, so that the vertex of a split tile's first entry is anywhere in it."""
    rng = np.random.default_rng(3)
    parts, at = [], 0
    for d in (1, 31, 33, 255, 257, 5000, 40_000):
        hub = at
        leaves = at + 1 + np.arange(d)
        parts.append(np.stack([np.full(d, hub), leaves], 1))
        parts.append(np.stack([leaves, at + 1 + d + rng.integers(0, 1 + d // 3, d)], 1))
        at += 2 + d + d // 3
        parts.append(np.array([[hub + d, at]]))
    return orc.build_csr(at + 37, np.concatenate(parts))


CSRS = {"hubs": hubs_and_paths(), "kron13": orc.build_csr(1 << 13, orc.kronecker(13)),
        "ragged": orc.build_csr(2049, np.random.default_rng(5).integers(0, 2049, size=(7000, 2)))}


@pytest.mark.parametrize("tile", [32, 64, 256, 4096])
@pytest.mark.parametrize("name", sorted(CSRS))
def test_level_loop(name, tile):
    ro, col = CSRS[name]
    deg = np.diff(ro)
    roots = [int(np.argmax(deg)), int(np.flatnonzero(deg > 0)[-1]), int(np.flatnonzero(deg == 1)[0])]
    want = {r: orc.bfs(ro, col, r) for r in roots}
    g = g5.Graph.from_csr(ro, col)
    # (mostly bottom-up, top-down only, the default switch)
    for alpha, beta in ((1e9, 1e9), (1e-9, 1e-9), (14.0, 24.0)):
        for kw in (dict(codec=g5.CODEC_D4), dict(codec=g5.CODEC_DM, want_levels=True),
                   dict(codec=g5.CODEC_D4, codec_threshold=20_000), dict(parent_mode=1),
                   dict(parent_mode=2, want_levels=True), dict(use_graph=False, want_levels=True)):
            s = g5.CudaBFS(g, alpha=alpha, beta=beta, tile_edges=tile, **kw)
            for r in roots + roots[:1]:
                parent, level = want[r][:2]
                pred = torch.empty(len(ro) - 1, dtype=torch.int64, device="cuda")
                lev = torch.empty(len(ro) - 1, dtype=torch.int32, device="cuda") if kw.get("want_levels") else None
                assert s.run(r, pred, lev) == 0
                assert np.array_equal(pred.cpu().numpy(), parent), (kw, alpha, r)
                if lev is not None:
                    assert np.array_equal(lev.cpu().numpy(), level), (kw, alpha, r)
            s.close()
    g.close()
