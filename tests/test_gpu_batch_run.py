"""The one-launch batched search where its paths change: graphs of one unit and
many, claimed and built item lists, hubs of many items, graphs that change
direction at different levels, many graphs, long chains, few and 64 roots; each
root's parents equal the oracle's, also through the level graph (launch/poll)
on the same workspace."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")


def oracle_u32(ro, col, r):
    return orc.bfs(ro, col, int(r))[0].astype(np.uint64).astype(np.uint32)


def check(csrs, roots, directions=((14.0, 24.0),), offset=0):
    graphs = [g5.Graph.from_csr(ro, col) for ro, col in csrs]
    bt = g5.Batch(graphs)
    counts = [len(r) for r in roots]
    total = sum(c * g.n for c, g in zip(counts, graphs))
    buf = torch.empty(total + 8, dtype=torch.int32, device="cuda")
    flat = np.concatenate([np.asarray(r, np.int64) for r in roots])
    want = [[oracle_u32(ro, col, r) for r in rs] for (ro, col), rs in zip(csrs, roots)]
    for alpha, beta in directions:
        bt.set_direction(alpha, beta)
        for graph_loop in (False, True, False):
            buf.fill_(7)
            torch.cuda.synchronize()
            out = buf[offset:offset + total]
            if graph_loop:
                bt.launch(flat, counts, out)
                assert bt.poll(wait=True)[0]
            else:
                assert bt.run(flat, counts, out) > 0
            got = buf.cpu().numpy().view(np.uint32)
            assert (got[:offset] == 7).all() and (got[offset + total:] == 7).all()
            at = offset
            for (ro, col), rs, w in zip(csrs, roots, want):
                n = len(ro) - 1
                block = got[at:at + n * len(rs)].reshape(n, len(rs))
                for j in range(len(rs)):
                    assert np.array_equal(block[:, j], w[j]), (alpha, graph_loop, n, rs[j])
                at += n * len(rs)
    bt.close()
    for g in graphs:
        g.close()


def random_csr(n, m, seed):
    return orc.build_csr(n, np.random.default_rng(seed).integers(0, n, size=(m, 2)))


@pytest.mark.parametrize("n,m", [(1, 0), (33, 50), (2048, 6000), (2049, 9000), (70_000, 400_000)])
@pytest.mark.parametrize("nroots", [1, 33, 64])
def test_sizes(n, m, nroots):
    rng = np.random.default_rng(n)
    check([random_csr(n, m, n)], [rng.integers(0, n, nroots)], offset=n % 4)


def test_directions():
    """Bottom-up from the start, top-down only, and back and forth."""
    csr = orc.build_csr(1 << 12, orc.kronecker(12))
    check([csr], [orc.select_roots(csr[0], 20)], directions=((1e12, 1e12), (1e-6, 1e-6), (1.0, 2.0), (14.0, 24.0)))


def test_hubs_past_the_claim_limit():
    """Two hubs of 400,000 entries: rows of many items, and a top-down level past
    the claim limit whose next level is built from the words."""
    n = 500_001
    leaves = np.arange(2, 400_002)
    edges = np.concatenate([np.stack([np.zeros_like(leaves), leaves], 1), np.stack([np.ones_like(leaves), leaves], 1),
                            np.stack([leaves[::5], 400_002 + leaves[::5] % 90_000], 1)])
    csr = orc.build_csr(n, edges)
    check([csr], [[0, 1, 17, 450_000]], directions=((1e-6, 1e-6), (14.0, 24.0)))


@pytest.mark.parametrize("d", [1023, 1024, 1025, 1032, 1033, 1536, 1545, 5000])
def test_long_rows_bottom_up(d):
    """A hub of d entries reached through one entry of its row only (roots at its
    start, at its end and at the pieces' edges), and a second hub which many
    entries of several pieces reach at once."""
    leaves = np.arange(2, 2 + d)
    own = 2 + d + np.arange(700)
    edges = np.concatenate([np.stack([np.zeros_like(leaves), leaves], 1),
                            np.stack([np.ones_like(own), own], 1),
                            np.stack([np.ones_like(leaves), leaves + 700 + d], 1),
                            np.stack([np.zeros_like(leaves), leaves + 700 + d], 1)])
    csr = orc.build_csr(2 + 2 * d + 700, edges)
    at = [x for x in (0, 7, 8, 511, 512, 513, 519, 520, 521, 1023, 1031, 1032, 1033, 1535, 1536, 2047) if x < d]
    roots = [0, 1, int(own[0]), int(own[-1])] + [2 + x for x in at] + [1 + d, 1 + 2 * d + 700]
    check([csr], [roots], directions=((1e12, 1e12), (14.0, 24.0)))


@pytest.mark.parametrize("scale,chains", [(12, 3), (13, 40), (14, 62)])
def test_roots_that_lag(scale, chains):
    """Roots at the ends of chains hung on a Kronecker graph are levels behind the
    others when it turns bottom-up, so that they expand top-down in that level;
    beside it a graph below the least size for that, and one of only such roots."""
    rng = np.random.default_rng(scale)
    n, edges, ends = 1 << scale, [orc.kronecker(scale)], []
    for c in range(chains):
        length = 1 + c % 5
        ids = np.concatenate([[rng.integers(0, 1 << scale)], n + np.arange(length)])
        edges.append(np.stack([ids[:-1], ids[1:]], 1))
        n += length
        ends.append(n - 1)
    csr = orc.build_csr(n, np.concatenate(edges))
    heads = orc.select_roots(csr[0], 64 - chains)
    roots = rng.permutation(np.concatenate([heads, ends]))
    small = random_csr(3000, 20_000, 5)
    check([csr, small, csr], [roots, rng.integers(0, 3000, 9), ends[:9]],
          directions=((14.0, 24.0), (200.0, 24.0), (1.0, 1e6)))


def test_many_uneven_graphs():
    """64 graphs, some without edges, whose directions change at different levels."""
    rng = np.random.default_rng(4)
    csrs, roots = [], []
    for i in range(64):
        n = int(rng.integers(1, 3000))
        csrs.append(random_csr(n, 0 if i % 9 == 0 else n * int(rng.integers(1, 12)), i))
        roots.append(rng.integers(0, n, int(rng.integers(0, 9))))
    k = 1 << 11
    csrs[5] = orc.build_csr(k, orc.kronecker(11))
    roots[5] = orc.select_roots(csrs[5][0], 64)
    check(csrs, roots)


def test_long_chain():
    n = 600
    csr = orc.build_csr(n, np.array([(i, i + 1) for i in range(n - 1)], np.int64))
    check([csr, random_csr(500, 900, 1)], [[0, 300, n - 1], [3, 4]])


def test_level_cap():
    n = 1200
    csr = orc.build_csr(n, np.array([(i, i + 1) for i in range(n - 1)], np.int64))
    g = g5.Graph.from_csr(*csr)
    bt = g5.Batch([g])
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    with pytest.raises(g5.G5Error) as e:
        bt.run(np.array([0], np.int64), [1], out)
    assert e.value.code == g5.G5_ERR_TIMEOUT
    assert bt.run(np.array([600], np.int64), [1], out) > 0
    assert np.array_equal(out.cpu().numpy().view(np.uint32), oracle_u32(*csr, 600))
    bt.close()
    g.close()


def test_degree_past_24_bits():
    """A star of 2^24 + 2 leaves: the hub's record holds no degree."""
    leaves = (1 << 24) + 2
    n = leaves + 1
    ro = np.concatenate([[0], leaves + np.arange(n)]).astype(np.int64)
    col = np.concatenate([np.arange(1, n), np.zeros(leaves)]).astype(np.uint32)
    g = g5.Graph.from_csr(ro, col)
    bt = g5.Batch([g])
    roots = np.array([0, 1, leaves], np.int64)
    out = torch.empty(3 * n, dtype=torch.int32, device="cuda")
    for alpha in (1e12, 14.0):
        bt.set_direction(alpha, 1e12 if alpha > 100 else 24.0)
        for graph_loop in (False, True):
            out.fill_(7)
            torch.cuda.synchronize()
            if graph_loop:
                bt.launch(roots, [3], out)
                assert bt.poll(wait=True)[0]
            else:
                assert bt.run(roots, [3], out) > 0
            got = out.view(n, 3)
            for j, r in enumerate(roots):
                want = torch.zeros(n, dtype=torch.int32, device="cuda")
                want[int(r)] = int(r)
                want[0] = int(r)
                assert torch.equal(got[:, j], want), (alpha, graph_loop, j)
    bt.close()
    g.close()
