"""Searches and batches beside another stream's long kernel of a block: they begin
and end while it runs."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")

CYCLES = 1_000_000_000  # about half a second
SIZES = [2000, 20_000, 200_000, (1 << 22) + 5]  # each form of the search


@pytest.fixture(scope="module", params=SIZES)
def case(request):
    n = request.param
    ro, col = orc.build_csr(n, np.random.default_rng(n).integers(0, n, (2 * n, 2)))
    roots = [1, n // 3, n - 1]
    g = g5.Graph.from_csr(ro, col)
    yield g, roots, [orc.bfs(ro, col, r)[0] for r in roots]
    g.close()


def held(stream):
    with torch.cuda.stream(stream):
        torch.cuda._sleep(CYCLES)
    return stream


def test_search(case):
    g, roots, want = case
    b = g5.CudaBFS(g)
    out = torch.zeros(g.n, dtype=torch.int64, pin_memory=True)
    assert b.run(roots[0], out, stats=False) == 0
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    held(stream)
    for r, w in zip(roots, want):
        assert b.run(r, out, stats=False) == 0
        assert not stream.query(), "the search waited for the other stream's kernel"
        assert np.array_equal(out.numpy(), w)
        out.zero_()
    b.close()


def test_many_roots(case):
    g, roots, want = case
    b = g5.CudaBFS(g)
    outs = [torch.zeros(g.n, dtype=torch.int64, pin_memory=True) for _ in roots]
    b.run_many(roots, outs)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    held(stream)
    b.run_many(roots, outs)
    assert not stream.query()
    for o, w in zip(outs, want):
        assert np.array_equal(o.numpy(), w)
    b.close()


def test_batch(case):
    g, roots, want = case
    bt = g5.Batch([g])
    out = torch.zeros(len(roots) * g.n, dtype=torch.int32, device="cuda")
    bt.run(np.array(roots), [len(roots)], out)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    held(stream)
    bt.run(np.array(roots), [len(roots)], out)
    assert not stream.query()
    torch.cuda.synchronize()
    p = out.cpu().numpy().reshape(g.n, len(roots))
    for i, w in enumerate(want):
        assert np.array_equal(p[:, i].astype(np.int64), w)  # (-1: all ones)
    bt.close()
