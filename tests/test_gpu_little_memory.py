"""Little device memory: where there is none left for the one-launch form of a
search or a batch, the level graph, which needs less, gives the same parents."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")


def fill_device():
    """Allocates what the device has left, in ever smaller pieces (untouched)."""
    held, size = [], 1 << 36
    while size >= 1 << 20:
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size >>= 1
    return held


def test_first_run_without_memory():
    graphs = [g5.Graph.kronecker(s) for s in (18, 20)]
    roots = [g5.select_roots(g, 5) for g in graphs]
    flat, counts = np.concatenate(roots), [len(r) for r in roots]
    total = sum(g.n * c for g, c in zip(graphs, counts))
    want, out = (torch.zeros(total, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    first = g5.Batch(graphs)
    first.run(flat, counts, want)
    b = g5.Batch(graphs)
    b.launch(flat, counts, out)  # (what a first launch of the level graph loads)
    b.poll(wait=True)
    assert torch.equal(out, want)
    expect = want.cpu().numpy()
    held = fill_device()
    try:
        for _ in range(2):
            out.zero_()
            torch.cuda.synchronize()
            assert b.run(flat, counts, out) > 0
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), expect)
    finally:
        del held
        torch.cuda.empty_cache()
    out.zero_()
    torch.cuda.synchronize()
    b.run(flat, counts, out)  # with memory again
    assert torch.equal(out, want)
    b.close()
    first.close()
    for g in graphs:
        g.close()


def test_search_workspace_in_little_memory():
    g = g5.Graph.kronecker(18, 256)  # (dense: many work items)
    roots = g5.select_roots(g, 3)
    outs = [torch.zeros(g.n, dtype=torch.int64, device="cuda") for _ in roots]
    first, loop = g5.CudaBFS(g), g5.CudaBFS(g, parent_mode=1)  # (the kernels of both are loaded)
    want = []
    for r, o in zip(roots, outs):
        assert loop.run(int(r), o) == 0 and first.run(int(r), o) == 0
        want.append(o.cpu().numpy())
    first.close()
    loop.close()
    room = g5.CudaBFS(g, parent_mode=1)  # what the level loop's workspace takes
    held = fill_device()
    room.close()
    try:
        b = g5.CudaBFS(g)
        for r, o, w in zip(roots, outs, want):
            assert b.run(int(r), o) == 0
            assert np.array_equal(o.cpu().numpy(), w)
        b.close()
    finally:
        del held
        torch.cuda.empty_cache()
    g.close()
