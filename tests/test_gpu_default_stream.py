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


def test_first_batch_of_queues():
    """g5_codec_encode_batch and g5_codec_decode_batch clear the chunks' records
    where these are new or have grown."""
    rng = np.random.default_rng(7)
    stream = torch.cuda.Stream()  # (non-blocking)
    c = g5.Codec(1 << 20)
    for sizes in ([3000, 40_000], [200_000, 1, 300_001, 70_000], [900_001] * 4):
        queues = [np.cumsum(rng.integers(1, 9, n), dtype=np.uint64).astype(np.uint32) for n in sizes]
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
        values = torch.from_numpy(np.concatenate(queues).view(np.int32)).cuda()
        out = torch.zeros(g5.Codec.batch_bound(off), dtype=torch.int32, device="cuda")
        back = torch.zeros_like(values)
        torch.cuda.synchronize()
        torch.cuda._sleep(CYCLES)
        at, words = c.encode_batch(values, off, out, stream=stream.cuda_stream)
        _, ok = c.decode_batch(out, at[:-1], words, np.diff(off), back, stream=stream.cuda_stream)
        assert ok.all()
        torch.cuda.synchronize()
        got = out.cpu().numpy().view(np.uint32)
        for q, o, w in zip(queues, at[:-1], words):
            assert np.array_equal(got[int(o):int(o) + int(w)], orc.encode(q, orc.D4))
        assert torch.equal(back, values)
    c.close()
