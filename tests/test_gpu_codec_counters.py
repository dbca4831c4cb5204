"""The asynchronous codec calls with one device counter for both lengths: the
values' count goes in and the words come back in its place, and the other way
round, while other work keeps some blocks of the calls from starting."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [0, 1, 100, 128, 3000, 4095, 4223, 6000, 100_000])
@pytest.mark.parametrize("kind", ["ids", "random"])
def test_one_counter_in_and_out(n, kind):
    rng = np.random.default_rng(n)
    x = (np.cumsum(rng.integers(1, 9, n), dtype=np.uint64).astype(np.uint32) if kind == "ids"
         else rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32))
    c = g5.Codec(max(n, 1) * 2 + 4096)
    values = torch.zeros(2 * n + 8192, dtype=torch.int32, device="cuda")
    values[:n] = torch.from_numpy(x.view(np.int32)).cuda()
    stream = torch.zeros(g5.Codec.bound(2 * n + 8192), dtype=torch.int32, device="cuda")
    back = torch.full((2 * n + 8192,), -1, dtype=torch.int32, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    busy = torch.ones(1 << 26, device="cuda")
    torch.cuda.synchronize()
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    for mode, omode in ((g5.CODEC_D4, orc.D4), (g5.CODEC_DM, orc.DM)):
        want = orc.encode(x, omode)
        for _ in range(10):
            with torch.cuda.stream(other):
                for _ in range(4):
                    busy.mul_(1.0)
            with torch.cuda.stream(s):
                count.fill_(n)
                c.encode_async(values, count, stream, count, mode, s.cuda_stream)
                words = count.clone()
                c.decode_async(stream, count, back, n + 128, count, mode, s.cuda_stream)
            torch.cuda.synchronize()
            assert c.status() == 0 and int(words) == len(want) and int(count) == n
            assert np.array_equal(stream.cpu().numpy().view(np.uint32)[:len(want)], want)
            got = back.cpu().numpy().view(np.uint32)
            assert np.array_equal(got[:n], x) and (got[n:] == 0xFFFFFFFF).all()
    c.close()
