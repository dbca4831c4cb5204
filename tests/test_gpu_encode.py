"""The one-launch encoder at the sizes where its chunks change: tails alone, a
last group with missing miniblocks, one and several groups per chunk, more
chunks than blocks; every width from 0 to 32.  Streams equal the oracle's."""
import numpy as np
import pytest

import oracle as orc
from test_gpu_decode import MODES, values

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")


def check(codec, x):
    n = len(x)
    din = torch.from_numpy(x.view(np.int32)).cuda() if n else torch.zeros(4, dtype=torch.int32, device="cuda")
    for mode, omode in MODES:
        out = torch.full((g5.Codec.bound(n) + 8,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        for _ in range(2):  # records of the call before are not read
            w = codec.encode(din, n, out, mode)
            assert np.array_equal(out[:w].cpu().numpy().view(np.uint32), orc.encode(x, omode)), (n, mode)


@pytest.mark.parametrize("kind", ["ids", "equal", "random", "jumps"])
@pytest.mark.parametrize("n", [0, 1, 127, 128, 2047, 2048, 2049, 304 * 2048, 304 * 2048 + 129, 1_300_001, 8_000_003])
def test_sizes(kind, n):
    c = g5.Codec(max(n, 1))
    check(c, values(kind, n, np.random.default_rng(n)))
    c.close()


def test_every_width():
    rng = np.random.default_rng(2)
    parts = []
    for b in range(33):  # 17 miniblocks of each width: groups mix two widths
        hi = (1 << b) - 1
        parts.append(rng.integers(0, hi + 1, 128 * 17, dtype=np.uint64))
    d = np.concatenate(parts)
    x = d.copy()
    for j in range(4, len(x)):  # d4: each lane runs on from four values before
        x[j] = (x[j] + x[j - 4]) & 0xFFFFFFFF
    c = g5.Codec(len(x))
    check(c, x.astype(np.uint32))
    c.close()


def test_length_past_the_workspace_is_refused():
    c = g5.Codec(1000)
    din = torch.zeros(4096, dtype=torch.int32, device="cuda")
    out = torch.full((8192,), -1, dtype=torch.int32, device="cuda")
    n = torch.tensor([4096], dtype=torch.int64, device="cuda")
    w = torch.full((1,), -5, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    c.encode_async(din, n, out, w)
    assert c.status() == g5.G5_ERR_CAPACITY
    assert int(w) == -5 and bool((out == -1).all())  # nothing is written
    n.fill_(700)
    torch.cuda.synchronize()
    c.encode_async(din, n, out, w)
    assert c.status() == 0 and int(w) > 0
    c.close()


@pytest.mark.parametrize("n", [10, 5000, 300_000])
def test_plugin_refuses_ids_past_32_bits(n):
    """One id below 0 or above 2^32 - 1 anywhere: refused; the queue without it
    goes through unchanged afterwards."""
    p = g5.GpuSimd()
    x = np.arange(n, dtype=np.int64) * 7
    for bad in (-1, 1 << 32, -(1 << 40)):
        for at in (0, n // 2, n - 1):
            y = x.copy()
            y[at] = bad
            with pytest.raises(g5.G5Error):
                p.compress(y)
    c, size = p.compress(x)
    assert np.array_equal(p.decompress(c, size, n), x)


@pytest.mark.parametrize("kind", ["ids", "random"])
@pytest.mark.parametrize("n", [1, 127, 128, 2049, 4095, 4096, 4097, 4223, 4224, 9000])
def test_queues_of_one_block(n, kind):
    """Around two groups, up to which one block does a queue alone; async calls of
    changing lengths on one codec (a lone block leaves the counters as the whole
    grid does)."""
    x = values(kind, n, np.random.default_rng(n))
    c = g5.Codec(50_000)
    check(c, x)
    long = values(kind, 50_000, np.random.default_rng(1))
    for q in (x, long, x):
        din = torch.from_numpy(q.view(np.int32)).cuda()
        out = torch.empty(g5.Codec.bound(len(q)) + 8, dtype=torch.int32, device="cuda")
        back = torch.full((len(q) + 128,), -1, dtype=torch.int32, device="cuda")
        cnt = torch.tensor([len(q)], dtype=torch.int64, device="cuda")
        words, n_back = torch.zeros_like(cnt), torch.zeros_like(cnt)
        torch.cuda.synchronize()
        c.encode_async(din, cnt, out, words)
        c.decode_async(out, words, back, len(q) + 128, n_back)
        assert c.status() == 0 and int(n_back) == len(q)
        assert np.array_equal(out[:int(words)].cpu().numpy().view(np.uint32), orc.encode(q, MODES[0][1]))
        assert np.array_equal(back[:len(q)].cpu().numpy().view(np.uint32), q)
    c.close()
