"""The one-launch decoder at the sizes where its paths change: one chunk and
many, more chunks than one look takes in, streams whose every vector could be
a group header, raw miniblocks that restart the sums, groups of one vector,
chunks that end in the tail.  Streams come from the oracle encoder, values
must come back exactly, and damaged streams are refused."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")

MODES = [(g5.CODEC_D4, orc.D4), (g5.CODEC_DM, orc.DM)]


def values(kind, n, rng):
    if kind == "ids":      # a frontier: about one id in three
        return np.cumsum(rng.integers(1, 6, n), dtype=np.uint64).astype(np.uint32)
    if kind == "equal":    # every delta 0: groups of one vector, every vector a header
        return np.full(n, 7, np.uint32)
    if kind == "steps":    # deltas of 0 and 1: narrow payloads that look like headers
        return np.cumsum(rng.integers(0, 2, n) * (rng.random(n) < 0.02), dtype=np.uint64).astype(np.uint32)
    if kind == "random":   # unsorted: mostly raw 32-bit miniblocks
        return rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    # sorted runs with jumps back: raw miniblocks between packed ones
    x = np.cumsum(rng.integers(1, 40, n), dtype=np.uint64)
    for at in range(1000, n, 5000):
        x[at:] -= min(int(x[at]), 100_000)
    return (x & 0xFFFFFFFF).astype(np.uint32)


def decode(codec, stream, n, mode):
    din = torch.from_numpy(stream.view(np.int32)).cuda()
    out = torch.full((n + 256,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    m = codec.decode(din, len(stream), out, n + 128, mode)
    got = out.cpu().numpy().view(np.uint32)
    return got[:m], got[m:]


@pytest.mark.parametrize("kind", ["ids", "equal", "steps", "random", "jumps"])
@pytest.mark.parametrize("n", [1, 127, 128, 2047, 2048, 2049, 40_000, 1_000_003, 3_000_001])
def test_values_come_back(kind, n):
    rng = np.random.default_rng(n)
    x = values(kind, n, rng)
    c = g5.Codec(n + 128)
    for mode, omode in MODES:
        s = orc.encode(x, omode)
        for _ in range(2):  # records of the call before are not read
            got, rest = decode(c, s, n, mode)
            assert np.array_equal(got, x), (kind, n, mode)
            assert (rest == 0xFFFFFFFF).all()
    c.close()


def test_more_chunks_than_one_look():
    """32-bit miniblocks: over 800,000 vectors, more than 512 chunks, in two waves."""
    n = 4_000_000
    x = values("random", n, np.random.default_rng(3))
    c = g5.Codec(n)
    for mode, omode in MODES:
        got, _ = decode(c, orc.encode(x, omode), n, mode)
        assert np.array_equal(got, x)
    c.close()


def test_damaged_streams_are_refused():
    n = 600_000
    rng = np.random.default_rng(9)
    x = values("ids", n, rng)
    c = g5.Codec(n + 128)
    for mode, omode in MODES:
        s = orc.encode(x, omode)
        bad = []
        b = s.copy(); b[4] ^= 0x01000000; bad.append(b)                 # the first group's length
        b = s.copy(); b[4] = 0x21212121; bad.append(b)                  # widths above 32
        b = s.copy(); b[0] -= 128 * 400; bad.append(b)                  # ends in the middle: too much tail
        b = s.copy(); b[0] += 128 * 40; bad.append(b)                   # ends before its last group
        bad.append(s[: len(s) // 2].copy())
        bad.append(s[: len(s) // 3 // 4 * 4].copy())
        bad.append(np.concatenate([s[:20000], s[20400:]]))              # a piece taken out
        for b in bad:
            with pytest.raises(g5.G5Error):
                decode(c, b, n, mode)
        got, _ = decode(c, s, n, mode)  # the workspace still works
        assert np.array_equal(got, x)
    c.close()


@pytest.mark.parametrize("n", [128 * 5, 128 * (16 * 40 + 3), 128 * (16 * 900 + 7) + 55])
def test_last_group_header_past_its_miniblocks(n):
    """The width bytes past the last group's miniblocks are not looked at."""
    x = values("ids", n, np.random.default_rng(n))
    c = g5.Codec(n + 128)
    for mode, omode in MODES:
        s = orc.encode(x, omode)
        p = 4  # the last group's header, down the chain
        for _ in range((n // 128 + 15) // 16 - 1):
            p += 4 + 4 * int(s[p:p + 4].view(np.uint8).sum())
        b = s.copy()
        b[p + 3] |= 0x000000FF  # width 15 of the group
        got, _ = decode(c, b, n, mode)
        assert np.array_equal(got, x)
    c.close()
