"""Streams that end before their first group: the header announces whole
miniblocks, the words are those of the header alone and up to three more.  Each
form of the decoder refuses them, and a well-formed stream still decodes."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")

MODES = [(g5.CODEC_D4, orc.D4), (g5.CODEC_DM, orc.DM)]
CUTS = [0, 1, 3, 4, 5, 6, 7, 8, 9]  # words kept; 8 and 9 hold the first group's header and no payload


def ids(n):
    return np.cumsum(np.random.default_rng(n).integers(1, 9, n), dtype=np.uint64).astype(np.uint32)


def device(words):
    t = torch.zeros(len(words) + 16, dtype=torch.int32, device="cuda")
    t[:len(words)] = torch.from_numpy(words.view(np.int32)).cuda()
    return t


@pytest.mark.parametrize("n", [128, 2048, 5000, 100_000])
@pytest.mark.parametrize("cut", CUTS)
def test_cut_streams_are_refused(n, cut):
    x = ids(n)
    c = g5.Codec(n + 128)
    out = torch.zeros(n + 128, dtype=torch.int32, device="cuda")
    count = torch.zeros(2, dtype=torch.int64, device="cuda")
    for mode, omode in MODES:
        s = orc.encode(x, omode)
        d = device(s)
        torch.cuda.synchronize()
        with pytest.raises(g5.G5Error) as e:
            c.decode(d, cut, out, n, mode)
        assert e.value.code == g5.G5_ERR_CORRUPT_STREAM
        # the length in device memory
        count[0], count[1] = cut, -1
        torch.cuda.synchronize()
        c.decode_async(d, count[0:], out, n, count[1:], mode, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert c.status() == g5.G5_ERR_CORRUPT_STREAM and int(count[1]) == 0
        # one of a batch
        with pytest.raises(g5.G5Error) as e:
            c.decode_batch(d, np.array([0], np.uint64), [cut], [n], out, mode=mode)
        assert e.value.stream_ok.tolist() == [0]
        assert c.decode(d, len(s), out, n, mode) == n
        assert np.array_equal(out.cpu().numpy().view(np.uint32)[:n], x)
    c.close()


@pytest.mark.parametrize("cut", CUTS)
def test_the_plugin_refuses_them(cut):
    x = ids(3000).astype(np.int64)
    p = g5.GpuSimd()
    s, size = p.compress(x)
    with pytest.raises(g5.G5Error) as e:
        p.decompress(s, cut, len(x))
    assert e.value.code == g5.G5_ERR_CORRUPT_STREAM
    assert np.array_equal(p.decompress(s, size, len(x)), x)
