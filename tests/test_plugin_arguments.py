"""The plugin looks at the ids before anything else can fail: one that does not fit
in 32 bits is an invalid argument with or without a device."""
import ctypes as C

import numpy as np
import pytest

import gpugraph500_gb300 as g5


@pytest.mark.parametrize("size", [1, 64, 65, 3000])
@pytest.mark.parametrize("bad", [-1, 1 << 32, 1 << 62, -(1 << 40)])
@pytest.mark.parametrize("at", [0, -1])
def test_ids_past_32_bits(size, bad, at):
    q = np.arange(size, dtype=np.int64)
    q[at] = bad
    out, n = C.c_void_p(), C.c_size_t()
    code = g5.lib().g5_plugin_compress(q.ctypes.data, size, C.byref(out), C.byref(n), 64, g5.CODEC_DM)
    assert code == g5.G5_ERR_INVALID_ARG and not out.value
