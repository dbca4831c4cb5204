"""g5_bfs_poll takes the result of a launch once: after other calls it changes
nothing that they left, and its device time is that of the last run or launch."""
import ctypes as C
import time

import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

g5 = pytest.importorskip("gpugraph500_gb300")
torch = pytest.importorskip("torch")


def poll(b, wait=False):
    done, ms = C.c_int(), C.c_double(-1.0)
    while True:
        code = g5.lib().g5_bfs_poll(b._h, C.byref(done), C.byref(ms))
        if done.value or not wait:
            return code, done.value, ms.value


def launch(b, root):
    assert g5.lib().g5_bfs_launch(b._h, int(root)) == 0


@pytest.fixture(scope="module", params=[2000, 20_000, 200_000])
def graph(request):
    n = request.param
    ro, col = orc.build_csr(n, np.random.default_rng(n).integers(0, n, (5 * n, 2)))
    g = g5.Graph.from_csr(ro, col)
    yield g
    g.close()


@pytest.mark.parametrize("kw", [{}, {"want_levels": True}, {"codec": 1}])
@pytest.mark.parametrize("first", ["nothing", "run", "launch"])
def test_after_many(graph, kw, first):
    b, one = g5.CudaBFS(graph, **kw), g5.CudaBFS(graph, **kw)
    if first == "run":
        assert b.run(5, None) == 0
    if first == "launch":
        launch(b, 5)
        assert poll(b, wait=True)[:2] == (0, 1)
    b.run_many([1, 7, 3, 11, 2], None)
    assert one.run(2, None) == 0
    for _ in range(2):
        assert poll(b)[:2] == (0, 1)
        assert np.array_equal(b.level_log(), one.level_log())
    launch(b, 3)  # and a launch's own result arrives
    assert poll(b, wait=True)[:2] == (0, 1)
    assert one.run(3, None) == 0
    assert np.array_equal(b.level_log(), one.level_log())
    b.close()
    one.close()


def test_an_earlier_failure_is_not_reported_again():
    n = 300
    ro, col = orc.build_csr(n, np.array([(i, i + 1) for i in range(n - 1)], np.int64))
    g = g5.Graph.from_csr(ro, col)
    b = g5.CudaBFS(g, max_levels=200)
    launch(b, 0)  # 299 levels
    assert poll(b, wait=True)[:2] == (g5.G5_ERR_TIMEOUT, 1)
    assert poll(b)[:2] == (g5.G5_ERR_TIMEOUT, 1)  # (still the last call's status)
    b.run_many([140, 150], None)
    assert poll(b)[:2] == (0, 1)
    assert b.run(0, None, stats=False) == g5.G5_ERR_TIMEOUT
    assert poll(b)[:2] == (g5.G5_ERR_TIMEOUT, 1)
    assert b.run(150, None, stats=False) == 0
    assert poll(b)[:2] == (0, 1)
    b.close()
    g.close()


def test_device_time_of_a_run_without_stats(graph):
    b = g5.CudaBFS(graph)
    for root in (1, 2, 3):
        t = time.perf_counter()
        assert b.run(root, None, stats=False) == 0
        wall = (time.perf_counter() - t) * 1e3
        code, done, ms = poll(b)
        assert (code, done) == (0, 1) and 0 < ms <= wall + 0.002  # (the clock steps by a microsecond or less)
    assert b.run(4, None, stats=True) == 0
    assert poll(b)[2] == b.stats.device_ms
    b.close()


def test_poll_leaves_no_error_behind(graph):
    b = g5.CudaBFS(graph)
    assert b.run(1, None, stats=False) == 0
    assert poll(b)[:2] == (0, 1)
    c = g5.Codec(1000)
    x = torch.arange(1000, dtype=torch.int32, device="cuda")
    out = torch.zeros(g5.Codec.bound(1000), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert c.encode(x, 1000, out) > 0
    c.close()
    b.close()
