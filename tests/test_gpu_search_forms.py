"""The kernel of the one-launch search by itself, in the forms and offset widths
that the library chooses by the graph's size only: small graphs take all of them
here.  And a wait that runs out: the search reports it, one queued behind it
does too, and a cleared ring serves the next."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WAIT = 16  # G5_DEVERR_WAIT


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    from gpugraph500_gb300 import build
    path = str(tmp_path_factory.mktemp("forms") / "search_forms")
    subprocess.run([build._nvcc(), *build.ARCH, "-O2", "-std=c++17", "-DG5_MEET_NS=50000000ull",
                    "-I" + build.INCLUDE, "-I" + build.CSRC, os.path.join(ROOT, "tests", "cpp", "search_forms.cu"),
                    "-o", path], check=True)
    return path


def graph_file(path, ro, col):
    with open(path, "wb") as f:
        np.array([len(ro) - 1, len(col)], np.int64).tofile(f)
        np.asarray(ro, np.int64).tofile(f)
        np.asarray(col, np.uint32).tofile(f)
    return str(path)


def run(exe, *args):
    r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr)


def graphs():
    rng = np.random.default_rng(5)
    yield "path", *orc.build_csr(70, np.array([(i, i + 1) for i in range(60)], np.int64))
    yield "star and hubs", *orc.build_csr(3001, np.concatenate([
        np.stack([np.zeros(3000, np.int64), np.arange(1, 3001)], 1), rng.integers(0, 3001, (4000, 2))]))
    yield "kronecker", *orc.build_csr(1 << 15, orc.kronecker(15))
    yield "ragged", *orc.build_csr(200_003, rng.integers(0, 200_003, (700_000, 2)))


@pytest.mark.parametrize("which", range(4))
def test_every_form_and_offset_width(exe, tmp_path, which):
    name, ro, col = list(graphs())[which]
    n = len(ro) - 1
    roots = [0, n // 2, n - 1] + [int(r) for r in np.argsort(np.diff(ro))[-2:]]
    out = tmp_path / "out"
    run(exe, "parents", graph_file(tmp_path / "g", ro, col), out, *roots)
    raw = open(out, "rb").read()
    forms = 3 if n > 4096 else 4
    assert len(raw) == 2 * forms * len(roots) * 12 * n
    at = 0
    for wide in range(2):
        for form in range(forms):
            for r in roots:
                pred, level = orc.bfs(ro, col, r)
                assert np.array_equal(np.frombuffer(raw, np.int64, n, at), pred), (name, wide, form, r)
                assert np.array_equal(np.frombuffer(raw, np.int32, n, at + 8 * n), level), (name, wide, form, r)
                at += 12 * n


def test_clusters_that_do_not_fit(exe, tmp_path):
    """No device holds a cluster of 32 blocks; the answer leaves no error behind."""
    ro, col = orc.build_csr(4, np.array([(0, 1)], np.int64))
    out = tmp_path / "out"
    run(exe, "clusters", graph_file(tmp_path / "g", ro, col), out, 32, 1, 8, 64)
    assert np.fromfile(out, np.int64).tolist() == [0, 1, 1, 0]


def test_waits_that_run_out(exe, tmp_path):
    n = 20_000
    ro, col = orc.build_csr(n, np.random.default_rng(1).integers(0, n, (90_000, 2)))
    out = tmp_path / "out"
    run(exe, "waits", graph_file(tmp_path / "g", ro, col), out, 7)
    got = np.fromfile(out, np.int64).reshape(2, 3, n + 1)  # grid forms, searches, error bits and parents
    want = orc.bfs(ro, col, 7)[0]
    for form in got:
        assert form[:, 0].tolist() == [WAIT, WAIT, 0]
        for p in form[:2, 1:]:  # they gave up before their first level
            assert p[7] == 7 and (np.delete(p, 7) == -1).all()
        assert np.array_equal(form[2, 1:], want)
