"""The tuner's tile sizes are all different searches: the one-launch search takes
no tile below its smallest work item (host logic, CPU)."""
import os
import re

from gpugraph500_gb300 import build, tune


def test_no_tile_below_the_smallest_item():
    with open(os.path.join(build.CSRC, "g5_search.cuh")) as f:
        shift = int(re.search(r"constexpr int kMinItemShift = (\d+);", f.read()).group(1))
    assert min(tune.TILES) >= 1 << shift
    assert len({max(t, 1 << shift) for t in tune.TILES}) == len(tune.TILES)
    assert tune.DEFAULT_SIZES[0] in tune.TILES
