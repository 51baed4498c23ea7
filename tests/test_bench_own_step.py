"""bench.py tells the library's own step (one launch where the grid is small
enough) from a tiling or two steps per pass, whose kernels its per-kernel pass
times."""
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))

import bench  # noqa: E402


@pytest.mark.parametrize("planes,active,own", [(0, False, True), (16, False, False), (0, True, False), (16, True, False)])
def test_own_step(planes, active, own):
    assert bench.own_step({"tiling": {"planes_per_block": planes}, "time_blocking": {"active": active}}) is own
