"""CPU: the launches a frame that bench.py counts follow the library's rule for
the tile order."""
import importlib.util
import os
import re

import pytest

from conftest import ROOT
from ivr_gb300 import api, build


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_frame_launches(bench):
    for skip, n in ((api.SKIP_NONE, 1), (api.SKIP_GRID, 1), (api.SKIP_LEARNED, 3)):
        extra = 0 if skip == api.SKIP_NONE else 2
        assert bench.frame_launches(skip, "raster", 1920, 1080, 152) == n
        assert bench.frame_launches(skip, "cost", 1920, 1080, 152) == n + extra
        assert bench.frame_launches(skip, "cost", 512, 512, 152) == n
        assert bench.frame_launches(skip, "cost", 1280, 4 * 151 + 1, 152) == n + extra  # 24,320 tiles
        assert bench.frame_launches(skip, "cost", 1280, 4 * 151, 152) == n


def test_least_number_of_tiles_is_the_library_s(bench):
    with open(os.path.join(build.CSRC, "ivr_march.cu")) as f:
        src = f.read()
    per_warp = int(re.search(r"kTilesPerWarp = (\d+);", src).group(1))
    blocks = int(re.search(r"#define IVR_CFG_BLOCKS_PER_SM (\d+)", src).group(1))
    threads = int(re.search(r"constexpr int kThreads = (\d+);", src).group(1))
    assert bench.ORDER_TILES_PER_SM == per_warp * blocks * threads // 32
