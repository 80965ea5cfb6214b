"""The per-tile sort where lists are short: sizes around a warp's two rounds and a chunk's end side by
side in neighbouring tiles, in frames of few entries per tile (eight tiles per CTA) and of many."""
import numpy as np
import pytest

from test_gpu_tile_sort import CAM, check_order, renderer, scene

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 0, 2047, 2048, 2049, 0, 3, 64, 65, 1]


@pytest.mark.parametrize("n", [8192, 40_000])
@pytest.mark.parametrize("equal", [False, True])
def test_neighbouring_lists(n, equal):
    rng = np.random.default_rng(n)
    xyz = np.tile(np.float32([0, 0, -5]), (n, 1))  # behind the camera: entries without pairs
    at = rng.permutation(n)[: sum(SIZES)]
    z = np.full(at.size, 4.0) if equal else rng.uniform(2.0, 9.0, at.size)
    tile = np.repeat(np.arange(len(SIZES)), SIZES) + 25  # 20 tiles a row
    px, py = 16 * (tile % 20) + 8.0, 16 * (tile // 20) + 8.0
    xyz[at] = np.stack([(px - CAM.cx) / CAM.fx * z, (py - CAM.cy) / CAM.fy * z, z], 1)
    count = check_order(renderer(scene(n, xyz, -8.0)), CAM)
    np.testing.assert_array_equal(count[25: 25 + len(SIZES)], SIZES)
