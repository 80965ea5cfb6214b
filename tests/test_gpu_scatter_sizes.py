"""The tile sort's scatter in each of its sizes of frame (up to 37888 entries, up to 2^21, above), with
rectangles from one tile to the whole view (8160 tiles), and lists whose chunks are merged: one pair in the
last chunk, and chunks of unequal depth ranges (needs a GPU)."""
import numpy as np
import pytest

from test_gpu_tile_sort import CAM, check_order, renderer, scene

from aniso_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [37_888, 37_889, (1 << 21) + 1])
def test_order_with_rectangles_of_every_size(n):
    rng = np.random.default_rng(n)
    cam = scenes.Camera(1920, 1088, 1000.0, 1000.0, 960.0, 544.0, np.eye(3), np.zeros(3))
    z = rng.uniform(2.0, 6.0, n)
    xyz = np.column_stack([rng.uniform(-0.9, 0.9, n) * z, rng.uniform(-0.5, 0.5, n) * z, z])
    scale = rng.uniform(-9.0, -6.0, n)
    big = slice(0, None, n // 100)
    scale[big] = rng.uniform(-3.0, 2.0, scale[big].size)
    check_order(renderer(scene(n, xyz, scale[:, None])), cam)


@pytest.mark.parametrize("n", [8193, 12_289, 20_000])
@pytest.mark.parametrize("sorted_input", [False, True])
def test_order_of_merged_chunks(n, sorted_input):
    """All pairs in one tile. With the input in depth order the chunks hold different depths: a merge then
    takes whole stretches from one side."""
    rng = np.random.default_rng(n)
    z = rng.uniform(2.0, 9.0, n)
    z[: n // 5] = 5.0
    if sorted_input:
        z.sort()
    u, v = 16 * 7 + 8.0, 16 * 5 + 8.0
    xyz = np.column_stack([(u - CAM.cx) / CAM.fx * z, (v - CAM.cy) / CAM.fy * z, z])
    count = check_order(renderer(scene(n, xyz, -12.0)), CAM)
    assert count.max() == n
