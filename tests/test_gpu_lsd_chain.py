"""The LSD chain in frames below 8192 entries, and for a given projection of any size: 8- and 9-bit tile
digits, three and four depth passes, digits counted by their own kernels (needs a GPU)."""
import numpy as np
import pytest

import kat
from aniso_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ab():
    import aniso_b200

    return aniso_b200


def batch(ab, rs, view_scene, cams, options):
    import torch

    b = ab.BatchRenderer(rs, view_scene, options)
    outs = [torch.zeros((c.height, c.width, 3), dtype=torch.uint8, device="cuda") for c in cams]
    for attempt in range(3):
        b.render_device(cams, [o.data_ptr() for o in outs], torch.cuda.current_stream().cuda_stream)
        try:
            b.sync()
            break
        except ab.AnisoError as e:
            if "pair capacity" not in str(e) or attempt == 2:
                raise
    return [o.cpu().numpy() for o in outs]


@pytest.mark.parametrize("tile", [(16, 16), (8, 8)])
def test_nine_bit_digits_in_small_batches(ab, tile):
    """20 views of 400 Gaussians at 1280x720: 72,000 or 288,000 tiles, 8000 entries."""
    r = ab.GpuRenderer(*kat.random_cloud(400, seed=31))
    cams = []
    for k in range(20):
        c = kat.gpu_test_camera(1280, 720)
        yaw = 0.02 * (k - 10)
        R = np.array([[np.cos(yaw), 0, np.sin(yaw)], [0, 1, 0], [-np.sin(yaw), 0, np.cos(yaw)]])
        cams.append(scenes.Camera(1280, 720, c.fx, c.fy, c.cx, c.cy, R @ np.asarray(c.R), np.asarray(c.t)))
    nine = batch(ab, [r], [0] * 20, cams, ab.BatchOptions(tile=tile, radix_bits=9))
    eight = batch(ab, [r], [0] * 20, cams, ab.BatchOptions(tile=tile, radix_bits=8))
    for k in range(20):
        np.testing.assert_array_equal(nine[k], eight[k], err_msg="view %d" % k)
        np.testing.assert_array_equal(nine[k], r.render(cams[k]), err_msg="view %d" % k)
    assert any(i.any() for i in nine)


@pytest.mark.parametrize("graph", [False, True])
def test_near_and_far_scenes_in_a_small_batch(ab, graph):
    """A scene with Gaussians past depth 8192 makes the batch sort depths in four 8-bit passes; its views
    alone, and the near scene's, equal the batch's."""
    g, sh, d = kat.random_cloud(2000, seed=22)
    g = g.copy()
    ratio = np.float32(12000.0) / g[:500, 2]
    g[:500, 0] *= ratio
    g[:500, 1] *= ratio
    g[:500, 2] = 12000.0
    rs = [ab.GpuRenderer(*kat.random_cloud(2000, seed=21)), ab.GpuRenderer(g, sh, d)]
    cams = [kat.gpu_test_camera(320, 240), kat.gpu_test_camera(333, 217), kat.gpu_test_camera(320, 240)]
    view_scene = [0, 1, 1]
    for k, img in enumerate(batch(ab, rs, view_scene, cams, ab.BatchOptions(use_graph=graph))):
        np.testing.assert_array_equal(img, rs[view_scene[k]].render(cams[k]), err_msg="view %d" % k)
        assert img.any()


@pytest.mark.parametrize("n,far", [(50_000, False), (50_000, True), (4_300_000, False), (4_300_000, True)])
def test_given_projections_against_a_plain_sort(ab, n, far):
    """Above 4M entries the digits are counted by kernels of their own; depths past 8192 take four passes."""
    rng = np.random.default_rng(n + far)
    tx, ty = 40, 30
    x0, y0 = rng.integers(0, tx, n), rng.integers(0, ty, n)
    x1, y1 = np.minimum(x0 + rng.integers(0, 2, n), tx - 1), np.minimum(y0 + rng.integers(0, 2, n), ty - 1)
    depth = np.round(rng.uniform(0.5, 9000.0 if far else 90.0, n), 2).astype(np.float32)  # many are equal
    touched = ((x1 - x0 + 1) * (y1 - y0 + 1)).astype(np.uint32)
    touched[rng.random(n) < 0.3] = 0
    rect = np.stack([x0, y0, x1, y1], 1).astype(np.uint32)
    tiles, values, ranges = ab.sort_projection(touched, rect, depth, tx, ty)
    idx = np.nonzero(touched)[0]
    count = touched[idx].astype(np.int64)
    owner = np.repeat(np.arange(idx.size), count)
    k = np.arange(owner.size) - np.repeat(np.cumsum(count) - count, count)
    w = (x1 - x0 + 1)[idx][owner]
    tile = (y0[idx][owner] + k // w) * tx + x0[idx][owner] + k % w
    order = np.lexsort((idx[owner], depth[idx].view(np.uint32)[owner], tile))
    np.testing.assert_array_equal(tiles, tile[order])
    np.testing.assert_array_equal(values, idx[owner][order])
    size = np.bincount(tile, minlength=tx * ty)
    end = np.cumsum(size)
    np.testing.assert_array_equal(ranges, np.where(size[:, None] > 0, np.stack([end - size, end], 1), 0))
