"""The per-tile sort (frames of 8192 entries and more): sorted pairs and ranges against the order a
plain sort of the reported projection gives, where its parts can go wrong -- depths that are all equal
or crowd together, lists of one chunk (2048 pairs), of several, and of more than one group of chunks,
rectangles counted by a lane, a warp and a CTA, more tiles than one scan CTA takes -- and the training
path's cut rectangles against the persistent sort's whole ones (needs a GPU)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from aniso_b200 import scenes

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def check_order(r, cam):
    """debug_sorted against a stable sort of debug_projection's pairs by (tile, depth bits, index)."""
    p = r.debug_projection(cam)
    tx = (cam.width + 15) // 16
    idx = np.nonzero(p["tiles_touched"])[0]
    x0, y0, x1, y1 = p["rect"][idx].astype(np.int64).T
    w, n = x1 - x0 + 1, p["tiles_touched"][idx].astype(np.int64)
    owner = np.repeat(np.arange(idx.size), n)
    k = np.arange(owner.size) - np.repeat(np.cumsum(n) - n, n)
    tile = (y0[owner] + k // w[owner]) * tx + x0[owner] + k % w[owner]
    depth = p["depth"][idx].view(np.uint32)[owner]
    order = np.lexsort((idx[owner], depth, tile))
    tiles, values, ranges = r.debug_sorted(cam, capacity=max(1, owner.size))
    np.testing.assert_array_equal(values, idx[owner][order])
    np.testing.assert_array_equal(tiles, tile[order])
    count = np.bincount(tile, minlength=ranges.shape[0])
    end = np.cumsum(count)
    want = np.where(count[:, None] > 0, np.stack([end - count, end], 1), 0)
    np.testing.assert_array_equal(ranges, want)
    return count


def scene(n, xyz, log_scale, seed=0):
    raw = scenes.make_raw_scene(n, (-1, -1, -1), (1, 1, 1), seed, sh_degree=0)
    raw.xyz[:] = xyz
    raw.scale[:] = log_scale
    return raw


def renderer(raw):
    from aniso_b200 import GpuRenderer

    return GpuRenderer.from_raw(raw)


CAM = scenes.Camera(320, 208, 300.0, 300.0, 160.0, 104.0, np.eye(3), np.zeros(3))


@pytest.mark.parametrize("n", [8192, 8193, 50_000])
@pytest.mark.parametrize("depths", ["equal", "two", "crowded", "spread"])
def test_order_over_depth_distributions(n, depths):
    rng = np.random.default_rng(n)
    z = {"equal": np.full(n, 4.0), "two": np.where(rng.random(n) < 0.5, 4.0, 4.5),
         "crowded": np.where(rng.random(n) < 0.02, rng.uniform(1, 400, n), 4 + 1e-5 * rng.random(n)),
         "spread": rng.uniform(1.0, 9000.0, n)}[depths]
    xy = rng.uniform(-0.5, 0.5, (n, 2)) * z[:, None]
    check_order(renderer(scene(n, np.column_stack([xy, z]), np.log(0.01 * z)[:, None])), CAM)


@pytest.mark.parametrize("n", [2048 * 4, 40_000, 1_100_000])
def test_order_of_long_lists(n):
    """Everything in a few tiles: lists of several chunks, and (1.1M) of more than one group of 512."""
    rng = np.random.default_rng(n)
    z = rng.uniform(50.0, 60.0, n)
    xyz = np.column_stack([rng.uniform(0.2, 0.4, n), rng.uniform(0.2, 0.4, n), z])
    count = check_order(renderer(scene(n, xyz, -7.0)), CAM)
    assert count.max() > 2048 and (n < 1_000_000 or count.max() > 512 * 2048)


def test_order_of_exactly_full_chunks():
    """Lists of 2047, 2048, 2049 and 4096 pairs: points at the centres of four tiles."""
    sizes = [2047, 2048, 2049, 4096]
    cx = np.repeat([24.0, 72.0, 120.0, 168.0], sizes)
    n = cx.size
    rng = np.random.default_rng(1)
    z = rng.uniform(2.0, 3.0, n)
    xyz = np.column_stack([(cx - 160.0) / 300.0 * z, np.full(n, (24.0 - 104.0) / 300.0) * z, z])
    count = check_order(renderer(scene(n, xyz, -12.0)), CAM)
    assert sorted(count[count > 0]) == sizes


def test_order_with_rectangles_of_every_size():
    """From one tile to the whole view (8160 tiles: the CTA's share of the scatter, two scan CTAs)."""
    n = 9000
    rng = np.random.default_rng(2)
    cam = scenes.Camera(1920, 1088, 1000.0, 1000.0, 960.0, 544.0, np.eye(3), np.zeros(3))
    z = rng.uniform(2.0, 6.0, n)
    xyz = np.column_stack([rng.uniform(-0.9, 0.9, n) * z, rng.uniform(-0.5, 0.5, n) * z, z])
    scale = rng.uniform(-9.0, -4.0, n)
    scale[::90] = rng.uniform(-3.0, 2.0, scale[::90].size)
    check_order(renderer(scene(n, xyz, scale[:, None])), cam)


def test_more_tiles_than_the_direct_scan_takes():
    """Three 1920x1080 views in 8x8 tiles: 97,200 tiles (above 65,536 the CTAs' totals come first)."""
    import torch

    from aniso_b200 import BatchOptions, BatchRenderer

    raw = scenes.make_raw_scene(20_000, (-2, -1.2, 2), (2, 1.2, 5), 3)
    r = renderer(raw)
    cams = [scenes.Camera(1920, 1080, 1000.0 + 50 * k, 1000.0, 960.0, 540.0, np.eye(3), np.zeros(3)) for k in range(3)]
    b = BatchRenderer([r], [0] * 3, BatchOptions(3, 1.0, (8, 8), 128))
    outs = [torch.empty(c.height, c.width, 3, dtype=torch.uint8, device="cuda") for c in cams]
    for _ in range(3):
        b.render_device(cams, [o.data_ptr() for o in outs])
        try:
            b.sync()
            break
        except RuntimeError:
            pass
    for o, c in zip(outs, cams):
        np.testing.assert_array_equal(o.cpu().numpy(), r.render(c))


def test_stats_count_whole_rectangles_and_overflow_grows():
    """The pair count reported stays the reference's (whole rectangles), and a frame beyond the first
    pair capacity (2^20) grows it."""
    n = 9000
    rng = np.random.default_rng(4)
    z = rng.uniform(2.0, 3.0, n)
    raw = scene(n, np.column_stack([rng.uniform(-0.3, 0.3, n), rng.uniform(-0.3, 0.3, n), z]), -1.0)
    raw.opacity[:] = -4.5  # faint: the bounds where alpha reaches 1/255 are far inside three sigma
    cam = scenes.Camera(1280, 720, 1000.0, 1000.0, 640.0, 360.0, np.eye(3), np.zeros(3))
    r = renderer(raw)
    stats = {}
    img = r.render(cam, stats)
    touched = r.debug_projection(cam)["tiles_touched"].astype(np.int64)
    assert stats["tile_pairs"] == touched.sum() > 1 << 20
    assert stats["visible"] == np.count_nonzero(touched)
    np.testing.assert_array_equal(renderer(raw).render(cam), img)


CHILD = r"""
import sys, numpy as np
sys.path.insert(0, ROOT); sys.path.insert(0, ROOT + '/tests')
import torch
from aniso_b200 import scenes
from aniso_b200.autograd import rasterize, rasterize_batch
rng = np.random.default_rng(9)
n = 9000
xyz = np.stack([rng.uniform(-1.5, 1.5, n), rng.uniform(-1, 1, n), rng.uniform(2, 7, n)], 1)
scale = rng.normal(-3.2, 0.6, (n, 3)); scale[::100] += 3.0
P = [xyz, scale, rng.normal(0, 1, (n, 4)), rng.normal(-1, 2, n), rng.normal(0, 0.3, (n, 16, 3))]
ts = [torch.tensor(p, dtype=torch.float32, device='cuda', requires_grad=True) for p in P]
cam = scenes.Camera(333, 217, 300.0, 300.0, 166.5, 108.5, np.eye(3), np.zeros(3))
out = {}
img = rasterize(*ts, cam)
for k, g in enumerate(torch.autograd.grad(img.square().sum(), ts)):
    out['g%d' % k] = g.cpu().numpy()
out['img'] = img.detach().cpu().numpy()
imgs = rasterize_batch([ts], [cam, cam], [0, 0], tile=(16, 32), use_graph=True)
for k, g in enumerate(torch.autograd.grad(sum(i.square().sum() for i in imgs), ts)):
    out['b%d' % k] = g.cpu().numpy()
np.savez(OUT, **out)
"""


def test_training_equals_the_persistent_sort(tmp_path):
    """Image and gradients bit for bit: the cut rectangles leave out only zeros, in the same order."""
    got = {}
    for mode in ("default", "persistent"):
        path = str(tmp_path / (mode + ".npz"))
        env = {k: v for k, v in os.environ.items() if k != "ANISO_B200_SORT"}
        if mode == "persistent":
            env["ANISO_B200_SORT"] = "persistent"
        run = subprocess.run([sys.executable, "-c", "ROOT = %r\nOUT = %r\n" % (ROOT, path) + CHILD], env=env,
                             capture_output=True, text=True, timeout=600)
        assert run.returncode == 0, run.stdout[-2000:] + run.stderr[-2000:]
        got[mode] = dict(np.load(path))
    for key in sorted(got["default"]):
        np.testing.assert_array_equal(got["default"][key], got["persistent"][key], err_msg=key)
    assert got["default"]["img"].any()
