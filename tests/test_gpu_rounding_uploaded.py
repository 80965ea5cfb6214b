"""Uploaded scenes, every colour degree: the preprocess's instantiations (one Gaussian per thread, two, many
views of a scene) give the same images and projections (needs a GPU)."""
import numpy as np
import pytest

import kat
from aniso_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [0, 1, 2, 3])
def test_company_and_views_leave_every_byte(degree):
    import torch

    from aniso_b200 import BatchOptions, BatchRenderer, GpuRenderer

    n = 20_000
    g, sh, _ = kat.random_cloud(n, seed=40 + degree)
    sh = np.ascontiguousarray(sh[:, : 3 * (degree + 1) ** 2])
    behind = np.tile(g[:1], (1 << 19, 1))
    behind[:, 2] = -5.0
    alone = GpuRenderer(g, sh, degree)
    together = GpuRenderer(np.concatenate([g, behind]), np.concatenate([sh, np.tile(sh[:1], (1 << 19, 1))]), degree)
    cam = scenes.Camera(640, 360, 500.0, 500.0, 320.0, 180.0, np.eye(3), np.zeros(3))
    image = alone.render(cam)
    assert image.any()
    np.testing.assert_array_equal(image, together.render(cam))
    p, q = alone.debug_projection(cam), together.debug_projection(cam)
    seen = p["tiles_touched"] > 0
    np.testing.assert_array_equal(p["tiles_touched"], q["tiles_touched"][:n])
    for key in ("uv", "conic_opacity", "depth", "rgb", "rect"):
        np.testing.assert_array_equal(p[key][seen], q[key][:n][seen], err_msg=key)
    views = 6  # of one scene: one Gaussian per thread, whatever its size
    b = BatchRenderer([together], [0] * views, BatchOptions(3, 1.0, (16, 16), 256))
    outs = [torch.zeros(360, 640, 3, dtype=torch.uint8, device="cuda") for _ in range(views)]
    b.render_device([cam] * views, [o.data_ptr() for o in outs])
    b.sync()
    for o in outs:
        np.testing.assert_array_equal(image, o.cpu().numpy())
