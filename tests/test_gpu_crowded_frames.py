"""Frames of many visible entries per tile are sorted by the LSD chain, on whole rectangles; the same view
beside a large, nearly empty one is sorted per tile, on cut ones. Both give the same images and gradients
(needs a GPU)."""
import numpy as np
import pytest

from aniso_b200 import scenes

pytestmark = pytest.mark.gpu

SMALL = scenes.Camera(61, 47, 50.0, 50.0, 30.0, 23.0, np.eye(3), np.zeros(3))
AWAY = scenes.Camera(1280, 720, 900.0, 900.0, 640.0, 360.0, np.diag([1.0, -1.0, -1.0]), np.zeros(3))  # looks along -z


def arrays(n, seed):
    rng = np.random.default_rng(seed)
    z = rng.uniform(2, 9, n)
    z[: n // 8] = 4.0  # equal depths: the index decides
    return [np.stack([rng.uniform(-0.7, 0.7, n) * z, rng.uniform(-0.6, 0.6, n) * z, z], 1), rng.normal(-5, 0.8, (n, 3)),
            rng.normal(0, 1, (n, 4)), rng.normal(-2, 1.5, n), rng.normal(0, 0.2, (n, 16, 3))]


# 12 tiles of 16x16, 11 of them within the scene's box at its centre's depth, and a quarter of the entries:
# the line lies near 88000. 600000 with eight views: more than the kernels that write the keys count digits for.
@pytest.mark.parametrize("n,views", [(60_000, 1), (100_000, 1), (150_000, 2), (600_000, 8)])
def test_images_equal_those_of_the_tile_sort(n, views):
    import torch

    from aniso_b200 import BatchOptions, BatchRenderer

    r = uploaded(n)
    small = [scenes.Camera(SMALL.width, SMALL.height, 50.0 + k, 50.0 + k, 30.0, 23.0, np.eye(3), np.zeros(3))
             for k in range(views)]
    got = []
    for cams in (small, small + [AWAY] * views):
        b = BatchRenderer([r], [0] * len(cams), BatchOptions(3, 1.0, (16, 16), 256))
        outs = [torch.full((c.height, c.width, 3), 9, dtype=torch.uint8, device="cuda") for c in cams]
        for attempt in range(3):
            b.render_device(cams, [o.data_ptr() for o in outs])
            try:
                b.sync()
                break
            except RuntimeError:
                assert attempt < 2
        got.append([o.cpu().numpy() for o in outs])
    for k in range(views):
        assert got[0][k].any()
        np.testing.assert_array_equal(got[0][k], got[1][k])
        np.testing.assert_array_equal(got[0][k], r.render(small[k]))


def far(tz, f, w=1280, h=720):
    return scenes.Camera(w, h, f, f, w / 2, h / 2, np.eye(3), np.array([0.0, 0.0, tz]))


def uploaded(n):
    from aniso_b200 import GpuRenderer

    a = arrays(n, n)
    g = np.concatenate([a[0], np.exp(a[1]), a[2] / np.linalg.norm(a[2], axis=1, keepdims=True),
                        1 / (1 + np.exp(-a[3]))[:, None]], 1).astype(np.float32)
    return GpuRenderer(g, a[4].reshape(n, -1).astype(np.float32), 3)


def test_scene_seen_from_afar_equals_the_tile_sort():
    """60000 Gaussians on eight tiles of 3600; a recorded batch whose camera goes there and back, beside one
    that another view keeps on the tile sort; a scene beside the view, and one that fills it."""
    import torch

    from aniso_b200 import BatchOptions, BatchRenderer

    r = uploaded(60_000)
    alone, beside = (BatchRenderer([r], [0] * k, BatchOptions(3, 1.0, (16, 16), 256)) for k in (1, 2))
    outs = [torch.zeros(720, 1280, 3, dtype=torch.uint8, device="cuda") for _ in range(3)]
    aside = scenes.Camera(1280, 720, 400.0, 400.0, 640.0, 360.0, np.eye(3), np.array([500.0, 0.0, 100.0]))
    for k, cam in enumerate((far(100.0, 400.0), far(0.0, 400.0), far(100.0, 400.0), aside, far(100.0, 9000.0))):
        for b, cams, ptrs in ((alone, [cam], outs[:1]), (beside, [cam, AWAY], outs[1:])):
            for attempt in range(3):
                b.render_device(cams, [o.data_ptr() for o in ptrs])
                try:
                    b.sync()
                    break
                except RuntimeError:
                    assert attempt < 2
        assert bool(outs[0].any()) == (cam is not aside)
        np.testing.assert_array_equal(outs[0].cpu().numpy(), outs[1].cpu().numpy(), err_msg=str(k))
        np.testing.assert_array_equal(outs[0].cpu().numpy(), r.render(cam), err_msg=str(k))


# In training the line lies at 4000 / 0.45 entries per tile, 106667 here.
@pytest.mark.parametrize("n", [106_000, 107_000, 130_000])
@pytest.mark.parametrize("graph", [False, True])
def test_gradients_equal_those_of_the_tile_sort(n, graph):
    import torch

    from aniso_b200.autograd import rasterize_batch

    raw = [torch.tensor(a, dtype=torch.float32, device="cuda") for a in arrays(n, n)]
    up = torch.randn(SMALL.height, SMALL.width, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6))
    got = []
    for cams in ([SMALL], [SMALL, AWAY]):
        leaves = [t.clone().requires_grad_(True) for t in raw]
        imgs = rasterize_batch([leaves], cams, [0] * len(cams), use_graph=graph)
        ups = [up] + [torch.zeros_like(i) for i in imgs[1:]]
        got.append([imgs[0].detach()] + list(torch.autograd.grad(imgs, leaves, ups)))
    assert got[0][0].any() and got[0][1].any()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
