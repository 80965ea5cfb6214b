"""A training batch whose views move to other scenes between steps is recorded again, also where every
size that the launches depend on stays as it was (needs a GPU)."""
import numpy as np
import pytest

from test_gpu_train_graph import assert_same, cameras, params_of, step

from aniso_b200 import scenes

pytestmark = pytest.mark.gpu


def test_views_change_places_between_equal_scenes():
    import torch

    sc = [params_of(torch, 2000, 51), params_of(torch, 2000, 52)]
    cams = [cameras(0.03)[0]] * 2
    gen = torch.Generator(device="cuda").manual_seed(3)
    ups = [torch.randn((c.height, c.width, 3), device="cuda", generator=gen) for c in cams]
    for view_scene in ([0, 1], [1, 0], [0, 1]):
        got = step(torch, sc, cams, view_scene, ups, use_graph=True)
        assert_same(got, step(torch, sc, cams, view_scene, ups, use_graph=False), str(view_scene))


def test_views_move_to_a_scene_with_longer_lists():
    """The same entries, tiles and blocks, but a tile's list can now exceed one sorted chunk (2048 pairs):
    3072 splats in front of one tile."""
    import torch

    sc = []
    for k, n in enumerate((2048, 2048, 2048, 2048, 1024, 3072)):
        rng = np.random.default_rng(60 + k)
        z = rng.uniform(3, 7, n)
        arrs = [np.stack([rng.uniform(0.0, 0.02, n) * z, rng.uniform(0.0, 0.02, n) * z, z], 1), rng.normal(-6, 0.2, (n, 3)),
                rng.normal(0, 1, (n, 4)), rng.normal(-3, 1, n), rng.normal(0, 0.3, (n, 16, 3))]
        sc.append([torch.tensor(a, dtype=torch.float32, device="cuda") for a in arrs])
    cams = [scenes.Camera(64, 48, 100.0, 100.0, 33.0, 17.0, np.eye(3), np.zeros(3))] * 4
    gen = torch.Generator(device="cuda").manual_seed(4)
    ups = [torch.randn((c.height, c.width, 3), device="cuda", generator=gen) for c in cams]
    for view_scene in ([0, 1, 2, 3], [0, 1, 4, 5]):
        got = step(torch, sc, cams, view_scene, ups, use_graph=True)
        assert_same(got, step(torch, sc, cams, view_scene, ups, use_graph=False), str(view_scene))
        assert all(i.any() for i in got[0])
