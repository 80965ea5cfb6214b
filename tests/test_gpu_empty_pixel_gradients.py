"""A pixel that no splat reaches takes no part in the adjoint, whatever its upstream gradient: sqrt of the
image, say, has an infinite one at 0 (needs a GPU)."""
import numpy as np
import pytest

from aniso_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (16, 32)])
def test_gradients_of_empty_pixels_are_not_read(bad, tile):
    import torch

    from aniso_b200.autograd import rasterize_batch

    rng = np.random.default_rng(8)
    n = 400
    z = rng.uniform(2, 5, n)
    arrs = [np.stack([rng.uniform(-0.6, 0.6, n) * z, rng.uniform(-0.5, 0.5, n) * z, z], 1), rng.normal(-5, 0.7, (n, 3)),
            rng.normal(0, 1, (n, 4)), rng.normal(0, 1, n), np.full((n, 16, 3), 0.02)]
    leaves = [torch.tensor(a, dtype=torch.float32, device="cuda", requires_grad=True) for a in arrs]
    cam = scenes.Camera(150, 115, 120.0, 120.0, 75.0, 57.5, np.eye(3), np.zeros(3))

    def grads(up):
        (img,) = rasterize_batch([leaves], [cam], [0], tile=tile, use_graph=False)
        return img.detach(), torch.autograd.grad(img, leaves, up)

    up = torch.randn(cam.height, cam.width, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    lit = grads(up)[0].sum(-1) > 0
    pair = lit.view(cam.height, -1, 2).any(-1).repeat_interleave(2, 1)  # a lane's two pixels
    assert lit.any() and (~pair).any()
    _, want = grads(torch.where(pair[..., None], up, torch.zeros_like(up)))
    _, got = grads(torch.where(pair[..., None], up, torch.full_like(up, bad)))
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
