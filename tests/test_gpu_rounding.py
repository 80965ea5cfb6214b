"""The projection rounds alike in every instantiation of the preprocess kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 3])
def test_culled_company_leaves_every_bit(degree):
    """2^19 Gaussians behind the camera take the frame to two Gaussians per thread; the image of the
    20000 in front of it keeps its bits (float32, through the training path)."""
    from aniso_b200.autograd import rasterize
    from aniso_b200.scenes import Camera
    import numpy as np

    g = torch.Generator(device="cuda").manual_seed(3)
    n, k = 20_000, (degree + 1) ** 2
    lo, hi = (torch.tensor(v, device="cuda") for v in ((-4.0, -4.0, 2.0), (4.0, 4.0, 12.0)))
    raw = [lo + (hi - lo) * torch.rand(n, 3, device="cuda", generator=g),
           torch.randn(n, 3, device="cuda", generator=g) * 0.5 - 3.0,
           torch.randn(n, 4, device="cuda", generator=g),
           torch.randn(n, device="cuda", generator=g),
           torch.randn(n, k, 3, device="cuda", generator=g) * 0.3]
    behind = [t[:1].expand(1 << 19, *t.shape[1:]).clone() for t in raw]
    behind[0][:, 2] = -5.0
    camera = Camera(640, 360, 500.0, 500.0, 320.0, 180.0, np.eye(3), np.zeros(3), "origin")
    with torch.no_grad():
        alone = rasterize(*raw, camera)
        together = rasterize(*[torch.cat(p) for p in zip(raw, behind)], camera)
    assert alone.abs().sum() > 0
    assert torch.equal(alone, together)
