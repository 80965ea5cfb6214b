"""The training loop's loss kernels (GPU) against the same loss in 64 bits, at image sizes around the
window (11) and the kernels' 32-pixel tiles (with the window's 10-pixel halo)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height,width", [(11, 11), (11, 75), (32, 33), (42, 43), (53, 97), (129, 200), (720, 1280)])
def test_loss_and_gradient_match_64_bits(height, width):
    import torch
    import torch.nn.functional as F

    from aniso_b200 import train

    gen = torch.Generator(device="cuda").manual_seed(height * 10_000 + width)
    r = lambda: torch.rand(height, width, 3, device="cuda", generator=gen)  # noqa: E731
    base = F.interpolate(torch.rand(1, 3, 9, 9, device="cuda", generator=gen), (height, width), mode="bilinear")[0]
    target = base.permute(1, 2, 0).contiguous()
    img = (target + 0.1 * (r() - 0.5)).requires_grad_(True)
    with torch.no_grad():
        img[height // 2] = target[height // 2]  # equal pixels: the L1 term has no slope there
    loss = train._loss(img, target)
    (grad,) = torch.autograd.grad(3.0 * loss, img)

    x, y = img.detach().double().requires_grad_(True), target.double()
    g = torch.exp(-((torch.arange(11, device="cuda") - 5) ** 2).double() / 4.5)
    w = (g[:, None] * g[None, :] / g.sum() ** 2)[None, None].repeat(3, 1, 1, 1)
    blur = lambda t: F.conv2d(t.permute(2, 0, 1)[None], w, groups=3)  # noqa: E731
    mx, my = blur(x), blur(y)
    sxx, syy, sxy = blur(x * x) - mx ** 2, blur(y * y) - my ** 2, blur(x * y) - mx * my
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    s = ((2 * mx * my + c1) * (2 * sxy + c2)) / ((mx ** 2 + my ** 2 + c1) * (sxx + syy + c2))
    want = 0.8 * (x - y).abs().mean() + 0.2 * (1 - s.mean())
    (want_grad,) = torch.autograd.grad(3.0 * want, x)
    # Variances are differences of fp32 sums near 1: absolute error about 2^-22 against B2 >= 9e-4, so
    # relative errors of a window's terms stay below 3e-4 and, over the image, far below.
    assert abs(loss.item() - float(want)) <= 1e-5
    assert float((grad.double() - want_grad).norm() / want_grad.norm()) <= 3e-4

    # And bit for bit the gradient of the loss composed from tensor operations.
    (grad,) = torch.autograd.grad(train._loss(img, target), img)
    composed = 0.8 * (img - target).abs().mean() + 0.2 * (1 - train.ssim(img, target))
    assert torch.equal(grad, torch.autograd.grad(composed, img)[0])


def test_loss_composes_other_inputs():
    """A differentiable target still gives the loss (and its own gradient); too small images still raise."""
    import torch

    from aniso_b200 import train

    gen = torch.Generator(device="cuda").manual_seed(5)
    img = torch.rand(24, 31, 3, device="cuda", generator=gen)
    target = torch.rand(24, 31, 3, device="cuda", generator=gen)
    want = float(train._loss(img, target))
    leaf = target.clone().requires_grad_(True)
    loss = train._loss(img, leaf)
    assert abs(float(loss) - want) <= 1e-5
    assert float(torch.autograd.grad(loss, leaf)[0].abs().sum()) > 0
    with pytest.raises(RuntimeError):
        train._loss(img[:8], target[:8])  # smaller than the window, as before
