"""The training loss takes its kernels for the images they are written for, (H, W, 3) of 11 to 32767
pixels a side; every other image goes to the composed expression, or raises as that does."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(24, 31), (24, 31, 1), (24, 31, 2), (24, 31, 4), (24, 31, 3, 1), (1, 24, 31, 3)])
def test_images_without_three_channels_raise(shape):
    import torch

    from aniso_b200 import train

    img = torch.rand(shape, device="cuda")
    with pytest.raises(RuntimeError):
        train._loss(img, torch.rand(shape, device="cuda"))


def test_images_beyond_the_kernels_sizes_are_composed():
    import torch

    from aniso_b200 import train

    img, target = (torch.rand(11, 32768, 3, device="cuda") for _ in range(2))
    want = 0.8 * (img - target).abs().mean() + 0.2 * (1 - train.ssim(img, target))
    assert torch.equal(train._loss(img, target), want)
