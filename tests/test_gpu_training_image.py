"""The training image against the oracle's 64-bit one, on scenes whose splats range from sub-pixel to
hundreds of pixels: a splat that the cell masks left out of a pixel it reaches would be off by at least
1/255 of what is left there (needs a GPU)."""
import numpy as np
import pytest

from test_gpu_block_bits import CASES, tensors

from aniso_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", sorted(CASES))
def test_training_image_matches_64_bits(case):
    import torch

    import oracle
    from aniso_b200.autograd import rasterize

    n, lo, hi, shift, (w, h, f, dist) = CASES[case]
    raw = scenes.make_raw_scene(n, lo, hi, seed=17)
    raw.scale = (raw.scale + np.float32(shift)).astype(np.float32)
    cam = scenes.front_camera(w, h, f, dist)
    params = tensors(torch, raw)
    with torch.no_grad():
        img = rasterize(*params, cam).cpu().numpy().astype(np.float64)
    want = oracle.Restatement().train_forward_f64([p.cpu().numpy() for p in params], cam)
    # Where no test falls the other way the two differ by fp32 rounding, well below 5e-4. A pixel evaluates some
    # hundreds of splats, each of which lies within the exponent's rounding (1e-6 or so) of the alpha test
    # with that probability: one pixel in a thousand is several times what that makes.
    off = np.abs(img - want).max(-1) > 5e-4
    assert off.mean() <= 1e-3, off.sum()
    assert want.max() > 0.5
