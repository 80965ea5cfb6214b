"""The blend's 4x4-cell lists: a splat left out of a cell must be one that no pixel there can take. One
splat per view, from round ones to needles at every angle, across tile edges and image borders: every
pixel against the same splat evaluated in 64 bits from the projection the library reports."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (16, 32)])
def test_no_pixel_loses_a_splat(tile):
    import torch

    from aniso_b200 import BatchOptions, BatchRenderer, GpuRenderer, scenes

    rng = np.random.default_rng(7)
    cam = scenes.Camera(93, 71, 90.0, 90.0, 46.5, 35.5, np.eye(3), np.zeros(3))
    out = torch.empty(cam.height, cam.width, 3, dtype=torch.uint8, device="cuda")
    checked = 0
    for k in range(120):
        # Half-axes from a fraction of a pixel to the whole image, up to 300 : 1 in the image plane.
        long, ratio = 10 ** rng.uniform(-2.3, 0.0), 10 ** rng.uniform(-2.5, 0.0)
        ang = rng.uniform(0, np.pi)
        g = np.zeros((1, 11), np.float32)
        g[0, :3] = rng.uniform(-0.5, 0.5), rng.uniform(-0.4, 0.4), 1.0
        g[0, 3:6] = long, long * ratio, long * ratio
        g[0, 6:10] = np.cos(ang / 2), 0.0, 0.0, np.sin(ang / 2)
        g[0, 10] = rng.choice([0.004, 0.02, 0.3, 0.9, 0.999])
        sh = np.full((1, 3), 0.5 / 0.28209479177387814, np.float32)  # white: 0.5 + 0.5
        r = GpuRenderer(g, sh, 0)
        p = r.debug_projection(cam)
        if tile == (16, 16):
            img = r.render(cam)
        else:
            b = BatchRenderer([r], [0], BatchOptions(0, 1.0, tile, 128))
            b.render_device([cam], [out.data_ptr()])
            b.sync()
            img = out.cpu().numpy()
        if not p["tiles_touched"][0]:
            assert not img.any()
            continue
        (u, v), (A, B, C, o) = p["uv"][0].astype(np.float64), p["conic_opacity"][0].astype(np.float64)
        dx = np.arange(cam.width)[None] + 0.5 - u
        dy = np.arange(cam.height)[:, None] + 0.5 - v
        terms = 0.5 * (A * dx * dx + C * dy * dy) + np.abs(B * dx * dy)
        power = -0.5 * (A * dx * dx + C * dy * dy) - B * dx * dy
        # fp32 rounding of the exponent: a few parts in 1e7 of its terms (they cancel along a needle),
        # and the MUFU exponential's 2^-22.
        slack = 1e-6 * (1.0 + terms)
        alpha = np.minimum(0.99, o * np.exp(power))
        clear = (alpha * (1 - slack) > 1.0 / 255.0) & (power < -slack)
        # The reference's own 8x8-tile rectangle bounds the splat too; stay well inside 3 sigma's radius.
        cov = np.linalg.inv(np.array([[A, B], [B, C]]))
        radius = 3 * np.sqrt(np.linalg.eigvalsh(cov)[-1])
        clear &= (np.abs(dx) < radius - 1) & (np.abs(dy) < radius - 1)
        low = np.floor(255 * alpha * (1 - slack) + 0.5 - 1e-3)
        assert (img[..., 0][clear] >= low[clear]).all(), (k, tile)
        checked += int(clear.sum())
    assert checked > 20_000


@pytest.mark.parametrize("tile", [(16, 16), (16, 32)])
def test_adjoint_rounds_are_cut_where_their_sums_run_out_of_room(tile):
    """Splats that each touch every cell of a tile: a round of 128 of them needs four times the places
    the 16x16 and 16x32 tiles have, so rounds are cut; an 8x8 tile has room for all of its round."""
    import torch

    from aniso_b200 import scenes
    from aniso_b200.autograd import rasterize_batch

    raw = scenes.make_raw_scene(700, (-1.0, -0.8, 2.0), (1.0, 0.8, 4.0), seed=5)
    n = raw.n
    sh = np.concatenate([raw.f_dc.reshape(n, 1, 3), raw.f_rest.reshape(n, 3, 15).transpose(0, 2, 1)], 1)
    arrays = [raw.xyz, raw.scale + np.float32(3.5), raw.rot, raw.opacity - np.float32(3.0), np.ascontiguousarray(sh)]
    cam = scenes.Camera(75, 61, 70.0, 70.0, 37.5, 30.5, np.eye(3), np.zeros(3))
    up = torch.randn(cam.height, cam.width, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    got = {}
    for shape in (tile, (8, 8)):
        leaves = [torch.tensor(a, dtype=torch.float32, device="cuda", requires_grad=True) for a in arrays]
        (img,) = rasterize_batch([leaves], [cam], [0], tile=shape, use_graph=False)
        got[shape] = [img.detach()] + list(torch.autograd.grad(img, leaves, up))
    assert torch.equal(got[tile][0], got[(8, 8)][0])
    # The same terms summed per tile of another grid: fp32 sums of up to 4575 pixels, 1e-5 norm-wise.
    for a, b in zip(got[tile][1:], got[(8, 8)][1:]):
        assert float((a.double() - b.double()).norm()) <= 1e-5 * float(b.double().norm())
