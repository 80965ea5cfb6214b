"""Frames of few entries per tile take blends of their own (short rounds without lists, empty tiles
left at once). The same splats beside 60000 culled ones make the frame an ordinary one: images and
gradients keep their bits (needs a GPU)."""
import numpy as np
import pytest

from aniso_b200 import scenes

pytestmark = pytest.mark.gpu

# Splats per tile around a short round's end (32), the rounds' and the adjoint's (32, 64, 128), and none.
SIZES = [0, 1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 0, 257, 300, 0, 3, 7]


@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (16, 32)])
@pytest.mark.parametrize("log_scale", [-7.0, -4.5, -1.5])
def test_sparse_frames_keep_every_bit(tile, log_scale):
    import torch

    from aniso_b200 import BatchOptions, BatchRenderer, GpuRenderer
    from aniso_b200.autograd import rasterize_batch

    rng = np.random.default_rng(12)
    n, company = 9000, 60_000  # 615 or 1230 tiles: at most 15 entries a tile, and at least 56 with the company
    w, h = (643, 478) if tile != (8, 8) else (323, 237)
    cam = scenes.Camera(w, h, 500.0, 500.0, w / 2, h / 2, np.eye(3), np.zeros(3))
    xyz = np.tile(np.float32([0, 0, -5]), (n, 1))
    at = rng.permutation(n)[: sum(SIZES)]
    where = np.repeat(np.arange(len(SIZES)), SIZES)
    px = tile[0] * (where + 2) + rng.uniform(1, tile[0] - 1, at.size)
    py = tile[1] * 3 + rng.uniform(1, tile[1] - 1, at.size)
    z = rng.uniform(2.0, 9.0, at.size)
    xyz[at] = np.stack([(px - cam.cx) / cam.fx * z, (py - cam.cy) / cam.fy * z, z], 1)
    arrs = [xyz, np.full((n, 3), log_scale) + rng.normal(0, 0.3, (n, 3)), rng.normal(0, 1, (n, 4)), rng.normal(-1.5, 1, n),
            rng.normal(0, 0.2, (n, 16, 3))]
    raw = [torch.tensor(a, dtype=torch.float32, device="cuda") for a in arrs]
    behind = [t[:1].expand(company, *t.shape[1:]).clone() for t in raw]
    behind[0][:] = torch.tensor([0.0, 0.0, -5.0])
    up = torch.randn(h, w, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    got = []
    for parts in (raw, [torch.cat(p) for p in zip(raw, behind)]):
        leaves = [t.clone().requires_grad_(True) for t in parts]
        (img,) = rasterize_batch([leaves], [cam], [0], tile=tile, use_graph=False)
        grads = torch.autograd.grad(img, leaves, up)
        act = torch.cat([parts[0], parts[1].exp(), torch.nn.functional.normalize(parts[2], dim=-1),
                         parts[3].sigmoid()[:, None]], 1).cpu().numpy()
        r = GpuRenderer(act, parts[4].reshape(len(act), -1).cpu().numpy(), 3)
        b = BatchRenderer([r], [0], BatchOptions(3, 1.0, tile, 256))
        out = torch.full((h, w, 3), 77, dtype=torch.uint8, device="cuda")
        b.render_device([cam], [out.data_ptr()])
        b.sync()
        got.append([img.detach(), out] + [g[:n] for g in grads])
    assert got[0][0].abs().sum() > 0 and got[0][1].any()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
