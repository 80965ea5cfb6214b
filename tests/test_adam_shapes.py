"""The fused Adam at the edges of its blocks (2048 elements, 16-byte words): odd counts, arrays that are
not 16-byte aligned, rows whose head crosses a word, against the update in 64 bits."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,offset,row,head", [(1, 0, 1, 0), (2047, 0, 48, 3), (2048, 0, 48, 3), (2049, 0, 7, 5),
                                                   (6151, 0, 3, 1), (6151, 1, 48, 3), (40_000, 3, 0, 0)])
def test_adam_matches_64_bits(count, offset, row, head):
    import torch

    from aniso_b200 import _lib
    from aniso_b200._lib import check, lib

    gen = torch.Generator(device="cuda").manual_seed(count + offset)
    p, g, m, v = (torch.randn(count + offset, device="cuda", generator=gen)[offset:] for _ in range(4))
    v.square_()
    start = [t.double() for t in (p, g, m, v)]
    lr, lr_head, eps, step = 1e-2, 3e-2, 1e-8, 7
    group = _lib.AdamGroup(p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), count, lr, lr_head, row, head, eps)
    empty = _lib.AdamGroup(None, None, None, None, 0, lr, lr, 0, 0, eps)
    check(lib.aniso_b200_adam_step((_lib.AdamGroup * 3)(empty, group, empty), 3, step, 0.9, 0.999,
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    p0, g0, m0, v0 = start
    rate = torch.full_like(p0, lr)
    if head:
        rate[torch.arange(count, device="cuda") % row < head] = lr_head
    m1 = 0.9 * m0 + 0.1 * g0
    v1 = 0.999 * v0 + 0.001 * g0 * g0
    p1 = p0 - rate / (1 - 0.9 ** step) * m1 / ((v1 / (1 - 0.999 ** step)).sqrt() + eps)
    # beta1 and beta2 are floats (1 - 0.9f is 2.4e-8 off 0.1, 1 - 0.999f 1.3e-8 off 0.001), then a few roundings.
    torch.testing.assert_close(m.double(), m1, rtol=2e-6, atol=1e-6)
    torch.testing.assert_close(v.double(), v1, rtol=2e-5, atol=1e-9)
    torch.testing.assert_close(p.double(), p1, rtol=2e-5, atol=2e-6)
