"""Rows of every alignment: the tile kernels read an image in 16-byte chunks whatever its address and
row length, and write label rows the same way.  Widths around the chunk and tile edges, every byte
offset of the input and element offset of the output; exact, and nothing outside the label rows is
written."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _views(h, w, pad, in_off, out_off):
    import torch
    src = torch.randint(0, 256, (in_off + (h - 1) * (w + pad) + w,), dtype=torch.uint8, device="cuda")
    dst = torch.full((out_off + (h - 1) * (w + pad) + w + 8,), -7, dtype=torch.int32, device="cuda")
    return (torch.as_strided(src, (h, w), (w + pad, 1), in_off),
            torch.as_strided(dst, (h, w), (w + pad, 1), out_off), dst)


@pytest.mark.parametrize("w", [1, 3, 15, 16, 17, 63, 64, 65, 79, 81, 255, 256, 257, 319, 513])
def test_2d_rows_of_every_alignment(ctx, w):
    import torch
    import labeling_b200 as be
    rng = np.random.default_rng(w)
    h = 67
    for in_off in range(16):
        pad, out_off, thr = int(rng.integers(0, 18)), in_off % 4, (0, 100, 200)[in_off % 3]
        img = rng.integers(0, 256, (h, w)).astype(np.uint8)
        ref, k = O.ccl2d(img, thr)
        src, dst, whole = _views(h, w, pad, in_off, out_off)
        src.copy_(torch.from_numpy(img).cuda())
        assert be.label2d(ctx, src, dst, threshold=thr, algo=be.ALGO_UF) == k, (in_off, pad)
        assert np.array_equal(dst.cpu().numpy(), ref), (in_off, pad)
        dst.fill_(-7)
        assert bool((whole == -7).all()), (in_off, pad)


@pytest.mark.parametrize("d2", [1, 2, 15, 17, 63, 64, 65, 68, 80, 127])
def test_3d_rows_of_every_alignment(ctx, d2):
    import torch
    import labeling_b200 as be
    rng = np.random.default_rng(d2)
    shape = (18, 33, d2)
    n = int(np.prod(shape))
    for off in range(16):
        vol = ((rng.random(shape) < 0.2) * rng.integers(1, 256, shape)).astype(np.uint8)
        ref, k = O.ccl3d(vol, 0)
        src = torch.zeros(off + n, dtype=torch.uint8, device="cuda")
        src[off:] = torch.from_numpy(vol.reshape(-1)).cuda()
        dst = torch.full((off % 4 + n + 8,), -7, dtype=torch.int32, device="cuda")
        out = dst[off % 4:off % 4 + n].view(shape)
        assert be.label3d(ctx, src[off:].view(shape), out) == k, off
        assert np.array_equal(out.cpu().numpy(), ref), off
        out.fill_(-7)
        assert bool((dst == -7).all()), off
