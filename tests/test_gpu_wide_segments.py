"""Rows that hold as many components as a tile's segment can: every second pixel of a row a component of
its own, 256 in a tile of 512 pixels' width.  Every 2D tile shape is taken through a loaded tuning table,
and batches are tuned on such images; labels and counts are exact."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _images():
    for h, w in ((1, 512), (5, 511), (33, 513), (64, 1024), (70, 1537)):
        y, x = np.indices((h, w))
        yield (x % 2 == 0) & (y % 2 == 0)                          # dots: every one a component
        yield (x % 2 == 0) & (y % 64 < 63)                         # stripes that go on below a tile's foot
        yield (x % 2 == 0) | (y == h - 1)                          # joined only at the image's foot
        yield ((x % 2 == 0) & (y % 2 == 0)) | ((x < w // 2) & (y % 32 == 31) & (x % 2 == 0))


def _table_class(h, w):
    return (2 << 16) | ((h.bit_length() - 1) << 8) | (w.bit_length() - 1)


@pytest.mark.parametrize("shape", [0, 1, 2])
def test_every_tile_shape_by_a_loaded_table(tmp_path, shape):
    import torch
    import labeling_b200 as be
    images = [(m * 255).astype(np.uint8) for m in _images()]
    path = tmp_path / "table.txt"
    path.write_text("".join(f"{c} {be.ALGO_UF} {shape} 1.0\n" for c in sorted({_table_class(*i.shape) for i in images})))
    with be.Context(0) as c:
        c.tune_load(str(path))
        for img in images:
            ref, k = O.ccl2d(img)
            out = torch.full(img.shape, -1, dtype=torch.int32, device="cuda")
            assert be.label2d(c, torch.from_numpy(img).cuda(), out) == k, img.shape
            assert np.array_equal(out.cpu().numpy(), ref), img.shape


def test_autotune_and_tuned_batch(ctx):
    import torch
    import labeling_b200 as be
    images = [(m * 255).astype(np.uint8) for m in _images()]
    dev = [(torch.from_numpy(i).cuda(), torch.full(i.shape, -1, dtype=torch.int32, device="cuda"), 0) for i in images]
    with be.Context(0) as c:
        for x, y, _ in dev:
            be.autotune2d(c, x, y)      # every candidate must agree
    b = be.Batch(ctx, dev)
    b.tune()
    for _, y, _ in dev:
        y.fill_(-1)
    b.run()
    refs = [O.ccl2d(i) for i in images]
    assert b.counts() == [k for _, k in refs]
    for (_, y, _), (ref, _) in zip(dev, refs):
        assert np.array_equal(y.cpu().numpy(), ref)
    b.close()
