"""The 2D tile pipelines at the edges of their tiles and of their run and link capacities, exact
against the oracle: the block pipeline (8-connectivity, 64 x 256 pixels) and the pixel pipeline that
serves the pixel and run forms (4-connectivity, 64 x 128 pixels)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 129), (63, 31), (64, 128), (64, 256), (65, 257), (66, 127), (128, 384), (130, 513), (191, 255)]


def _images(h, w, rng):
    y, x = np.indices((h, w))
    yield "checkerboard", (x + y) % 2 == 0                       # every pixel a run, all 8-connected
    yield "columns", x % 2 == 0                                  # as many runs as a tile can have
    yield "far columns", (x % 4 == 0) | (y % 64 == 63)           # every block a run, joined at the tile's foot
    for period, shift in ((4, 2), (8, 4), (6, 3)):               # bricks: every run touches two above
        yield f"bricks {period}", ((x + shift * (y // 2)) % period != 0) | (rng.random((h, w)) < 0.01)
    yield "bottom first", np.where(y % 8 == 0, x % 16 > 9, np.where(y % 8 == 1, x % 16 < 5, (y % 8 == 3) | ((y % 8 == 2) & (x % 16 < 12))))
    yield "near the threshold", rng.random((h, w)) < 0.593
    yield "noise", rng.random((h, w)) < 0.45


@pytest.mark.parametrize("conn8", [True, False])
@pytest.mark.parametrize("size", SIZES)
def test_tile_edges_and_capacities(ctx, size, conn8):
    import torch
    import labeling_b200 as be
    rng = np.random.default_rng(size[0] * 1000 + size[1])
    for name, mask in _images(*size, rng):
        img = (mask * 255).astype(np.uint8)
        ref, k = O.ccl2d(img, 0, conn8)
        src = torch.from_numpy(img).cuda()
        for algo, coh in ((be.ALGO_UF, be.COH_8),) if conn8 else ((be.ALGO_PIXEL, be.COH_4), (be.ALGO_RUNS, be.COH_DEFAULT)):
            out = torch.full(size, -1, dtype=torch.int32, device="cuda")
            assert be.label2d(ctx, src, out, algo=algo, coh=coh) == k, (name, algo)
            assert np.array_equal(out.cpu().numpy(), ref), (name, algo)


def test_forms_of_one_context_keep_apart(ctx):
    """Calls of growing and shrinking sizes and alternating forms share a context's workspaces."""
    import torch
    import labeling_b200 as be
    rng = np.random.default_rng(5)
    for i in range(30):
        h, w = int(rng.integers(1, 500)), int(rng.integers(1, 900))
        img = ((rng.random((h, w)) < 0.5) * 255).astype(np.uint8)
        src = torch.from_numpy(img).cuda()
        for algo, coh, conn8 in ((be.ALGO_UF, be.COH_8, True), (be.ALGO_RUNS, be.COH_4, False),
                                 (be.ALGO_PIXEL, be.COH_8, True), (be.ALGO_PIXEL, be.COH_4, False)):
            out = torch.full((h, w), -1, dtype=torch.int32, device="cuda")
            k = be.label2d(ctx, src, out, algo=algo, coh=coh)
            ref, kr = O.ccl2d(img, 0, conn8)
            assert k == kr and np.array_equal(out.cpu().numpy(), ref), (i, h, w, algo, coh)


@pytest.mark.parametrize("conn8", [True, False])
@pytest.mark.parametrize("size", [(257, 1025), (400, 777)])
def test_links_across_tile_borders(ctx, size, conn8):
    """One path through every tile many times, and separate components that touch on both diagonals
    across every tile border."""
    import torch
    import labeling_b200 as be
    h, w = size
    y, x = np.indices((h, w))
    snake = (y % 2 == 0) | ((x == 0) & (y % 4 == 1)) | ((x == w - 1) & (y % 4 == 3))
    weave = np.where(y // 2 % 2 == 0, x % 4 < 2, x % 4 >= 2)
    for name, mask in (("snake", snake), ("snake back", snake[::-1, ::-1]), ("weave", weave), ("thin weave", weave & (y % 2 == 1))):
        img = (mask * 255).astype(np.uint8)
        ref, k = O.ccl2d(img, 0, conn8)
        src = torch.from_numpy(img).cuda()
        out = torch.full(size, -1, dtype=torch.int32, device="cuda")
        algo, coh = (be.ALGO_UF, be.COH_8) if conn8 else (be.ALGO_PIXEL, be.COH_4)
        assert be.label2d(ctx, src, out, algo=algo, coh=coh) == k, name
        assert np.array_equal(out.cpu().numpy(), ref), name


@pytest.mark.parametrize("tiles", [2, 37, 38, 98, 99, 148, 149])
def test_rows_of_a_tile_shared_by_ctas(ctx, tiles):
    """Numbers of tiles on both sides of the lines where fewer CTAs share a tile's rows (148 SMs)."""
    import torch
    import labeling_b200 as be
    img = ((np.random.default_rng(tiles).random((64 * tiles - 3, 45)) < 0.5) * 255).astype(np.uint8)
    src = torch.from_numpy(img).cuda()
    for algo, coh, conn8 in ((be.ALGO_UF, be.COH_8, True), (be.ALGO_PIXEL, be.COH_4, False)):
        ref, k = O.ccl2d(img, 0, conn8)
        out = torch.full(img.shape, -1, dtype=torch.int32, device="cuda")
        assert be.label2d(ctx, src, out, algo=algo, coh=coh) == k
        assert np.array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("sides", [[(128, 128), (130, 120), (1, 1)], [(64, 256), (60, 500), (3, 129)], [(65, 128), (64, 256)]])
def test_batch_tile_shape_by_tiles(ctx, sides):
    """Batches that square tiles cover with fewer, with more and with as many tiles as the default's."""
    import torch
    import labeling_b200 as be
    rng = np.random.default_rng(len(sides))
    imgs = [((rng.random(s) < 0.5) * 255).astype(np.uint8) for s in sides]
    dev = [(torch.from_numpy(i).cuda(), torch.full(i.shape, -1, dtype=torch.int32, device="cuda"), 0) for i in imgs]
    be.Batch(ctx, dev).run()
    torch.cuda.synchronize()
    for img, (_, out, _) in zip(imgs, dev):
        assert np.array_equal(out.cpu().numpy(), O.ccl2d(img, 0, True)[0])
