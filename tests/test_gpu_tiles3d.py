"""The 3D tile pipeline at the edges of its tiles (16 x 32 x 64 voxels) and of its run and link
capacities, exact against the oracle: links that cross one, two and three tile faces at once, volumes
whose every block is a run, and more links than a tile's union queue holds."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (15, 31, 63), (16, 32, 64), (17, 33, 65), (33, 34, 130), (2, 97, 129), (48, 3, 67), (18, 66, 2)]


def _volumes(shape, rng):
    x, y, z = np.indices(shape)
    yield "corners", (x % 16 >= 14) & (y % 32 >= 30) & (z % 64 >= 62) | (x % 16 == 0) & (y % 32 == 0) & (z % 64 == 0)
    yield "anti-corners", ((x % 16 == 15) & (y % 32 == 0) & (z % 64 == 63)) | ((x % 16 == 0) & (y % 32 == 31) & (z % 64 == 0))
    yield "sheets along d2", (z % 2 == 0) & (rng.random(shape) < 0.95)
    yield "points", (x % 2 == 0) & (y % 2 == 0) & (z % 2 == 0)
    yield "columns of blocks", (z % 4 == 1) & ((x + y) % 3 != 0)
    yield "late first voxel", np.where(x % 2 == 0, (y % 4 == 3) & (z % 5 < 3), (y % 4 < 2) | (z % 7 == 0))
    for p in (0.03, 0.1, 0.2, 0.3, 0.5):
        yield f"noise {p}", rng.random(shape) < p


@pytest.mark.parametrize("shape", SIZES)
def test_tile_edges_and_capacities_3d(ctx, shape):
    import torch
    import labeling_b200 as be
    rng = np.random.default_rng(sum(shape))
    for name, mask in _volumes(shape, rng):
        vol = (mask * 255).astype(np.uint8)
        ref, k = O.ccl3d(vol, 0)
        src = torch.from_numpy(vol).cuda()
        for algo in (be.ALGO_UF, be.ALGO_PIXEL):
            out = torch.full(shape, -1, dtype=torch.int32, device="cuda")
            assert be.label3d(ctx, src, out, algo=algo) == k, (name, algo)
            assert np.array_equal(out.cpu().numpy(), ref), (name, algo)
        # batched (persistent CTAs) beside a second volume
        outs = [torch.full(shape, -1, dtype=torch.int32, device="cuda") for _ in range(2)]
        b = be.Batch(ctx, [(src, outs[0]), (src, outs[1])])
        b.run()
        assert b.counts() == [k, k], name
        assert all(np.array_equal(o.cpu().numpy(), ref) for o in outs), name
        b.close()


@pytest.mark.parametrize("tiles", [1, 2, 74, 75, 197, 198, 296, 297])
def test_rows_of_a_tile_shared_by_ctas(ctx, tiles):
    """Numbers of tiles on both sides of the lines where fewer CTAs share a tile's rows (148 SMs)."""
    import torch
    import labeling_b200 as be
    vol = (np.random.default_rng(tiles).random((16 * tiles - 5, 31, 13)) < 0.25).astype(np.uint8)
    ref, k = O.ccl3d(vol)
    out = torch.full(vol.shape, -1, dtype=torch.int32, device="cuda")
    assert be.label3d(ctx, torch.from_numpy(vol).cuda(), out) == k
    assert np.array_equal(out.cpu().numpy(), ref)
