"""Images of a row or a column of many pixels in the pixel and run forms: exact, and in scratch of a few
bytes a pixel, not of a whole tile for every few pixels."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 1 << 23   # one row: 2^15 or 2^16 tiles, more than 512 MiB of tile scratch in every form


@pytest.mark.parametrize("shape", [(1, N), (1, N + 5), (N, 1), (2, N), (N, 3)])
@pytest.mark.parametrize("algo,coh,conn8", [("ALGO_PIXEL", "COH_4", False), ("ALGO_RUNS", "COH_DEFAULT", False), ("ALGO_PIXEL", "COH_8", True)])
def test_thin_images(shape, algo, coh, conn8):
    import torch
    import labeling_b200 as be
    rng = np.random.default_rng(shape[0])
    img = (rng.random(shape) < 0.7).astype(np.uint8)
    img.reshape(-1)[N // 3:-100] = 1         # one run of most of it
    ref, k = O.ccl2d(img, 0, conn8)
    src = torch.from_numpy(img).cuda()
    out = torch.full(shape, -1, dtype=torch.int32, device="cuda")
    with be.Context(0) as c:
        free = torch.cuda.mem_get_info()[0]
        for count in (True, False):
            out.fill_(-1)
            n = be.label2d(c, src, out, algo=getattr(be, algo), coh=getattr(be, coh), want_count=count)
            assert not count or n == k
            assert np.array_equal(out.cpu().numpy(), ref)
        assert free - torch.cuda.mem_get_info()[0] < 40 * img.size
        lab, n, _ = be.label2d_host(c, img, algo=getattr(be, algo), coh=getattr(be, coh))
        assert n == k and np.array_equal(lab, ref)


@pytest.mark.parametrize("shape", [(1, 1, 1 << 21), (1 << 19, 1, 1), (1, 1 << 20, 2)])
def test_thin_volumes(shape):
    import torch
    import labeling_b200 as be
    vol = (np.random.default_rng(1).random(shape) < 0.5).astype(np.uint8)
    ref, k = O.ccl3d(vol)
    out = torch.full(shape, -1, dtype=torch.int32, device="cuda")
    with be.Context(0) as c:
        free = torch.cuda.mem_get_info()[0]
        assert be.label3d(c, torch.from_numpy(vol).cuda(), out, algo=be.ALGO_PIXEL) == k
        assert np.array_equal(out.cpu().numpy(), ref)
        assert free - torch.cuda.mem_get_info()[0] < (64 << 20)


@pytest.mark.parametrize("left", [430, 780])
def test_little_memory_left(left):
    """680 MB of tile scratch on a device with `left` MiB free: without the usual headroom, or iterative."""
    import torch
    import labeling_b200 as be
    img = (np.random.default_rng(left).random((8, 1 << 22)) < 0.5).astype(np.uint8)
    ref, k = O.ccl2d(img, 0, False)
    ref = torch.from_numpy(ref).cuda()
    src, out = torch.from_numpy(img).cuda(), torch.full(img.shape, -1, dtype=torch.int32, device="cuda")
    with be.Context(0) as c:
        be.label2d(c, src[:, :64], out[:, :64], algo=be.ALGO_PIXEL, coh=be.COH_4)   # kernels loaded
        torch.cuda.empty_cache()
        taken = torch.empty(torch.cuda.mem_get_info()[0] - (left << 20), dtype=torch.uint8, device="cuda")
        try:
            assert be.label2d(c, src, out, algo=be.ALGO_PIXEL, coh=be.COH_4) == k
        finally:
            del taken
            torch.cuda.empty_cache()
        assert torch.equal(out, ref)
