"""First calls of a context, and first runs of a batch, on a stream of their own: scratch is cleared in that
stream's order (a clear on the default stream would not hold up a non-blocking stream)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_first_calls_on_a_side_stream():
    import torch
    import labeling_b200 as be
    img = ((np.random.default_rng(2).random((5000, 1900)) < 0.5) * 255).astype(np.uint8)
    vol = ((np.random.default_rng(3).random((40, 300, 200)) < 0.2) * 255).astype(np.uint8)
    refs = {True: O.ccl2d(img, 0, True), False: O.ccl2d(img, 0, False)}
    ref3, k3 = O.ccl3d(vol)
    src, vsrc = torch.from_numpy(img).cuda(), torch.from_numpy(vol).cuda()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for rep in range(5):
        with be.Context(0) as c:
            for algo, coh, conn8 in ((be.ALGO_UF, be.COH_8, True), (be.ALGO_RUNS, be.COH_4, False), (be.ALGO_ITER, be.COH_8, True)):
                out = torch.full(img.shape, -1, dtype=torch.int32, device="cuda")
                torch.cuda.synchronize()
                k = be.label2d(c, src, out, algo=algo, coh=coh, stream=side)
                assert k == refs[conn8][1] and np.array_equal(out.cpu().numpy(), refs[conn8][0]), (rep, algo)
            out = torch.full(vol.shape, -1, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            assert be.label3d(c, vsrc, out, stream=side) == k3 and np.array_equal(out.cpu().numpy(), ref3), rep
            outs = [torch.full(img.shape, -1, dtype=torch.int32, device="cuda") for _ in range(2)]
            torch.cuda.synchronize()
            b = be.Batch(c, [(src, o, 0) for o in outs])
            b.run(stream=side)
            side.synchronize()
            assert all(np.array_equal(o.cpu().numpy(), refs[True][0]) for o in outs), rep
            b.close()
