"""Launches of several scan chunks (more than 4096 segments) that follow launches of other sizes and forms
in one context: what those left in the workspace must not be taken for the scan's status words.  A first
image with nine components leaves prefixes of 9 where the next, smaller one's status words would lie if
they moved with the size -- a published sum of 9 to the second launch of a context."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _image(shape, seed, p=0.5):
    return ((np.random.default_rng(seed).random(shape) < p) * 255).astype(np.uint8)


@pytest.mark.parametrize("algo,second", [("ALGO_RUNS", (1992, 1936)), ("ALGO_PIXEL", (1992, 1936)), ("ALGO_UF", (1992, 1808))])
def test_second_launch_over_prefixes_of_the_first(algo, second):
    import torch
    import labeling_b200 as be
    algo, conn8 = getattr(be, algo), algo == "ALGO_UF"
    sparse = np.zeros((2048, 2048), np.uint8)
    sparse[3, 10:100:10] = 255
    noise = _image(second, 1)
    ref, k = O.ccl2d(noise, 0, conn8)
    ref = torch.from_numpy(ref).cuda()
    a, b = torch.from_numpy(sparse).cuda(), torch.from_numpy(noise).cuda()
    out_a, out_b = torch.empty(a.shape, dtype=torch.int32, device="cuda"), torch.empty(b.shape, dtype=torch.int32, device="cuda")
    for rep in range(20):
        with be.Context(0) as c:
            assert be.label2d(c, a, out_a, algo=algo) == 9
            out_b.fill_(-1)
            assert be.label2d(c, b, out_b, algo=algo) == k, rep
            assert torch.equal(out_b, ref), rep


def test_alternating_sizes_and_forms_of_many_chunks():
    import torch
    import labeling_b200 as be
    sizes = [(2048, 2048), (1992, 1936), (4099, 300), (1500, 1100), (9000, 257), (1021, 1787)]
    cases = []
    for i, s in enumerate(sizes):
        img = _image(s, i, 0.02 if i % 2 else 0.5)
        for algo, coh, conn8 in ((be.ALGO_UF, be.COH_8, True), (be.ALGO_RUNS, be.COH_4, False), (be.ALGO_PIXEL, be.COH_8, True)):
            ref, k = O.ccl2d(img, 0, conn8)
            cases.append((torch.from_numpy(img).cuda(), algo, coh, torch.from_numpy(ref).cuda(), k))
    vol = _image((33, 200, 130), 9, 0.2)
    ref, k = O.ccl3d(vol, 0)
    vols = [(torch.from_numpy(vol).cuda(), algo, torch.from_numpy(ref).cuda(), k) for algo in (be.ALGO_UF, be.ALGO_PIXEL)]
    rng = np.random.default_rng(0)
    with be.Context(0) as c:
        for rep in range(150):
            img, algo, coh, ref, k = cases[int(rng.integers(len(cases)))]
            out = torch.full(img.shape, -1, dtype=torch.int32, device="cuda")
            assert be.label2d(c, img, out, algo=algo, coh=coh) == k, (rep, tuple(img.shape), algo)
            assert torch.equal(out, ref), (rep, tuple(img.shape), algo)
            if rep % 5 == 0:
                img, algo, ref, k = vols[rep // 5 % 2]
                out = torch.full(img.shape, -1, dtype=torch.int32, device="cuda")
                assert be.label3d(c, img, out, algo=algo) == k and torch.equal(out, ref), rep
