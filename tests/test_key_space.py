"""Sides above 2^30 have a key-space shift (31), so that calls outside the key space are refused: a shift
counted in 32 bits never reached them and the call did not return."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shift_of_every_side(tmp_path):
    from labeling_b200 import build
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "key_space")
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-I" + os.path.join(ROOT, "include"), "-I" + build.CSRC,
                    os.path.join(ROOT, "tests", "native", "key_space.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_calls_outside_the_key_space_are_refused():
    import torch
    import labeling_b200 as be
    x = torch.zeros(64, dtype=torch.uint8, device="cuda")
    y = torch.zeros(64, dtype=torch.int32, device="cuda")
    cols = (1 << 30) + 1
    with be.Context(0) as c:
        for algo in (be.ALGO_PIXEL, be.ALGO_RUNS, be.ALGO_ITER):   # refused before anything is read
            rc = be.lib().be_label2d(c.handle, x.data_ptr(), cols, 1, cols, 0, be.COH_DEFAULT, algo, y.data_ptr(), cols, None, None)
            assert be.STATUS[rc] == "BE_ERR_INVALID", algo
