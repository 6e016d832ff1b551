"""The scan's status words keep their place: launches of any two sizes and geometries that share a
context's workspace have one head (launch epoch, error flags, status words), and no other array of
either lies over it.  A word of another array that happens to carry the launch's epoch would be taken
for a chunk's published sum."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launches_of_one_allocation_share_its_head(tmp_path):
    import labeling_b200 as be
    from labeling_b200 import build
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    be.lib()
    exe = str(tmp_path / "workspace_layout")
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-I" + os.path.join(ROOT, "include"), "-I" + build.CSRC,
                    os.path.join(ROOT, "tests", "native", "workspace_layout.cu"), "-o", exe, be.LIB_PATH,
                    "-Xlinker", "-rpath," + os.path.dirname(be.LIB_PATH)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
