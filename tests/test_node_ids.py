"""Node ids (tile * nodes per tile + node) are 32 bits: launches of more tiles are refused, where ids that
wrapped would have joined components of far-apart tiles."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launches_of_too_many_tiles_are_refused(tmp_path):
    import labeling_b200 as be
    from labeling_b200 import build
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    be.lib()
    exe = str(tmp_path / "node_ids")
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-I" + os.path.join(ROOT, "include"), "-I" + build.CSRC,
                    os.path.join(ROOT, "tests", "native", "node_ids.cu"), "-o", exe, be.LIB_PATH,
                    "-Xlinker", "-rpath," + os.path.dirname(be.LIB_PATH)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
