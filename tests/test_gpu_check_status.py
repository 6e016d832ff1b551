"""The report of failed index checks: of whichever union-find form ran last, and the bounds-checked build
run on the pixel and run forms and on every 2D tile shape (images that end inside tiles, hold as many
runs as a tile can, and link across every tile border), with labels exact and no check failed."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import json, sys
sys.path.insert(0, ROOT)
import numpy as np, torch
import labeling_b200 as be
from labeling_b200 import workloads as W
from oracle import oracle as O
bad = []
def images():
    yield "noise", W.bernoulli((700, 1031), 0.5, seed=3)
    yield "sparse", W.bernoulli((513, 777), 0.08, seed=4)
    yield "spiral", W.spiral(600, 900)
    y, x = np.indices((300, 1100))
    yield "checkerboard", (((x + y) % 2 == 0) * 255).astype(np.uint8)
    yield "stripes", ((x % 2 == 0) * 255).astype(np.uint8)
    yield "dots", (((x % 2 == 0) & (y % 2 == 0)) * 255).astype(np.uint8)
    yield "one tile", W.bernoulli((60, 100), 0.4, seed=5)
for shape in (0, 1, 2):
    ctx = be.Context(0)
    open(TABLE, "w").write("".join(f"{(2 << 16) | (a << 8) | b} {be.ALGO_UF} {shape} 1.0\n" for a in range(12) for b in range(12)))
    ctx.tune_load(TABLE)
    forms = [(be.ALGO_AUTO, be.COH_8, True)]
    if shape == 0:
        forms += [(be.ALGO_PIXEL, be.COH_4, False), (be.ALGO_RUNS, be.COH_4, False), (be.ALGO_PIXEL, be.COH_8, True)]
    for name, img in images():
        src = torch.from_numpy(img).cuda()
        for algo, coh, conn8 in forms:
            out = torch.full(img.shape, -1, dtype=torch.int32, device="cuda")
            n = be.label2d(ctx, src, out, algo=algo, coh=coh)
            site, val = ctx.check_status(2)
            ref, k = O.ccl2d(img, 0, conn8)
            if site or n != k or not np.array_equal(out.cpu().numpy(), ref):
                bad.append((name, shape, algo, site, val, n, k))
    vol = W.bernoulli((40, 70, 130), 0.25, seed=6)
    out = torch.full(vol.shape, -1, dtype=torch.int32, device="cuda")
    n = be.label3d(ctx, torch.from_numpy(vol).cuda(), out, algo=be.ALGO_PIXEL)
    site, val = ctx.check_status(3)
    ref, k = O.ccl3d(vol)
    if site or n != k or not np.array_equal(out.cpu().numpy(), ref):
        bad.append(("volume", site, val, n, k))
    ctx.close()
print("RESULT", json.dumps(bad))
"""


def test_checked_build_on_every_form_and_shape(tmp_path):
    from labeling_b200 import build
    if not os.path.exists(build.LIB_CHECK):
        build.build(checked=True)
    code = CHILD.replace("ROOT", repr(ROOT)).replace("TABLE", repr(str(tmp_path / "table.txt")))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, BE_B200_LIB=build.LIB_CHECK), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    line = [l for l in r.stdout.splitlines() if l.startswith("RESULT ")]
    assert line, r.stdout[-2000:] + r.stderr[-2000:]
    assert json.loads(line[0][7:]) == []


def test_status_is_of_the_last_form(tmp_path):
    import labeling_b200 as be
    from labeling_b200 import build
    exe = str(tmp_path / "check_status")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I" + os.path.join(ROOT, "include"), "-I" + build.CSRC,
                    os.path.join(ROOT, "tests", "native", "check_status.cu"), "-o", exe, be.LIB_PATH,
                    "-Xlinker", "-rpath," + os.path.dirname(be.LIB_PATH)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
