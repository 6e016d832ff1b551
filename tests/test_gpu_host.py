"""Host-memory calls: rows with and without gaps on either side, aligned and odd widths."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _image(shape, seed):
    return (np.random.default_rng(seed).random(shape) < 0.45).astype(np.uint8)


@pytest.fixture(scope="module")
def ctx():
    import labeling_b200 as be
    c = be.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (64, 257), (65, 1023), (1021, 1787)])
@pytest.mark.parametrize("algo", ["ALGO_AUTO", "ALGO_ITER"])
def test_contiguous(ctx, shape, algo):
    import labeling_b200 as be
    img = _image(shape, shape[1])
    ref, k = O.ccl2d(img)
    lab, n, us = be.label2d_host(ctx, img, algo=getattr(be, algo))
    assert n == k and us > 0 and np.array_equal(lab, ref)


@pytest.mark.parametrize("pad_in,pad_out", [(0, 5), (3, 0), (16, 8)])
def test_pitched_host_rows(ctx, pad_in, pad_out):
    import labeling_b200 as be
    rows, cols = 611, 1291
    img = _image((rows, cols), 9)
    ref, k = O.ccl2d(img)
    src = np.full((rows, cols + pad_in), 255, np.uint8)
    src[:, :cols] = img
    out = np.full((rows, cols + pad_out), -7, np.int32)
    n, us = ctypes.c_int64(0), ctypes.c_double(0)
    ctx.check(be.lib().be_label2d_host(ctx.handle, src.ctypes.data, cols + pad_in, rows, cols, 0, be.COH_DEFAULT, be.ALGO_AUTO,
                                       out.ctypes.data, cols + pad_out, ctypes.byref(n), ctypes.byref(us)))
    assert n.value == k and np.array_equal(out[:, :cols], ref) and (out[:, cols:] == -7).all()
