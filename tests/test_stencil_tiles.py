"""The filter and gradient kernels at the edges of their tiles (64 columns by 16
or 64 rows; 32 by 32): sizes below one tile, one tile and one pixel either
side of it, and tiles that lie inside the image.  Bit for bit against the
oracle, and in place for the smoothing (its input is also its output)."""
import ctypes

import numpy as np
import pytest

from dice_b200 import abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(3, 3), (4, 5), (13, 13), (31, 33), (36, 40), (41, 72), (63, 65), (64, 64), (70, 103), (129, 130), (600, 1300)]


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _image(h, w):
    return (np.random.default_rng(h * w).random((h, w)) * 65535).astype(np.float32)


@pytest.mark.parametrize("h,w", SIZES)
def test_gradients_at_tile_edges(h, w):
    torch = pytest.importorskip("torch")
    lib, img = abi.load_library(), _image(h, w)
    t = torch.from_numpy(img).cuda()
    for method in (abi.FINITE_DIFFERENCE, abi.CONVOLUTION_5_POINT):
        gx, gy = torch.full_like(t, float("nan")), torch.full_like(t, float("nan"))
        assert lib.dicegpu_image_gradients(w, h, _ptr(t), _ptr(gx), _ptr(gy), method, None) == 0
        torch.cuda.synchronize()
        ox, oy = O.gradients(img, method)
        assert np.array_equal(gx.cpu().numpy(), ox) and np.array_equal(gy.cpu().numpy(), oy)


@pytest.mark.parametrize("m", [5, 7, 9, 11, 13])
@pytest.mark.parametrize("h,w", SIZES)
def test_filter_at_tile_edges(h, w, m):
    torch = pytest.importorskip("torch")
    lib, img = abi.load_library(), _image(h, w)
    t = torch.from_numpy(img).cuda()
    out = torch.full_like(t, float("nan"))
    rc = lib.dicegpu_gauss_filter(w, h, _ptr(t), _ptr(out), m, None)
    assert rc == (0 if min(h, w) >= m else abi.ERR_ARG)
    torch.cuda.synchronize()
    if rc == 0:
        assert np.array_equal(out.cpu().numpy(), O.gauss_filter(img, m))


@pytest.mark.parametrize("entry", ["dicegpu_image_gradients", "dicegpu_image_gradients_noalloc"])
def test_smoothing_over_its_input(entry):
    torch = pytest.importorskip("torch")
    lib, img = abi.load_library(), _image(90, 140)
    t = torch.from_numpy(img).cuda()
    gy = torch.empty_like(t)
    assert getattr(lib, entry)(140, 90, _ptr(t), _ptr(t), _ptr(gy), abi.CONVOLUTION_5_POINT, None) == 0
    torch.cuda.synchronize()
    ox, oy = O.gradients(img, abi.CONVOLUTION_5_POINT)
    assert np.array_equal(t.cpu().numpy(), ox) and np.array_equal(gy.cpu().numpy(), oy)
