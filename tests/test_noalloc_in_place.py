"""dicegpu_image_gradients_noalloc where an output is also the input, the case
that copies the image to the library's static array: calls in a row of
different sizes, up to the array's full size, either output in place, bit for
bit against the entry with outputs of their own."""
import ctypes

import numpy as np
import pytest

from dice_b200 import abi

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("over", ["gx", "gy"])
def test_calls_in_a_row_in_place(over):
    torch = pytest.importorskip("torch")
    lib = abi.load_library()
    rng = np.random.default_rng(5)
    for h, w in [(300, 417), (1024, 1024), (37, 65), (512, 384)]:
        img = torch.from_numpy((rng.random((h, w)) * 65535).astype(np.float32)).cuda()
        want = [torch.empty_like(img), torch.empty_like(img)]
        assert lib.dicegpu_image_gradients(w, h, _ptr(img), _ptr(want[0]), _ptr(want[1]), abi.CONVOLUTION_5_POINT, None) == 0
        other = torch.empty_like(img)
        got = [img, other] if over == "gx" else [other, img]
        assert lib.dicegpu_image_gradients_noalloc(w, h, _ptr(img), _ptr(got[0]), _ptr(got[1]), abi.CONVOLUTION_5_POINT,
                                                   None) == 0
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
