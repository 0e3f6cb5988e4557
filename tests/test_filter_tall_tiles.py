"""The Gaussian filter's tiles of eight rows a thread (64 columns by 64 rows),
which images of two such CTAs per SM and more take: both remainders, one row or
column of tiles beside the border only, and a full square of tiles and one
pixel more.  Bit for bit against the oracle."""
import ctypes

import numpy as np
import pytest

from dice_b200 import abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [5, 7, 9, 11, 13])
@pytest.mark.parametrize("h,w", [(1090, 1170), (1216, 1216), (1217, 1217), (70, 9601), (9601, 70)])
def test_filter_of_large_images(h, w, m):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert -(-h // 64) * -(-w // 64) >= 2 * sms   # the rule of the dispatch
    img = (np.random.default_rng(h + m).random((h, w)) * 65535).astype(np.float32)
    t = torch.from_numpy(img).cuda()
    out = torch.full_like(t, float("nan"))
    p = lambda a: ctypes.c_void_p(a.data_ptr())  # noqa: E731
    assert abi.load_library().dicegpu_gauss_filter(w, h, p(t), p(out), m, None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), O.gauss_filter(img, m))
