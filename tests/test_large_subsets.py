"""Frames of large affine subsets, stored lean (the residuals formed again in the
sweeps): sizes on either side of where the rows would leave an SM two, one or
no CTA in shared memory, every interpolant, pixel lists, reference gradients,
and subsets that reach over the image's border.  Bit for bit against the
oracle."""
import numpy as np
import pytest

from dice_b200 import abi
from dice_b200 import synthetic as syn
from oracle import oracle as O
from tests._exact import assert_rows_equal

pytestmark = pytest.mark.gpu


def _pair(size):
    ref = syn.speckle_image(size, size, seed=size, blur_sigma=0.8)
    deff = syn.warp_image(ref, lambda X, Y: (0.3 + 0.002 * X, -0.2 + 0.001 * Y), noise_sigma=1.0, seed=3, clip=(0.0, 255.0))
    return ref.numpy(), deff.numpy()


@pytest.mark.parametrize("subset,size,step,interp,defgrad,lists",
                         [(37, 420, 6, abi.KEYS_FOURTH, 1, False), (61, 420, 10, abi.KEYS_FOURTH, 1, False),
                          (61, 420, 7, abi.BICUBIC, 1, True), (61, 420, 10, abi.BILINEAR, 0, False),
                          (65, 420, 9, abi.KEYS_FOURTH, 0, True), (99, 330, 2, abi.KEYS_FOURTH, 1, False)])
def test_large_subsets_equal_oracle(subset, size, step, interp, defgrad, lists):
    from dice_b200.schema import Schema
    ref, deff = _pair(size)
    cx, cy = syn.grid_points(size, size, subset, step)
    cx[:4], cy[:4] = [subset // 2, 3, size - 4, size // 2], [subset // 2, size // 2, 5, size - 2]   # over the border
    p = abi.default_params(subset_size=subset, enable_rotation=1, enable_normal_strain=1, enable_shear_strain=1,
                           fast_solver_tolerance=1e-3, interpolation=interp, use_def_gradients=defgrad,
                           optimization=abi.GRADIENT_BASED)
    f = syn.init_fields(cx, cy)
    kw = {}
    if lists:
        h = subset // 2
        dy, dx = np.mgrid[-h:h + 1, -h:h + 1]
        keep = (dx * dx + dy * dy <= h * h + h)
        dx, dy = dx[keep], dy[keep]
        px = (cx[:, None] + dx[None]).astype(np.int32).ravel()
        py = (cy[:, None] + dy[None]).astype(np.int32).ravel()
        kw = dict(offsets=(np.arange(len(cx) + 1) * len(dx)).astype(np.int32), px=px, py=py)
    with Schema(p) as s:
        s.set_ref_image(ref)
        s.set_fields(f)
        if lists:
            s.set_subset_pixels(kw["offsets"], kw["px"], kw["py"])
        s.set_def_image(deff)
        s.execute_correlation()
        got = s.fields()
    want = f.copy()
    O.execute_frame(p, ref, deff, want, first_frame=True, nthreads=8, **kw)
    assert_rows_equal(got, want)
