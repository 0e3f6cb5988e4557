"""Where a frame of square affine subsets keeps its per-pixel rows: residual rows
while they leave an SM four CTAs, lean where that fits more CTAs, the rows
again where one CTA fits either way, global scratch beyond a CTA's shared
memory."""
import pytest

from dice_b200 import abi
from dice_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _schema(subset, step, size=640):
    from dice_b200.schema import Schema
    ref = syn.speckle_image(size, size, seed=size, blur_sigma=0.8)
    deff = syn.warp_image(ref, lambda X, Y: (0.3 + 0.002 * X, -0.2 + 0.001 * Y), noise_sigma=1.0, seed=3, clip=(0.0, 255.0))
    cx, cy = syn.grid_points(size, size, subset, step)
    s = Schema(abi.default_params(subset_size=subset, enable_rotation=1, enable_normal_strain=1, enable_shear_strain=1,
                                  fast_solver_tolerance=1e-3, optimization=abi.GRADIENT_BASED))
    s.set_ref_image(ref.numpy())
    s.set_fields(syn.init_fields(cx, cy))
    s.set_def_image(deff.numpy())
    return s


# pixels, step (a 640 x 640 image then holds more than six subsets per CTA of the
# rows' grid, below which
# eight-warp CTAs take the frame), storage
@pytest.mark.parametrize("subset,step,storage", [(37, 6, abi.STORAGE_ROWS), (41, 7, abi.STORAGE_LEAN),
                                                 (61, 10, abi.STORAGE_LEAN), (81, 10, abi.STORAGE_ROWS),
                                                 (99, 5, abi.STORAGE_SCRATCH)])
def test_storage_by_subset_size(subset, step, storage):
    with _schema(subset, step) as s:
        with pytest.raises(RuntimeError):
            s.frame_launch()   # none yet
        s.execute_correlation()
        assert s.frame_launch()[:2] == (storage, 4)
