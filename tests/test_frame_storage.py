"""Where a frame of square affine subsets keeps its per-pixel rows: residual rows
while they leave an SM four CTAs, lean where that fits more CTAs, the rows
again where one CTA fits either way, global scratch beyond a CTA's shared
memory."""
import numpy as np
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


def test_storage_does_not_depend_on_who_set_the_launch_shape():
    """61 px: one CTA per SM with rows, three of four warps lean."""
    with _schema(61, 10) as s:
        f = s.fields()
        s.execute_correlation()
        want = s.fields()
        assert s.frame_launch()[:2] == (abi.STORAGE_LEAN, 4)
        ctas = s.frame_launch()[2]
        for shape, storage, grid in [((4, 0), abi.STORAGE_LEAN, ctas), ((4, 1), abi.STORAGE_ROWS, ctas // 3),
                                     ((4, 2), abi.STORAGE_LEAN, ctas // 3 * 2), ((8, 0), abi.STORAGE_LEAN, None),
                                     ((2, 0), abi.STORAGE_LEAN, None), ((1, 0), abi.STORAGE_LEAN, None)]:
            # a context of its own: 0 CTAs per SM keeps an earlier value
            with _schema(61, 10) as t:
                t.set_launch_shape(*shape)
                t.execute_correlation()
                assert t.frame_launch()[:2] == (storage, shape[0])
                assert grid is None or t.frame_launch()[2] == grid
                got = t.fields()
            if shape[0] == 4:
                assert np.array_equal(got, want)   # the same warps: the same sums
            else:
                # a shape may move a double sum's last bit, and a float of the
                # parameters (below 16) with it, before the last iterations
                ok = want[:, abi.F_SIGMA] >= 0
                assert ok.mean() > 0.9
                uv = slice(abi.F_DISP_X, abi.F_DISP_Y + 1)
                assert np.abs(got[ok, uv] - want[ok, uv]).max() < 1e-4
        s.load_fields(f)
        s.autotune()
        s.load_fields(f)
        s.execute_correlation()
        assert s.frame_launch()[0] == abi.STORAGE_LEAN
    with _schema(61, 10) as s:   # the tuner's cache
        s.autotune()
        s.execute_correlation()
        assert s.frame_launch()[0] == abi.STORAGE_LEAN


def test_lean_frames_in_a_captured_sequence():
    torch = pytest.importorskip("torch")
    with _schema(61, 10) as s:
        f = s.fields()
        s.execute_correlation()
        want = s.fields()
    frame = syn.warp_image(syn.speckle_image(640, 640, seed=640, blur_sigma=0.8),
                           lambda X, Y: (0.3 + 0.002 * X, -0.2 + 0.001 * Y), noise_sigma=1.0, seed=3, clip=(0.0, 255.0)).cuda()
    with _schema(61, 10) as g:
        g.set_stream(torch.cuda.Stream())
        reset = torch.from_numpy(f).cuda()
        torch.cuda.synchronize()
        g.capture_sequence([frame], reset_fields=reset)
        assert g.frame_launch()[:2] == (abi.STORAGE_LEAN, 4)
        for _ in range(2):
            g.launch_sequence()
            assert np.array_equal(g.fields(), want)
