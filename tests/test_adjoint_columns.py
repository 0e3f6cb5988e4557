"""The adjoint of square subsets (a column per lane, sliding windows) against the
same subsets as pixel lists (a pixel per lane): subsets of one and several
bands or chunks of columns, over the border, rotated so far that windows
often do not slide, both shapes, objectives and gradient sources.  The two
take the same float operations per pixel and differ in the order of double
sums (relative 1e-12 of the largest) and of the image derivative's float sums
(a pixel takes a few thousand terms: 1e-5 of the largest)."""
import numpy as np
import pytest

from dice_b200 import abi
from dice_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subset", [5, 9, 15, 25, 31, 33, 41, 51, 65])
@pytest.mark.parametrize("shape,objective,source", [(abi.AFFINE_SF, 0, 0), (abi.AFFINE_SF, 1, 1), (abi.QUADRATIC_SF, 0, 0)])
def test_columns_equal_lists(subset, shape, objective, source):
    torch = pytest.importorskip("torch")
    from dice_b200.schema import Schema
    size = 160
    ref = syn.speckle_image(size, size, seed=5, blur_sigma=0.8).cuda()
    deff = syn.warp_image(ref, lambda X, Y: (0.4 + 0 * X, -0.3 + 0 * Y), noise_sigma=1.0, seed=6)
    rng = np.random.default_rng(subset)
    n = 60
    cx, cy = rng.integers(0, size, n).astype(float), rng.integers(0, size, n).astype(float)
    quad = shape == abi.QUADRATIC_SF
    f = syn.init_fields(cx, cy, quadratic=quad)
    t = np.where(np.arange(n) % 3 == 0, 0.7, 0.01)
    if quad:
        f[:, abi.F_QUAD_A + 0], f[:, abi.F_QUAD_A + 1], f[:, abi.F_QUAD_A + 5] = np.cos(t), -np.sin(t), 0.3
        f[:, abi.F_QUAD_A + 6], f[:, abi.F_QUAD_A + 7], f[:, abi.F_QUAD_A + 11] = np.sin(t), np.cos(t), -0.2
        f[:, abi.F_QUAD_A + 3] = 1e-4
    else:
        f[:, abi.F_DISP_X], f[:, abi.F_DISP_Y], f[:, abi.F_ROT_Z] = 0.3, -0.2, t
        f[:, abi.F_STRETCH_XX:abi.F_SHEAR_XY + 1] = rng.normal(0, 0.01, (n, 3))
    h = subset // 2
    dy, dx = (a.ravel() for a in np.mgrid[-h:h + 1, -h:h + 1])
    rows = torch.from_numpy(f).cuda()
    seed = torch.from_numpy(rng.uniform(0.5, 1.5, n)).cuda()
    out = []
    for lists in (False, True):
        with Schema(abi.default_params(subset_size=subset, shape_function=shape, enable_rotation=1, enable_normal_strain=1,
                                       enable_shear_strain=1)) as s:
            s.set_ref_image(ref)
            s.set_fields(f)
            if lists:
                s.set_subset_pixels(np.arange(n + 1) * len(dx), (cx[:, None] + dx).ravel(), (cy[:, None] + dy).ravel())
            s.set_def_image(deff)
            d = torch.zeros_like(deff)
            value, dparams = s.adjoint(rows, seed, objective=objective, grad_source=source, ddef=d)
            torch.cuda.synchronize()
            out.append([a.double().cpu().numpy() for a in (value, dparams, d)])
    for a, b, tol in zip(out[0], out[1], (1e-12, 1e-12, 1e-5)):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
