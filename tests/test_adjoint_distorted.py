"""The adjoint's two launches for square subsets: columns for those near a
translation, pixels for those whose displacement gradients add up to more.  A
field of both kinds and of sums on either side of the limit (0.34), a row of
NaN, and more subsets than the second launch looks at in one round, against
the same subsets as pixel lists.  Tolerances as in test_adjoint_columns: the
order of double sums (1e-12 of the largest) and of the image derivative's
float sums, whose largest pixel takes `terms` of them in turn: their rounding
adds up to terms / 2 units of 2^-24 at most, a random walk of sqrt(terms) in
earnest, with a factor of four to spare."""
import numpy as np
import pytest

from dice_b200 import abi
from dice_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,subset,shape", [(300, 25, abi.AFFINE_SF), (300, 15, abi.QUADRATIC_SF), (90001, 9, abi.AFFINE_SF)])
def test_both_launches_equal_lists(n, subset, shape):
    torch = pytest.importorskip("torch")
    from dice_b200.schema import Schema
    size, h = 420, subset // 2
    ref = syn.speckle_image(size, size, seed=5, blur_sigma=0.8).cuda()
    deff = syn.warp_image(ref, lambda X, Y: (0.4 + 0 * X, -0.3 + 0 * Y), noise_sigma=1.0, seed=6)
    rng = np.random.default_rng(n)
    cx, cy = rng.integers(0, size, n).astype(float), rng.integers(0, size, n).astype(float)
    quad = shape == abi.QUADRATIC_SF
    f = syn.init_fields(cx, cy, quadratic=quad)
    t = np.array([0.0, 0.05, 0.1699, 0.1701, 0.4, 1.57, -0.9])[rng.integers(0, 7, n)]   # twice the rotation against 0.34
    if quad:
        f[:, abi.F_QUAD_A + 0], f[:, abi.F_QUAD_A + 1], f[:, abi.F_QUAD_A + 5] = np.cos(t), -np.sin(t), 0.3
        f[:, abi.F_QUAD_A + 6], f[:, abi.F_QUAD_A + 7], f[:, abi.F_QUAD_A + 11] = np.sin(t), np.cos(t), -0.2
        f[7, abi.F_QUAD_A] = np.nan
    else:
        f[:, abi.F_DISP_X], f[:, abi.F_DISP_Y], f[:, abi.F_ROT_Z] = 0.3, -0.2, t
        f[7, abi.F_ROT_Z] = np.nan
    dy, dx = (a.ravel() for a in np.mgrid[-h:h + 1, -h:h + 1])
    rows = torch.from_numpy(f).cuda()
    seed = torch.from_numpy(rng.uniform(0.5, 1.5, n)).cuda()
    out = []
    for lists in (False, True):
        with Schema(abi.default_params(subset_size=subset, shape_function=shape, enable_rotation=1)) as s:
            s.set_ref_image(ref)
            s.set_fields(f)
            if lists:
                s.set_subset_pixels(np.arange(n + 1) * len(dx), (cx[:, None] + dx).ravel(), (cy[:, None] + dy).ravel())
            s.set_def_image(deff)
            d = torch.zeros_like(deff)
            value, dparams = s.adjoint(rows, seed, ddef=d)
            torch.cuda.synchronize()
            out.append([a.double().cpu().numpy() for a in (value, dparams, d)])
    assert out[0][0][7] == -1.0 and out[1][0][7] == -1.0
    terms = 36.0 * n * subset ** 2 / size ** 2
    for a, b, tol in zip(out[0], out[1], (1e-12, 1e-12, max(1e-5, 4 * np.sqrt(terms) * 2.0 ** -24))):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
