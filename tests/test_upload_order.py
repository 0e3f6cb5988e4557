"""Tables that a call builds on the host and its kernels read right after, on a
non-blocking stream: the upload has to be done, or ordered before them, on that
stream.  Large neighbour grids, wave plans and pixel lists, rebuilt at every
call, against the same calls on the legacy stream.  (A late upload would show
as a stale table, and only sometimes.)"""
import numpy as np
import pytest

from dice_b200 import abi
from dice_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def test_rebuilt_tables_on_a_non_blocking_stream():
    torch = pytest.importorskip("torch")
    from dice_b200.schema import Schema
    rng = np.random.default_rng(2)
    size, n, side = 512, 40000, 5
    ref = syn.speckle_image(size, size, seed=1, blur_sigma=0.8).cuda()
    deff = syn.warp_image(ref, lambda X, Y: (0.3 + 0 * X, -0.2 + 0 * Y), noise_sigma=0.5, seed=2)
    dy, dx = (a.ravel() for a in np.mgrid[-side:side + 1, -side:side + 1])
    inputs = []
    for k in range(6):
        cx, cy = rng.integers(20, size - 20, n).astype(float), rng.integers(20, size - 20, n).astype(float)
        f = syn.init_fields(cx, cy)
        f[:, abi.F_DISP_X], f[:, abi.F_DISP_Y] = 0.3 + 1e-3 * cx, -0.2
        inputs.append((f, (cx[:, None] + dx).ravel().astype(np.int32), (cy[:, None] + dy).ravel().astype(np.int32)))
    offsets = (np.arange(n + 1) * len(dx)).astype(np.int32)
    p = abi.default_params(subset_size=0, optimization=abi.GRADIENT_BASED, fast_solver_tolerance=1e-2)
    out = []
    for stream in (torch.cuda.default_stream(), torch.cuda.Stream()):
        torch.cuda.synchronize()
        with Schema(p, stream=stream) as s:
            s.set_ref_image(ref)
            s.set_def_image(deff)
            got = []
            for f, px, py in inputs:
                s.set_fields(f)
                s.set_subset_pixels(offsets, px, py)
                s.execute_correlation()
                got.append(s.fields())
                s.load_fields(np.where(np.arange(abi.FIELD_STRIDE) == abi.F_SIGMA, 0.01, f))
                got.append(s.vsg_strain(9))
            out.append(got)
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
