"""VSG strain, a thread per subset in cell order: fields smaller and larger than
a block, ragged cells, subsets in any order, failed ones, and a window with
fewer than three neighbours.  Bit for bit against the oracle (integer centres:
the double sums are exact)."""
import numpy as np
import pytest

from dice_b200 import abi
from dice_b200 import synthetic as syn
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,step,window", [(1, 1, 5, 21), (2, 3, 4, 30), (11, 12, 5, 41), (43, 3, 7, 30), (37, 29, 3, 25),
                                               (16, 16, 20, 15)])
def test_strain_equals_oracle(nx, ny, step, window):
    from dice_b200.schema import Schema
    rng = np.random.default_rng(nx * 100 + ny)
    X, Y = np.meshgrid(40 + step * np.arange(nx), 50 + step * np.arange(ny))
    order = rng.permutation(nx * ny)
    f = syn.init_fields(X.ravel()[order].astype(float), Y.ravel()[order].astype(float))
    f[:, abi.F_DISP_X] = (0.01 * f[:, 0] + rng.normal(0, 0.05, len(f))).astype(np.float32)
    f[:, abi.F_DISP_Y] = (-0.02 * f[:, 1] + rng.normal(0, 0.05, len(f))).astype(np.float32)
    f[:, abi.F_SIGMA] = np.where(rng.random(len(f)) < 0.1, -1.0, 0.01)
    with Schema(abi.default_params(subset_size=21)) as s:
        s.set_fields(f)
        got = s.vsg_strain(window)
        match = s.fields()[:, abi.F_MATCH]
    want, failed = O.vsg_strain(f, window)
    assert np.array_equal(got[:, :7], want)
    assert np.array_equal(match == -1.0, failed != 0)
