"""VSG strain after a caller moved subset centres through the fields' device
pointer by up to one pixel, which the neighbour grid of the first call allows
for: the neighbourhoods are those of the new coordinates.  Bit for bit against
the oracle (integer centres: the double sums are exact)."""
import numpy as np
import pytest

from dice_b200 import abi
from dice_b200 import synthetic as syn
from oracle import oracle as O

pytestmark = pytest.mark.gpu


class _Rows:
    """The context's field rows as a CUDA array."""

    def __init__(self, schema):
        self.__cuda_array_interface__ = {"shape": (schema.n, abi.FIELD_STRIDE), "typestr": "<f8",
                                         "data": (schema.fields_device_ptr(), False), "version": 2}


@pytest.mark.parametrize("every", [1, 3])
@pytest.mark.parametrize("window", [30, 41])
def test_strain_follows_moved_centres(every, window):
    torch = pytest.importorskip("torch")
    from dice_b200.schema import Schema
    rng = np.random.default_rng(window)
    X, Y = np.meshgrid(40 + 5 * np.arange(23), 50 + 5 * np.arange(19))
    f = syn.init_fields(X.ravel().astype(float), Y.ravel().astype(float))
    f[:, abi.F_DISP_X] = (0.01 * f[:, 0] + rng.normal(0, 0.05, len(f))).astype(np.float32)
    f[:, abi.F_DISP_Y] = (-0.02 * f[:, 1] + rng.normal(0, 0.05, len(f))).astype(np.float32)
    f[:, abi.F_SIGMA] = np.where(rng.random(len(f)) < 0.1, -1.0, 0.01)
    moved = f.copy()
    moved[::every, abi.F_COORD_X] += 1.0
    moved[::every, abi.F_COORD_Y] -= 1.0
    with Schema(abi.default_params(subset_size=21)) as s:
        s.set_fields(f)
        first = s.vsg_strain(window)
        torch.as_tensor(_Rows(s), device="cuda").copy_(torch.from_numpy(moved))
        torch.cuda.synchronize()
        got = s.vsg_strain(window)
    assert np.array_equal(first[:, :7], O.vsg_strain(f, window)[0])
    assert np.array_equal(got[:, :7], O.vsg_strain(moved, window)[0])
