"""The adjoint of squares wider than a warp, taken by columns in two and three
chunks of 32 lanes (sides of which three quarters of the lanes or more have a
column), against the same subsets as pixel lists: the comparison and tolerances
of test_adjoint_columns, whose sides above 31 but for 51 are taken by pixels.
Also one side of a single band that nearly fills the warp, and 3 px, ten bands."""
import pytest

from dice_b200 import abi
from tests import test_adjoint_columns as columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subset", [3, 29, 49, 57, 63, 85, 95])
@pytest.mark.parametrize("shape,objective,source", [(abi.AFFINE_SF, 0, 0), (abi.AFFINE_SF, 1, 1), (abi.QUADRATIC_SF, 0, 0)])
def test_chunks_equal_lists(subset, shape, objective, source):
    columns.test_columns_equal_lists(subset, shape, objective, source)
