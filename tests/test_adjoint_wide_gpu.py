"""Adjoints of grids so wide that one block per strip of columns is more
items than the partial-sum table has rows for in one launch (4096 strips of
60 columns in double, of 120 in float). Against the float64 numpy adjoint, at
the tolerance of the other adjoint tests."""
import numpy as np
import pytest

from test_adjoint_tiles_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,dtype,n", [
    ("star2d1r", np.float64, (1, 245761)), ("star2d1r", np.float64, (3, 300000)), ("box2d2r", np.float64, (2, 250001)),
    ("j2d5pt", np.float32, (1, 491521)), ("j2d5pt", np.float32, (2, 700001)), ("j2d9pt", np.float32, (2, 500000)),
], ids=str)
def test_linear_wide(name, dtype, n):
    check(name, dtype, n, 3, 2, 21)


@pytest.mark.parametrize("dtype,n", [(np.float64, (1, 245761)), (np.float64, (3, 300001)), (np.float32, (2, 491521))],
                         ids=str)
def test_gradient2d_wide(dtype, n):
    check("gradient2d", dtype, n, 3, 2, 22)
