"""Double 2-D kernels at every length of a block's last group of rows: blocks
whose rows and overlap are a whole number of groups, one row more and one
less, for the last block too, against the CPU oracle (exact mode bit for bit)
and the exact mode's result (FMA mode, 1e-12 relative)."""
import numpy as np
import pytest

import pyoracle as po
from gbstencil import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["star2d1r", "box2d1r", "box2d2r", "star2d3r", "gradient2d"])
@pytest.mark.parametrize("sl", range(1, 9))
@pytest.mark.parametrize("bt", [1, 2])
def test_block_tails(name, sl, bt):
    n, T = 41, 4
    A = po.init_grid(name, n, np.float64)
    want = A.copy()
    po.run(name, want, n, T)
    d, _ = capi.make_desc(name, np.float64, n, T, fp_mode="exact", bt=bt, sl=sl)
    exact = A.copy()
    capi.run_host(d, exact)
    assert np.array_equal(exact[T % 2], want[T % 2])
    d, _ = capi.make_desc(name, np.float64, n, T, fp_mode="fma", bt=bt, sl=sl)
    fma = A.copy()
    capi.run_host(d, fma)
    assert np.allclose(fma[T % 2], want[T % 2], rtol=1e-12, atol=0)
