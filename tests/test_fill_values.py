"""Local Radon transform of grids in which a fill value for missing data stands in a
few rows or columns: window sums a tile shares then span more binades than its
integers hold.  Bit for bit against the oracle."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

ANGLES = [0, 1, 30, 45, 46, 90, 91, 135, 179]


@pytest.mark.parametrize("fill", [1e15, 1e16, 1e17, -1e18, 1e20, -3e25, 1e38])
@pytest.mark.parametrize("dims", [(40, 230), (230, 40), (129, 140)])
def test_local_radon_beside_fill_values(gpu_lib, oracle, dims, fill):
    import skewengine_gb300 as ske
    dimx, dimy = dims
    x = np.ascontiguousarray(synthetic.blurred_texture(max(dims), 5)[0][:dimy, :dimx], np.float32)
    if dimy >= dimx:
        x[3:6] = fill
    else:
        x[:, -4:] = fill
    with ske.SkewEngine(dimx, dimy) as eng:
        got = eng.run("localradon", x, angles=ANGLES)
    want = oracle.run_angles(5, x, ANGLES)
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert bits_equal(np.where(nan, 0, got), np.where(nan, 0, want))
