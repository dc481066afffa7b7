"""Radon on non-square grids, rows inside their width, up to twice it (the limit of
the path whose row sums gather the skewed cells and whose deskew reads the
filtered row values) and beyond.  A whole run against the same sectors through
the per-sector calls (skew, row sums of the skewed grid, back-projection,
deskew), in binary64: equal bits.  The float32 mode against binary64 within its
stated error (1e-5 of the largest value, test_radon_float32_mode_error)."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

SIZES = [(1, 2), (2, 1), (33, 64), (64, 33), (40, 80), (80, 40), (41, 83), (96, 40), (65, 97), (190, 129)]


@pytest.mark.parametrize("accum", ["reference", "kahan"])
@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("dims", SIZES)
def test_radon_run_equals_sectors(gpu_lib, dims, special, accum):
    import skewengine_gb300 as ske
    dimx, dimy = dims
    x = synthetic.ellipse_phantom(dimx, 3, side_y=dimy)
    if special:
        x[dimy // 2, dimx // 2] = np.inf
        x[-1, -1] = np.nan
    with ske.SkewEngine(dimx, dimy) as eng:
        got = eng.run("radon", x, accum=accum)
        eng.prepare(x)
        for a in range(180):
            eng.skew(a)
            eng.kernel("radon")
            eng.deskew(0, accum=accum)
        want = eng.reduce()
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert bits_equal(np.where(nan, 0, got), np.where(nan, 0, want))


@pytest.mark.parametrize("dims", SIZES)
def test_radon_float32_error_non_square(gpu_lib, dims):
    import skewengine_gb300 as ske
    dimx, dimy = dims
    x = synthetic.ellipse_phantom(dimx, 5, side_y=dimy)
    with ske.SkewEngine(dimx, dimy) as eng:
        want = eng.run("radon", x)
        got = eng.run("radon", x, flags=ske.FLAG_RADON_F32)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
