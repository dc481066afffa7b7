"""Deskew kernels on both sides of the size where a thread per cell gives way to
tiles (320 x 320 cells for sums, 512 x 512 for the maximum): identity runs against
the oracle, reference order bit for bit and compensated within 1e-5, on grids with
and without rows that overrun their width and with row widths the tiles stage by
TMA and not."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

ANGLES = [0, 1, 17, 44, 45, 46, 89, 90, 91, 134, 135, 136, 179]


@pytest.mark.parametrize("dims", [(1, 1), (31, 33), (320, 320), (321, 319), (320, 321), (324, 324), (200, 512),
                                  (201, 513)])
def test_identity_deskew_matches_oracle(gpu_lib, oracle, dims):
    import skewengine_gb300 as ske
    dimx, dimy = dims
    x = synthetic.ellipse_phantom(dimx, 2, side_y=dimy)
    want = oracle.run_angles(3, x, ANGLES)
    with ske.SkewEngine(dimx, dimy) as eng:
        assert bits_equal(eng.run("identityimg", x, angles=ANGLES), want)
        kahan = eng.run("identityimg", x, angles=ANGLES, accum="kahan")
    assert np.abs(kahan - want).max() <= 1e-5 * max(1.0, float(np.abs(want).max()))


@pytest.mark.parametrize("side", [511, 512, 513])
def test_cepstrum_max_deskew_equals_sector_sums(gpu_lib, side):
    """The maximum keeps only the encoded angle of the last sector and the largest
    bin: a run over all angles of one type equals its sectors one by one."""
    import skewengine_gb300 as ske
    x, _, _ = synthetic.blurred_texture(side, 4)
    angles = [0, 5, 10]
    with ske.SkewEngine(side, side) as eng:
        got = eng.run("cepstrum", x, angles=angles)
        eng.prepare(x)
        for a in angles:
            eng.skew(a)
            eng.kernel("cepstrum")
            eng.deskew(1)
        assert bits_equal(got, eng.reduce(is_max=1))
