"""Float32 Radon: the root mean square error of its output against binary64, as a
share of the largest value, is no larger than with a row's columns summed by a
warp's lanes (every 32nd column to a lane, the lanes by pairs): measured with that
form on the same images, the mean over six seeds."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

BY_LANES = {("phantom", 64, 64): 3.716e-08, ("texture", 64, 64): 1.293e-07, ("phantom", 200, 200): 7.706e-08,
            ("texture", 200, 200): 3.713e-07, ("phantom", 383, 509): 1.116e-07, ("texture", 383, 509): 1.262e-07,
            ("phantom", 512, 512): 1.812e-07, ("texture", 512, 512): 8.966e-07, ("phantom", 640, 480): 1.274e-07,
            ("texture", 640, 480): 1.384e-07, ("phantom", 1024, 1024): 3.668e-07, ("texture", 1024, 1024): 1.679e-06,
            ("phantom", 97, 190): 5.349e-08, ("texture", 97, 190): 7.927e-08, ("phantom", 1000, 700): 1.449e-07,
            ("texture", 1000, 700): 1.151e-07}


@pytest.mark.parametrize("kind,dimx,dimy", list(BY_LANES))
def test_error_no_larger_than_by_lanes(gpu_lib, kind, dimx, dimy):
    import skewengine_gb300 as ske
    rms = []
    with ske.SkewEngine(dimx, dimy) as eng:
        for seed in range(6):
            if kind == "phantom":
                x = synthetic.ellipse_phantom(dimx, seed, side_y=dimy)
            else:
                x = synthetic.blurred_texture(max(dimx, dimy), seed)[0][:dimy, :dimx]
            x = np.ascontiguousarray(x, np.float32)
            want = eng.run("radon", x).astype(np.float64)
            diff = eng.run("radon", x, flags=ske.FLAG_RADON_F32) - want
            rms.append(np.sqrt((diff ** 2).mean()) / np.abs(want).max())
    assert np.mean(rms) <= BY_LANES[kind, dimx, dimy], np.mean(rms)


@pytest.mark.parametrize("dims", [(1024, 1024), (700, 1200)])
def test_row_sums_do_not_depend_on_the_number_of_sectors(gpu_lib, dims):
    """The sectors of one type in one run, whose row sums keep 16 columns in flight,
    against each by itself (32 in flight), added up in turn: the same bits."""
    import skewengine_gb300 as ske
    x = synthetic.ellipse_phantom(dims[0], 3, side_y=dims[1])
    angles = list(range(0, 44))
    with ske.SkewEngine(*dims) as eng:
        together = eng.run("radon", x, angles=angles, flags=ske.FLAG_RADON_F32)
        want = np.zeros_like(together)
        for a in angles:
            want += eng.run("radon", x, angles=[a], flags=ske.FLAG_RADON_F32)
    assert bits_equal(together, want)
