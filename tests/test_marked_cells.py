"""Cells left to the binary64 kernels, by how many a warp reads at a time (one for a
sector of 64 x 64, 256 for all of 512 x 512): runs of a few sectors and of many on
images all, some or none of whose cells are left open.  The cepstrum against the
same sectors through the per-sector calls, the local Radon transform against the
oracle."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu


def _image(kind, dimx, dimy):
    x = synthetic.blurred_texture(max(dimx, dimy), 8)[0][:dimy, :dimx]
    if kind == "tiny":
        x = x * 1e-30
    elif kind == "band":  # all marked in a band of rows
        x = np.where(np.abs(np.arange(dimy) - dimy / 2)[:, None] < dimy / 8, 0.3, x)
    return np.ascontiguousarray(x, np.float32)


@pytest.mark.parametrize("kind", ["tiny", "band"])
@pytest.mark.parametrize("dimx,dimy,angles", [(64, 64, [30]), (40, 90, [100, 5]), (200, 150, [45]), (512, 512, [60]),
                                              (512, 512, [20, 50, 110, 140])])
def test_cepstrum(gpu_lib, kind, dimx, dimy, angles):
    import skewengine_gb300 as ske
    x = _image(kind, dimx, dimy)
    with ske.SkewEngine(dimx, dimy) as eng:
        got = eng.run("cepstrum", x, angles=angles)
        eng.prepare(x)
        for a in angles:
            eng.skew(a)
            eng.kernel("cepstrum")
            eng.deskew(1)
        assert bits_equal(got, eng.reduce(is_max=1))


@pytest.mark.parametrize("kind", ["tiny", "band"])
@pytest.mark.parametrize("dimx,dimy,angles", [(64, 64, [30]), (40, 90, [100, 5]), (200, 150, [45]),
                                              (300, 300, [20, 50, 110, 140])])
def test_local_radon(gpu_lib, oracle, kind, dimx, dimy, angles):
    import skewengine_gb300 as ske
    x = _image(kind, dimx, dimy)
    with ske.SkewEngine(dimx, dimy) as eng:
        got = eng.run("localradon", x, angles=angles)
    assert bits_equal(got, oracle.run_ordered(5, x, angles))
