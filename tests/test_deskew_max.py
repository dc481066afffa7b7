"""The maximum deskew (skewEngine.cuh:774-785) on both sides of the size where a
thread per cell gives way to tiles (512 x 512): per-type accumulators of a run over
sectors of all four types against NumPy on the sectors' own skewed cells, and the
whole grid's cells against those of the same sectors one by one."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

ANGLES = [3, 130, 44, 60, 100, 45, 91, 179, 20, 89, 150, 120]


@pytest.mark.parametrize("dims", [(40, 33), (511, 511), (512, 512), (513, 513), (640, 400), (400, 656)])
def test_maximum_keeps_last_angle_and_largest_bin(gpu_lib, dims):
    import skewengine_gb300 as ske
    dimx, dimy = dims
    x = np.ascontiguousarray(synthetic.blurred_texture(max(dims), 4)[0][:dimy, :dimx], np.float32)
    want = np.zeros((4, dimx * dimy), np.float32)
    used = 0
    with ske.SkewEngine(dimx, dimy) as eng:
        acc, mask = eng.accumulate("cepstrum", x, ANGLES)
        eng.prepare(x)
        for a in ANGLES:
            g = ske.geometry(dimx, dimy, a)
            eng.skew(a)
            eng.kernel("cepstrum")
            so = eng.skewed()[1]
            rows, cols = g["dim_o"], g["dim_i"]
            r = np.arange(rows)[:, None] + g["target"][None, :cols]
            at = r * cols + np.arange(cols)[None, :]
            lo, hi = so[at], so[at + cols]
            v = np.maximum(want[g["sector_type"]].reshape(rows, cols), np.maximum(lo, hi))
            bins = (v / np.float32(1000)).astype(np.int32)
            want[g["sector_type"]] = (a + 1000 * bins).astype(np.float32).ravel()
            used |= 1 << g["sector_type"]
    assert mask == used == 0xf
    assert bits_equal(acc, want)
