"""Viewshed sweep where its batches, masks and levels end: row lengths around one
and two observers to a lane (32, 64, 128 and their neighbours), every level
schedule, an observer height of zero and below, and terrain whose slopes tie.
Reference order against the oracle, bit for bit."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

ANGLES = [0, 1, 30, 44, 45, 89, 90, 120, 135, 179]
SHAPES = [(64, 0, 0), (32, 0, 0), (16, 48, 1), (48, 16, 0), (64, 64, 2)]


def _terrain(kind, dimx, dimy):
    if kind == "flat":
        return np.full((dimy, dimx), 3.0, np.float32)
    if kind == "plane":
        return (np.arange(dimx, dtype=np.float32)[None, :] * 0.25 + np.zeros((dimy, 1), np.float32)).copy()
    if kind == "below":
        return synthetic.fractal_dem(dimx, 7, side_y=dimy) - np.float32(400.0)
    return synthetic.fractal_dem(dimx, 7, side_y=dimy)


@pytest.mark.parametrize("kind,dims,povh", [
    ("dem", (31, 33), 1.5), ("dem", (64, 65), 0.0), ("dem", (97, 63), -2.0), ("dem", (127, 129), 1.5),
    ("dem", (160, 161), 1.5), ("dem", (193, 40), 1.5), ("flat", (130, 96), 0.0), ("flat", (130, 96), 1.5),
    ("plane", (161, 64), 0.0), ("below", (129, 100), 1.5),
])
def test_sweep_matches_oracle_at_its_edges(gpu_lib, oracle, kind, dims, povh):
    import skewengine_gb300 as ske
    x = _terrain(kind, *dims)
    want = oracle.run_ordered(0, x, ANGLES, povh=povh)
    with ske.SkewEngine(*dims) as eng:
        for shape in SHAPES:
            eng.set_sweep_shape(*shape)
            assert bits_equal(eng.run(0, x, angles=ANGLES, povh=povh, accum="reference"), want), shape
