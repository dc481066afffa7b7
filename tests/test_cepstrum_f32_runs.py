"""Float32 cepstrum: how many runs a tile's sectors are cut into depends on the
number of tiles, and must not show.  A batch whose tiles fill the GPU (one run)
against its images alone (eight), bit for bit: all angles, lists out of order, and
lists with fewer sectors of a type than runs; images with zero powers, whose
logarithms are infinite, and images every cell of which is left open."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

SIDE = 32  # one tile per type: 38 images make 152 tiles
KINDS = ("texture", "impulses", "signs", "zero", "flat")


def _image(kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "texture":
        x = synthetic.blurred_texture(SIDE, seed)[0]
    elif kind == "impulses":
        x = rng.random((SIDE, SIDE)) < 0.01
    elif kind == "signs":
        x = rng.integers(-1, 2, (SIDE, SIDE))
    else:
        x = np.full((SIDE, SIDE), 0.0 if kind == "zero" else 0.7)
    return np.ascontiguousarray(x, np.float32)


@pytest.mark.parametrize("angles", [None, [179, 3, 90, 45, 7, 120, 33], [50, 0, 44, 1, 2, 3, 4, 5, 6, 8, 9, 100]])
def test_runs_of_sectors_join_to_the_same_bits(gpu_lib, angles):
    import skewengine_gb300 as ske
    images = [_image(KINDS[i % len(KINDS)], i) for i in range(38)]
    batch = ske.run_batch(4, images, povh=synthetic.POVH, angles=angles, flags=ske.FLAG_CEPSTRUM_F32)
    for x, got in zip(images[:10], batch):
        with ske.SkewEngine(SIDE, SIDE) as eng:
            alone = eng.run(4, x, povh=synthetic.POVH, angles=angles, flags=ske.FLAG_CEPSTRUM_F32)
        assert bits_equal(got, alone)


def test_windows_of_one_value(gpu_lib):
    """An empty image and the cells of a flat one whose whole window is inside: no
    ascent anywhere, as in the exact operator."""
    import skewengine_gb300 as ske
    n = 128
    with ske.SkewEngine(n, n) as eng:
        zero = np.zeros((n, n), np.float32)
        assert bits_equal(eng.run(4, zero, flags=ske.FLAG_CEPSTRUM_F32), eng.run(4, zero))
        for value in (0.7, -3.0, 1e6):
            flat = np.full((n, n), value, np.float32)
            got = eng.run(4, flat, angles=[0], flags=ske.FLAG_CEPSTRUM_F32)
            assert bits_equal(got[:, 32:96], eng.run(4, flat, angles=[0])[:, 32:96])
            assert np.all(got[:, 32:96] == 0)
