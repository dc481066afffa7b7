"""Float32 cepstrum of images whose cells the bounded evaluation leaves open: a tile
that goes without it for some sectors gives the bits of one that never does.  A run
over one type's sectors against each by itself (a lone sector is always tried
first), joined as the maximum does: the last angle and the largest bin; an infinite
value empties the cell (angle - 1000, which the fold's zero hides)."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

ANGLES = list(range(2, 44))


def _image(kind, n):
    y, x = np.mgrid[0:n, 0:n]
    t = synthetic.blurred_texture(n, 6)[0]
    image = {"flat": 0 * t + 0.7, "tiny": t * 1e-30, "huge": t * 1e25, "half flat": np.where(x < n // 2, 0.7, t),
             "band": np.where(np.abs(y - n / 2) < n / 6, t, 0.3), "ramp": 0.5 * x + 0.25 * y,
             "spot": np.exp(-((x - n / 2) ** 2 + (y - n / 2) ** 2) / (2.0 * n)), "zero": 0 * t}[kind]
    return np.ascontiguousarray(image, np.float32)


@pytest.mark.parametrize("kind", ["flat", "tiny", "huge", "half flat", "band", "ramp", "spot", "zero"])
@pytest.mark.parametrize("n", [97, 300])
def test_run_equals_its_sectors_joined(gpu_lib, n, kind):
    import skewengine_gb300 as ske
    x = _image(kind, n)
    with ske.SkewEngine(n, n) as eng:
        got = eng.run(4, x, angles=ANGLES, flags=ske.FLAG_CEPSTRUM_F32)
        bins = np.zeros((n, n), np.float32)
        for a in ANGLES:
            one = eng.run(4, x, angles=[a], flags=ske.FLAG_CEPSTRUM_F32)
            bins = np.where(one == 0, -1, np.maximum(bins, (one - a) / 1000))
    assert bits_equal(got, np.maximum(0, ANGLES[-1] + 1000 * bins))
    batch = ske.run_batch(4, [x] * 20, angles=ANGLES, flags=ske.FLAG_CEPSTRUM_F32)  # fewer runs of sectors
    assert all(bits_equal(b, got) for b in batch)
