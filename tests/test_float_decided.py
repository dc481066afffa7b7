"""Operators whose float stage decides a cell and leaves the rest to binary64:
the local Radon transform against the oracle, and the cepstrum of a whole run
(bins decided in float) against the same sectors through the per-sector calls
(every value in binary64).  Equal bits on inputs that take each route: textures,
rows at the tiles' edges, flat and empty images (nothing decided), values far
from one, infinities and NaN."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (31, 33), (64, 64), (65, 127), (129, 66), (97, 97)]
ANGLES = [0, 1, 30, 44, 45, 46, 60, 89, 90, 91, 120, 135, 150, 179]


@pytest.fixture(scope="module")
def ske(gpu_lib):
    import skewengine_gb300 as ske
    return ske


def image(kind, dimx, dimy):
    rng = np.random.default_rng(17)
    x = synthetic.blurred_texture(max(dimx, dimy, 8), 5)[0][:dimy, :dimx]
    if kind == "bytes":
        x = rng.integers(0, 766, (dimy, dimx))
    elif kind == "zero":
        x = np.zeros((dimy, dimx))
    elif kind == "flat":
        x = np.full((dimy, dimx), 0.7)
    elif kind == "half":  # an empty half, as a phantom's background
        x = np.where(np.arange(dimx)[None, :] < dimx // 2, 0.0, x)
    elif kind == "signed":
        x = rng.standard_normal((dimy, dimx))
    elif kind == "tiny":
        x = x * 1e-25
    elif kind == "huge":
        x = x * 1e25
    elif kind == "wide":  # exponents too far apart for exact integer sums
        x = x * 10.0 ** rng.uniform(-12, 6, (dimy, dimx))
    elif kind == "nonfinite":
        x = np.array(x, np.float32)
        x[dimy // 2, dimx // 3] = np.inf
        x[dimy // 3, dimx // 2] = np.nan
        x[0, 0] = -np.inf
    return np.ascontiguousarray(x, np.float32)


KINDS = ["texture", "bytes", "zero", "flat", "half", "signed", "tiny", "huge", "wide", "nonfinite"]


def same(a, b):
    nan = np.isnan(a)
    return np.array_equal(nan, np.isnan(b)) and bits_equal(np.where(nan, 0, a), np.where(nan, 0, b))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dims", SIZES)
def test_local_radon_equals_oracle(ske, oracle, dims, kind):
    dimx, dimy = dims
    x = image(kind, dimx, dimy)
    with ske.SkewEngine(dimx, dimy) as eng:
        got = eng.run("localradon", x, angles=ANGLES)
    assert same(got, oracle.run_angles(5, x, ANGLES))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dims", SIZES)
def test_cepstrum_run_equals_binary64_sectors(ske, dims, kind):
    dimx, dimy = dims
    x = image(kind, dimx, dimy)
    with ske.SkewEngine(dimx, dimy) as eng:
        got = eng.run("cepstrum", x, angles=ANGLES)
        eng.prepare(x)
        for a in ANGLES:
            eng.skew(a)
            eng.kernel("cepstrum")
            eng.deskew(1)
        want = eng.reduce(is_max=1)
    assert same(got, want)
