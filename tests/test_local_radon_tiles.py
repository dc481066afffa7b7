"""Float32 local Radon in tiles of 32 rows (few tiles) and of 128: the sectors of one
type in one run against each by itself, added up in turn, the same bits; textures,
and images whose cells never ascend."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["texture", "ramp", "zero"])
@pytest.mark.parametrize("dims", [(400, 400), (321, 417)])
def test_tiles_of_both_heights_agree(gpu_lib, dims, kind):
    import skewengine_gb300 as ske
    dimx, dimy = dims
    if kind == "texture":
        x = synthetic.blurred_texture(max(dims), 2)[0][:dimy, :dimx]
    else:
        x = np.add.outer(np.arange(dimy), 2.0 * np.arange(dimx)) * (kind == "ramp")
    x = np.ascontiguousarray(x, np.float32)
    angles = list(range(40))
    with ske.SkewEngine(dimx, dimy) as eng:
        together = eng.run("localradon", x, angles=angles, flags=ske.FLAG_LOCAL_RADON_F32)
        want = np.zeros_like(x)
        for a in angles:
            want += eng.run("localradon", x, angles=[a], flags=ske.FLAG_LOCAL_RADON_F32)
    assert bits_equal(together, want)
