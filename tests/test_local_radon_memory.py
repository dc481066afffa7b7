"""Local Radon transform by the memory its window sums get: none, sectors in groups,
and a child engine that borrows its parent's.  The same bits."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu


def _image(dimx, dimy, seed=3):
    return np.ascontiguousarray(synthetic.blurred_texture(max(dimx, dimy), seed)[0][:dimy, :dimx], np.float32)


@pytest.mark.parametrize("dims", [(1, 1), (33, 64), (70, 31), (97, 97)])
def test_without_memory_for_the_window_sums(gpu_lib, oracle, dims):
    """The allocation fails: the run still gives the reference's values, and the next
    one has its window sums again."""
    import skewengine_gb300 as ske
    x = _image(*dims)
    x[dims[1] // 2:, : dims[0] // 3] = 0
    x[0, 0] = np.inf
    angles = [0, 1, 44, 45, 46, 90, 91, 135, 179]
    want = oracle.run_angles(5, x, angles)
    nan = np.isnan(want)
    with ske.SkewEngine(*dims) as eng:
        eng.run("cepstrum", x, angles=angles)  # every other buffer
        try:
            gpu_lib.ske_inject_alloc_failure(0)
            first = eng.run("localradon", x, angles=angles)
        finally:
            gpu_lib.ske_inject_alloc_failure(-1)
        second = eng.run("localradon", x, angles=angles)
    for got in (first, second):
        assert np.array_equal(nan, np.isnan(got))
        assert bits_equal(np.where(nan, 0, got), np.where(nan, 0, want))


def test_groups_of_sectors(gpu_lib):
    """1500 x 1500 at 180 angles: 36 MB of window sums a sector, 119 sectors at a time
    and the rest, against two lists of 90."""
    import skewengine_gb300 as ske
    x = _image(1500, 1500)
    with ske.SkewEngine(1500, 1500) as eng:
        whole = eng.accumulate_resume("localradon", x, list(range(180)), None)
        half = eng.accumulate_resume("localradon", x, list(range(90)), None)
        half = eng.accumulate_resume("localradon", x, list(range(90, 180)), half)
    assert bits_equal(whole["acc"], half["acc"]) and whole["used"] == half["used"]


def test_children_borrow_the_window_sums(gpu_lib):
    import skewengine_gb300 as ske
    grids = [_image(a, b, 3 + a) for a, b in ((40, 40), (100, 80), (128, 128), (31, 90), (128, 128))]
    with ske.SkewEngine(128, 128) as eng:
        for _ in range(2):
            got = ske.run_batch("localradon", grids, engine=eng)
        alone = eng.run("localradon", grids[2])
    assert bits_equal(got[2], alone)
    for x, y in zip(grids, got):
        with ske.SkewEngine(x.shape[1], x.shape[0]) as eng:
            assert bits_equal(y, eng.run("localradon", x))
