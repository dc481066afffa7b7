"""Engines of different sizes in several threads at once: a kernel's limit of shared
memory is the process's, and one thread's launch must not take another's away."""
import threading

import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["sdem", "radon"])
def test_sizes_in_parallel(gpu_lib, op):
    """Short calls of one small and several larger sizes, over and over: the small
    ones' limit is below the others' need (Radon: more than 48 KB from 2049 rows)."""
    import skewengine_gb300 as ske
    sides = [(16, 16), (700, 40), (2000, 10), (24, 300)] if op == "sdem" else [(600, 30), (3000, 8), (2200, 12), (1500, 20)]
    angles = [0, 90] if op == "sdem" else [0, 45, 90]
    grids = [synthetic.fractal_dem(x, 3, side_y=y) for x, y in sides]
    alone = []
    for g in grids:
        with ske.SkewEngine(g.shape[1], g.shape[0]) as eng:
            alone.append(eng.run(op, g, angles=angles))
    errors = []

    def work(i):
        try:
            with ske.SkewEngine(grids[i].shape[1], grids[i].shape[0]) as eng:
                for _ in range(300):
                    if not bits_equal(eng.run(op, grids[i], angles=angles), alone[i]):
                        raise AssertionError(f"{grids[i].shape} differs")
        except Exception as ex:  # noqa: BLE001 - reported below, whatever it is
            errors.append(repr(ex))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(grids))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
