"""Float32 cepstrum over angle lists that name angles more than once, also more often
than there are sectors: the maximum has an angle's bins from its last place in the
list."""
import numpy as np
import pytest

from skewengine_gb300 import synthetic
from tests.conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("angles", [[7, 3, 7], [30, 100, 30, 50, 140, 100], [5] * 400, list(range(180)) * 3,
                                    [20, 10] * 150 + [33]])
def test_last_place_of_a_repeated_angle_counts(gpu_lib, angles):
    import skewengine_gb300 as ske
    n = 90
    x = np.ascontiguousarray(synthetic.blurred_texture(n, 3)[0], np.float32)
    x[20:30, 40:60] = 0.5
    once = list(reversed(list(dict.fromkeys(reversed(angles)))))
    with ske.SkewEngine(n, n) as eng:
        got = eng.run(4, x, angles=angles, flags=ske.FLAG_CEPSTRUM_F32)
        assert bits_equal(got, eng.run(4, x, angles=once, flags=ske.FLAG_CEPSTRUM_F32))
        if len(angles) <= 6:  # the exact operator folds every sector of the list
            exact = eng.run(4, x, angles=angles)
            assert np.mean(exact != got) <= 1e-2 and np.array_equal(exact % 1000, got % 1000)
