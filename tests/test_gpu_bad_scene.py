"""A scene with a material index out of range is refused as invalid whatever
else its creation runs into: here an allocation cap that the scene, good or
bad, does not fit."""
import numpy as np
import pytest

import lisa_gb300 as L

pytestmark = pytest.mark.gpu
N = L._native


@pytest.mark.parametrize("estimator", [0, 1])
@pytest.mark.parametrize("cap", [1024, 100 * 1000])
def test_bad_material_comes_before_the_allocation_cap(gpu, cap, estimator):
    t = 1000
    g = np.random.default_rng(1)
    v = g.uniform(-1, 1, (3 * t, 3)).astype(np.float32)
    n = np.tile(np.array([0, 0, 1], np.float32), (3 * t, 1))
    mats = np.array([[1, 1, 0, 1, 1, 1, 0, 0, 0, 0]], np.float32)

    def code(mi):
        with pytest.raises(L.LisaError) as e:
            L.Renderer(L.params_from_arrays(v, n, mi, mats, 4, 4, (0, 0, 9), (0, 0, 0), 40, 1, 1), alloc_cap_bytes=cap,
                       estimator=estimator)
        return e.value.code, str(e.value)

    good, bad = np.zeros(t, np.int32), np.zeros(t, np.int32)
    bad[[700, 900]] = (1, -1)
    assert code(good)[0] == N.LISA_ERR_OOM
    c, text = code(bad)
    assert c == N.LISA_ERR_INVALID and text.endswith("triangle 700")
