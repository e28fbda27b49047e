"""bvh_info's build_ms is the construction's own time: it does not grow with
the copy of the normals, which travels beside the build.  Pages of a fresh
array of zeros are only made when the copy first reads them, which takes longer
than the build."""
import numpy as np
import pytest

import lisa_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [60000, 2000000])
def test_build_time_leaves_the_normals_copy_out(gpu, t):
    g = np.random.default_rng(3)
    v = (g.uniform(-1, 1, (t, 1, 3)) + g.normal(size=(t, 3, 3)) * t ** (-1 / 3)).astype(np.float32).reshape(-1, 3)
    mats = np.array([[1, 1, 0, 1, 1, 1, 0, 0, 0, 0]], np.float32)
    mi = np.zeros(t, np.int32)

    def build_ms(normals):
        r = L.Renderer(L.params_from_arrays(v, normals, mi, mats, 4, 4, (0, 0, 9), (0, 0, 0), 40, 1, 1))
        ms = r.bvh_info()["build_ms"]
        r.close()
        return ms

    touched = np.tile(np.array([0, 0, 1], np.float32), (3 * t, 1))
    warm = min(build_ms(touched) for _ in range(4))
    assert 0.0 < warm < 50.0
    assert build_ms(np.zeros((3 * t, 3), np.float32)) <= 1.5 * warm + 0.3
