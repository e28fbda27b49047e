"""FP64 mean and sample variance of an image (k_moments) against the sums of
the CPU oracle.

Sizes: one pixel, one past a warp, more values than one block, and more than
the launch has threads; one sample a pixel (no variance), two, and several;
with and without the FP64 mean's own sum; each output also alone.
"""
import numpy as np
import pytest

import lisa_gb300 as L
from lisa_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accum", [0, 1])
@pytest.mark.parametrize("width,height,spp", [(1, 1, 2), (11, 1, 1), (11, 3, 5), (97, 89, 2), (320, 180, 2)])
def test_moments_are_the_oracles(gpu, oracle, width, height, spp, accum):
    sc = S.cornell_box(width=width, height=height, num_samples=spp, num_bounces=3)
    r = L.Renderer(L.params_from_scene(sc), accum_fp64=accum)
    r.render()
    rgb, var, mean = r.image(variance=True, fp64=True)
    s, sq, _ = oracle.Scene.from_scene(sc).render(use_bvh=True)
    s, sq = s.reshape(height, width, 3), sq.reshape(height, width, 3)
    mu = s / spp if accum else rgb.astype(np.float64)
    same = (np.abs(rgb - s / spp) <= 1e-5 * np.maximum(1.0, np.abs(s / spp))).all(axis=2)
    assert (~same).mean() <= 0.002  # pixels whose paths are the oracle's
    if accum:
        assert np.allclose(mean[same], mu[same], rtol=1e-12, atol=0)
    else:
        assert np.array_equal(mean, mu)
    ref = np.maximum((sq / spp - mu * mu) * spp / (spp - 1.0), 0.0) if spp > 1 else np.zeros_like(mu)
    # the sums' own rounding, a few ulp of sq / n each, is all that may differ
    assert (np.abs(var - ref)[same] <= 1e-14 * spp * (sq / spp + mu * mu)[same] + 1e-300).all()
    # each output alone is the same
    assert np.array_equal(r.image(variance=True)[1], var)
    assert np.array_equal(r.image(fp64=True)[1], mean)
    assert np.array_equal(r.image(), rgb)
    alone = np.empty_like(mean)
    L._native.check(L._native.lib().lisa_get_image(r._h, 0, None, None, None, alone.ctypes.data))
    assert np.array_equal(alone, mean)
