"""One stream per pixel: small waves run a pixel's samples one after the other
in one launch (k_paths); with stage timing every sample is a wave of its own.
The same paths either way, so images, moments and ray counts are equal bit
for bit: fewer pixels than a warp has lanes, a queue that holds two and a
half samples of every pixel, less than one, several scenes with different
sample counts, further passes that go on with the pixels' streams.
"""
import numpy as np
import pytest

import lisa_gb300 as L
from lisa_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _both(params, **opt):
    out = []
    for timing in (0, 1):
        r = L.Renderer(params, rng=L._native.LISA_RNG_PER_PIXEL, accum_fp64=1, stage_timing=timing, **opt)
        st = [r.render(), r.render_progressive(3), r.render()]
        n = len(params) if isinstance(params, list) else 1
        out.append(([r.image(k, variance=True, fp64=True) for k in range(n)], st))
        assert all(x.device_status == 0 for x in st)
        r.close()
    (a, sa), (b, sb) = out
    for x, y in zip(a, b):
        for u, v in zip(x, y):
            assert np.array_equal(u, v)
    for x, y in zip(sa, sb):
        assert x.launches_nee == 0 and y.launches_nee > 0  # two different routes
        for k in ("paths", "rays_primary", "rays_bounce", "rays_shadow", "nee_vertices", "shadow_traversals"):
            assert getattr(x, k) == getattr(y, k), k
    return sa


@pytest.mark.parametrize("estimator", [0, 1])
@pytest.mark.parametrize("width,height,spp,queue", [(1, 1, 5, 0), (5, 3, 4, 0), (40, 25, 7, 0), (40, 25, 7, 2500),
                                                    (40, 25, 4, 999), (211, 97, 3, 0)])
def test_chains_are_the_waves(gpu, estimator, width, height, spp, queue):
    sc = S.hard_indirect(level=2, width=width, height=height, num_samples=spp, num_bounces=5)
    sa = _both(L.params_from_scene(sc), estimator=estimator, aperture=0.01, paths_in_flight=queue)
    assert sa[0].paths == width * height * spp
    if queue == 0:
        assert sa[0].launches_trace == 1


@pytest.mark.parametrize("queue", [0, 3000])
def test_scenes_in_one_wave(gpu, queue):
    params = [L.params_from_scene(S.cornell_box(width=w, height=h, num_samples=n, num_bounces=4))
              for w, h, n in ((23, 29, 3), (64, 1, 1), (17, 40, 6))]
    _both(params, paths_in_flight=queue)
