"""Small waves run whole paths in one kernel (k_paths); with stage timing the
same waves run stage by stage.  Both trace the same paths, so the images, the
moments and the ray counts are equal bit for bit."""
import numpy as np
import pytest

import lisa_gb300 as L
from lisa_gb300 import scenes as S

pytestmark = pytest.mark.gpu
PB = L._native.LISA_ESTIMATOR_PHYSICAL


def _both(params, passes=1, **opt):
    out = []
    for timing in (0, 1):
        r = L.Renderer(params, accum_fp64=1, stage_timing=timing, **opt)
        for _ in range(passes):
            st = r.render()
        assert st.device_status == 0
        n = len(params) if isinstance(params, list) else 1
        out.append(([r.image(k, variance=True, fp64=True) for k in range(n)], st))
        r.close()
    (a, sa), (b, sb) = out
    assert sa.launches_nee == 0 and sb.launches_nee > 0  # two different routes
    for x, y in zip(a, b):
        for u, v in zip(x, y):
            assert np.array_equal(u, v)
    for k in ("rays_primary", "rays_bounce", "rays_shadow", "nee_vertices", "shadow_traversals"):
        assert getattr(sa, k) == getattr(sb, k), k
    return a


@pytest.mark.parametrize("estimator", [0, PB])
@pytest.mark.parametrize("width,height,spp,bounces", [(1, 1, 1, 1), (31, 1, 1, 2), (33, 1, 3, 7), (160, 90, 1, 5),
                                                      (200, 130, 8, 3)])
def test_sizes(gpu, estimator, width, height, spp, bounces):
    sc = S.cornell_box(width=width, height=height, num_samples=spp, num_bounces=bounces)
    img = _both(L.params_from_scene(sc), estimator=estimator)[0][0]
    if width * height > 1000:
        assert img.max() > 0


@pytest.mark.parametrize("kw", [dict(rng=1), dict(aperture=0.03), dict(use_graph=0), dict(refill_idle=1),
                                dict(threads_per_block=32, blocks_per_sm=1), dict(paths_in_flight=1000)],
                         ids=lambda k: "-".join(k))
@pytest.mark.parametrize("estimator", [0, PB])
def test_options(gpu, estimator, kw):
    sc = S.hard_indirect(level=3, width=61, height=47, num_samples=3, num_bounces=6)
    _both(L.params_from_scene(sc), passes=2, estimator=estimator, **kw)


@pytest.mark.parametrize("estimator", [0, PB])
def test_scenes(gpu, estimator):
    """Uneven scenes in one wave: many emitters (their own BVH), none, dielectrics, no triangles."""
    ext = 100.0 * (300 / 20000) ** (1 / 3)
    soup = S.sphere_soup(n_spheres=300, width=40, height=30, num_samples=2, num_bounces=9, extent=ext)
    soup.eye, soup.look_at = (ext / 2, ext / 2, ext * 1.75), (ext / 2, ext / 2, ext / 2)
    dark = S.icosphere_box(level=3, width=17, height=19, num_samples=4, num_bounces=4)
    dark.meshes = [m for m in dark.meshes if m.name != "light"]
    box = S.cornell_box(width=23, height=29, num_samples=3, num_bounces=1)
    params = [L.params_from_scene(s) for s in (soup, dark, box)]
    params.append(L.params_from_arrays(np.zeros((0, 3)), np.zeros((0, 3)), np.zeros(0), np.zeros((0, 10)), 5, 3,
                                       (0, 0, 1), (0, 0, 0), 40, 2, 3))
    a = _both(params, estimator=estimator)
    assert a[0][0].max() > 0 and a[3][0].max() == 0
