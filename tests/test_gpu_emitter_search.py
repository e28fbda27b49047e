"""The emitter search's candidate tries (k_nee) against the CPU oracle.

The search passes over tries whose line misses the emitters' bounds; the
paths, and the rays counted, must be those of the oracle, which traces every
try.  Emitters are placed where the test's decision is hardest: a point-like
light, bounds that enclose every vertex, a light far away and one in the
plane of a wall, none at all.  Frames have fewer vertices than a warp takes
from the queue at once, one more, and many.
"""
import numpy as np
import pytest

import lisa_gb300 as L
from lisa_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _scene(light, width, height, spp):
    mats, meshes = S._box_walls(light=False)
    quads = {
        "point": [((-1e-3, 0.3, -1e-3), 2e-3)],
        "around": [((-3.0, -2.0, -3.0), 6.0), ((-3.0, 2.0, -3.0), 6.0)],
        "far": [((-2e3, 4e3, -2e3), 4e3)],
        "wall": [((-0.5, -0.5, -0.5), 0.25)],
        "none": [],
    }[light]
    for i, ((x, y, z), e) in enumerate(quads):
        v, n = S.quad((x, y, z), (x, y, z + e), (x + e, y, z + e), (x + e, y, z), (0, -1, 0))
        meshes.append(S.Mesh(f"light{i}", "light", v, n))
    if light in ("around", "far"):
        meshes = [m for m in meshes if m.name != "ceiling"]  # the light comes in from above
    return S.Scene(mats, meshes, width=width, height=height, num_samples=spp, num_bounces=5, name=light,
                   **S._BOX_CAMERA)


@pytest.mark.parametrize("light", ["point", "around", "far", "wall", "none"])
@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (33, 1, 1), (24, 17, 4)])
def test_candidate_tries_give_the_oracles_paths(gpu, oracle, light, width, height, spp):
    sc = _scene(light, width, height, spp)
    r = L.Renderer(L.params_from_scene(sc))
    st = r.render()
    img = r.image()
    s, _, rays = oracle.Scene.from_scene(sc).render(use_bvh=True)
    ref = (s / spp).reshape(height, width, 3)
    bad = (np.abs(img - ref) > 1e-5 * np.maximum(1.0, np.abs(ref))).any(axis=2)
    assert bad.mean() <= 0.002
    assert st.device_status == 0
    assert st.rays_primary == rays[0]
    assert abs(int(st.rays_bounce) - int(rays[1])) <= 0.002 * rays[1]
    assert abs(int(st.rays_shadow) - int(rays[2])) <= 0.002 * rays[2]
