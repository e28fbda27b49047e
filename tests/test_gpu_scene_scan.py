"""The device scan of a new scene's triangles: material check, emissive
triangles and their bounds, leaf materials.

Triangle counts lie at the edges of a mask word (32) and of the size from
which the normals travel on a stream of their own (65,536); the emitters are
the first and last triangle or every one.  Images follow the CPU oracle,
which finds its emitters by itself.
"""
import numpy as np
import pytest

import lisa_gb300 as L
from lisa_gb300 import scenes as S

pytestmark = pytest.mark.gpu

COUNTS = [1, 31, 32, 33, 64, 65535, 65536, 65567]


def _scene(n, emitters, width=24, height=16, spp=2):
    g = np.random.default_rng(n)
    at = g.uniform(-1.0, 1.0, (n, 1, 3))
    size = min(0.5, 2.0 * n ** -0.4)
    v = (at + g.uniform(-size, size, (n, 3, 3))).astype(np.float32)
    e = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    nrm = np.repeat((e / np.linalg.norm(e, axis=1, keepdims=True))[:, None, :], 3, axis=1).astype(np.float32)
    mats, _ = S._box_walls(light=False)
    plain = next(m.name for m in mats if not m.emit and m.alpha >= 1.0)
    cut = {"edges": [0, 1, max(n - 1, 1), n], "all": [0, n, n, n]}[emitters]
    meshes = []
    for k, name in enumerate(["light", plain, "light"]):
        a, b = cut[k], cut[k + 1]
        if a < b:
            meshes.append(S.Mesh(f"part{k}", name, v[a:b], nrm[a:b]))
    return S.Scene(mats, meshes, width=width, height=height, num_samples=spp, num_bounces=4, name="scan",
                   **S._BOX_CAMERA)


@pytest.mark.parametrize("estimator", [0, 1])
@pytest.mark.parametrize("n,emitters", [(n, "edges") for n in COUNTS] + [(32, "all"), (33, "all"), (1000, "all")])
def test_emitters_of_the_scan_are_the_oracles(gpu, oracle, n, emitters, estimator):
    sc = _scene(n, emitters)
    r = L.Renderer(L.params_from_scene(sc), estimator=estimator)
    st = r.render()
    img = r.image()
    s, _, rays = oracle.Scene.from_scene(sc, estimator=estimator).render(use_bvh=True)
    ref = (s / sc.num_samples).reshape(sc.height, sc.width, 3)
    bad = (np.abs(img - ref) > 1e-5 * np.maximum(1.0, np.abs(ref))).any(axis=2)
    assert bad.mean() <= 0.005
    assert st.device_status == 0
    assert st.rays_primary == rays[0]
    for a, b in ((st.rays_bounce, rays[1]), (st.rays_shadow, rays[2])):
        assert abs(int(a) - int(b)) <= 0.005 * int(b) + 1


@pytest.mark.parametrize("n", COUNTS)
def test_first_bad_material_is_named(gpu, n):
    sc = _scene(n, "edges", 8, 8, 1)
    v, nrm, mi = sc.soup()
    mats = sc.material_table()
    for first in sorted({0, n // 2, n - 1}):
        m = mi.copy()
        m[first] = -1
        m[-1] = 99 if first < n - 1 else m[-1]
        p = L.params_from_arrays(v, nrm, m, mats, 8, 8, sc.eye, sc.look_at, sc.fov, 1, 2)
        with pytest.raises(L.LisaError, match=rf"triangle {first}$") as e:
            L.Renderer(p)
        assert e.value.code == L._native.LISA_ERR_INVALID
    L.Renderer(L.params_from_scene(sc)).close()  # the GPU is as before
