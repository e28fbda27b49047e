"""Guided waves whose bounces are all the BSDF's (fraction 1, as in the warm-up)
run without the network (k_bsdf_bounce).  With the largest fraction below 1
the network runs, and the same paths are drawn but for one draw in 2^24: the
mixture's share of the density, 2^-24 of at most about 0.3, moves a weight by
2e-8 over the cosine's density.

Vertices: fewer than a warp, past a block of 256, and more than the launch
has threads.
"""
import numpy as np
import pytest

import lisa_gb300 as L
from lisa_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _render(params, estimator, **opt):
    r = L.Renderer(params, mode=L._native.LISA_MODE_GUIDED, estimator=estimator, guide_min_spp=1,
                   guide_spp_per_wave=0, **opt)
    st = r.render()
    img = r.image()
    assert st.device_status == 0
    return img, st


@pytest.mark.parametrize("estimator", [0, 1])
@pytest.mark.parametrize("width,height,spp", [(3, 2, 1), (33, 9, 1), (320, 180, 4)])
def test_bounces_without_the_network(gpu, estimator, width, height, spp):
    sc = S.hard_indirect(level=2, width=width, height=height, num_samples=spp, num_bounces=6)
    p = L.params_from_scene(sc)
    a, sa = _render(p, estimator, guide_bsdf_fraction=1.0, guide_warmup_waves=0)
    w, sw = _render(p, estimator, guide_bsdf_fraction=0.25, guide_warmup_waves=1 << 30)
    assert np.array_equal(a, w)  # a warm-up wave is the same
    b, sb = _render(p, estimator, guide_bsdf_fraction=float(np.nextafter(np.float32(1), np.float32(0))),
                    guide_warmup_waves=0)
    far = (np.abs(a - b) > 1e-4 * np.maximum(np.abs(a), 1e-3)).any(axis=2)
    assert far.mean() <= 0.002
    assert sa.guide_infer_rows == sw.guide_infer_rows == 0 < sb.guide_infer_rows  # two different routes
    for k in ("rays_primary", "rays_bounce", "rays_shadow", "nee_vertices"):
        x, y, z = getattr(sa, k), getattr(sb, k), getattr(sw, k)
        assert x == z and abs(x - y) <= 0.001 * x, k
