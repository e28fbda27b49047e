"""Soups whose trees are deep and whose rays meet much of them: triangles of
sizes that span three decades around one point, and triangles that all overlap.
A ray's stack must hold what it has pushed: no call fails, and every closest
hit equals the brute-force scan's on the GPU, bit for bit."""
import os
import re

import numpy as np
import pytest

import lisa_gb300 as L
from helpers import random_rays
from lisa_gb300 import scenes as S
from test_gpu_build import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,t", [("nested", 65536), ("overlapping", 65536), ("overlapping", 1 << 20)])
def test_rays_through_deep_trees(gpu, kind, t):
    g = np.random.default_rng(10)
    if kind == "nested":
        c, size = g.uniform(-1, 1, (t, 1, 3)), np.exp2(g.uniform(-10, 0, (t, 1, 1)))
        v = (c + g.normal(size=(t, 3, 3)) * 0.3) * size
    else:
        v = g.uniform(-1, 1, (t, 3, 3))
    v = v.astype(np.float32).reshape(-1, 3)
    assert (_check(v, random_rays(v, 2000, seed=t)) >= 0).any()


def test_stack_covers_the_largest_scene_by_construction(gpu):
    """At most seven entries a level, for the 4,480,000-triangle sphere soup."""
    text = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lisa_gb300", "csrc",
                             "lisa_device.cuh")).read()
    entries = int(re.search(r"TRAV_STACK = (\d+);", text).group(1))
    r = L.Renderer(L.params_from_scene(S.sphere_soup(), num_samples=1))
    assert 7 * (r.bvh_info()["depth"] - 1) <= entries
    r.close()
