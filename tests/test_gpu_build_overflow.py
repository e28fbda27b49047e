"""BVH builds of soups whose SAH costs overflow: finite triangles some 1e17
across that overlap in their thousands, so that a subtree's cost is infinite
while its box's area is not.  Every subtree still has a partition to take, and
every closest hit equals the brute-force scan's on the GPU, bit for bit."""
import numpy as np
import pytest

from helpers import random_rays
from test_gpu_build import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,t", [("overlapping", 255), ("overlapping", 256), ("overlapping", 2000),
                                    ("overlapping", 65536), ("coincident", 256), ("coincident", 2000)])
def test_costs_that_overflow(gpu, kind, t):
    g = np.random.default_rng(t)
    v = g.uniform(-1.35e17, 1.35e17, (t, 3, 3))
    if kind == "coincident":
        v[:] = v[0]
    v = v.astype(np.float32).reshape(-1, 3)
    rays = random_rays(v, 2000, seed=t)
    rays[:, 4:7] *= np.float32(1e17)  # distances near 1, so that the triangle test does not overflow
    hit = _check(v, rays)
    assert (hit >= 0).any()
    if kind == "coincident":
        assert hit.max() == 0  # of equal hits the first triangle's
