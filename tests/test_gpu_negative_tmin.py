"""Given rays whose interval reaches behind their origin (tmin < 0): the
closest hit is the least t in (tmin, tmax), also a negative one, as the scan of
all triangles finds it, in every kernel that takes given rays (1,000 rays: one
a warp; 20,000: 32 a warp; 200,003: more)."""
import ctypes as C

import numpy as np
import pytest

import lisa_gb300 as L
from helpers import random_rays

pytestmark = pytest.mark.gpu
N = L._native


@pytest.mark.parametrize("n", [1000, 20000, 200003])
@pytest.mark.parametrize("tmin,tmax", [(-1.0, 1e16), (-np.inf, np.inf), (-3.0, -0.05), (-0.0, 1e16), (-0.25, 0.25)])
def test_hits_behind_the_origin(gpu, tmin, tmax, n):
    import torch

    g = np.random.default_rng(n)
    t = 700
    v = (g.uniform(-1, 1, (t, 1, 3)) + g.uniform(-0.3, 0.3, (t, 3, 3))).astype(np.float32).reshape(-1, 3)
    v[-9:] = v[:9]  # the first three triangles again: the lowest index wins
    rays = random_rays(v, n, seed=n)
    rays[:, 3], rays[:, 7] = tmin, tmax
    k = n // 20  # rays that start in a triangle's plane, at its first vertex
    rays[:k, :3] = v[::3][g.integers(0, t, k)]
    mats = np.array([[1, 1, 0, 1, 1, 1, 0, 0, 0, 0]], np.float32)
    r = L.Renderer(L.params_from_arrays(v, np.tile(np.array([0, 0, 1], np.float32), (3 * t, 1)), np.zeros(t), mats, 4,
                                        4, (0, 0, 9), (0, 0, 0), 40, 1, 1))
    d, verts = torch.from_numpy(rays).cuda(), torch.from_numpy(v).cuda()
    got = []
    for f in ("lisa_trace_brute_device", "lisa_trace_closest_device", "lisa_trace_soup_noalloc"):
        prim = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        dist = torch.full((n,), -7.0, dtype=torch.float32, device="cuda")
        out = (C.c_void_p(d.data_ptr()), n, C.c_void_p(prim.data_ptr()), C.c_void_p(dist.data_ptr()), None)
        torch.cuda.synchronize()
        first = (C.c_void_p(verts.data_ptr()), t) if f == "lisa_trace_soup_noalloc" else (r.handle,)
        N.check(getattr(N.lib(), f)(*first, *out))
        got.append((prim.cpu().numpy(), dist.cpu().numpy()))
    (p, x) = got[0]
    for q, y in got[1:]:
        assert np.array_equal(p, q)
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    hit = p >= 0
    assert hit.any() and (x[hit] > tmin).all() and (x[hit] < tmax).all()
    if tmin < 0:
        assert (x[hit] < 0).any()
    r.close()
