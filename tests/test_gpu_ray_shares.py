"""Closest hits of given rays at the counts where the launch changes its shape
(one ray a resident warp, 32 a warp, more than a warp has lanes): every ray is
answered once, as by the scan of all triangles.  Some rays have no direction
(a miss), some none left to hit."""
import ctypes as C

import numpy as np
import pytest

import lisa_gb300 as L
from helpers import random_rays

pytestmark = pytest.mark.gpu
N = L._native


@pytest.mark.parametrize("n", [1, 2, 33, 4863, 4864, 4865, 9729, 155647, 155648, 155649, 200003, 311297])
def test_every_ray_once(gpu, n):
    import torch

    g = np.random.default_rng(n)
    v = (g.uniform(-1, 1, (300, 1, 3)) + g.uniform(-0.2, 0.2, (300, 3, 3))).astype(np.float32).reshape(-1, 3)
    rays = random_rays(v, n, seed=n)
    rays[::7, 4:7] = 0.0
    mats = np.array([[1, 1, 0, 1, 1, 1, 0, 0, 0, 0]], np.float32)
    r = L.Renderer(L.params_from_arrays(v, np.tile(np.array([0, 0, 1], np.float32), (900, 1)), np.zeros(300), mats, 4, 4,
                                        (0, 0, 9), (0, 0, 0), 40, 1, 1))
    d = torch.from_numpy(rays).cuda()
    got = []
    for f in ("lisa_trace_closest_device", "lisa_trace_brute_device"):
        prim = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        dist = torch.full((n,), -7.0, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        N.check(getattr(N.lib(), f)(r.handle, C.c_void_p(d.data_ptr()), n, C.c_void_p(prim.data_ptr()),
                                    C.c_void_p(dist.data_ptr()), None))
        got.append((prim.cpu().numpy(), dist.cpu().numpy()))
    some = ~(rays[:, 4:7] == 0).all(axis=1)
    assert np.array_equal(got[0][0][some], got[1][0][some])
    assert np.array_equal(got[0][1][some].view(np.uint32), got[1][1][some].view(np.uint32))
    assert (got[0][0][~some] == -1).all() and np.isinf(got[0][1][~some]).all()
    if n > 100:
        assert (got[0][0] >= 0).any()
    visits = r.trace_count(rays)[0]
    assert visits >= some.sum() > 0 or n == 1
    r.close()
