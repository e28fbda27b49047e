"""BVH builds at the sizes where the builder changes: one leaf, the first
nodes, the edges of a sort tile and of the two tile sizes; and soups whose
triangles (and so Morton codes) repeat or are very far apart.  Every closest hit equals the brute-force scan's on the GPU,
bit for bit."""
import ctypes as C

import numpy as np
import pytest

import lisa_gb300 as L
from helpers import random_rays

pytestmark = pytest.mark.gpu
N = L._native


def _check(v, rays):
    import torch

    n, t = rays.shape[0], v.shape[0] // 3
    mats = np.array([[1, 1, 0, 1, 1, 1, 0, 0, 0, 0]], np.float32)
    r = L.Renderer(L.params_from_arrays(v, np.tile(np.array([0, 0, 1], np.float32), (3 * t, 1)), np.zeros(t), mats, 4, 4,
                                        (0, 0, 9), (0, 0, 0), 40, 1, 1))
    info = r.bvh_info()
    assert info["tri_slots"] == t and 1 <= info["nodes"] <= t // 3 + 1
    d = torch.from_numpy(rays).cuda()
    got = []
    for f in ("lisa_trace_closest_device", "lisa_trace_brute_device"):
        prim = torch.empty(n, dtype=torch.int32, device="cuda")
        dist = torch.empty(n, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        N.check(getattr(N.lib(), f)(r.handle, C.c_void_p(d.data_ptr()), n, C.c_void_p(prim.data_ptr()),
                                    C.c_void_p(dist.data_ptr()), None))
        got.append((prim.cpu().numpy(), dist.cpu().numpy()))
    if t <= 65536:
        prim = torch.empty(n, dtype=torch.int32, device="cuda")
        dist = torch.empty(n, dtype=torch.float32, device="cuda")
        verts = torch.from_numpy(np.ascontiguousarray(v)).cuda()
        torch.cuda.synchronize()
        N.check(N.lib().lisa_trace_soup_noalloc(C.c_void_p(verts.data_ptr()), t, C.c_void_p(d.data_ptr()), n,
                                                C.c_void_p(prim.data_ptr()), C.c_void_p(dist.data_ptr()), None))
        got.append((prim.cpu().numpy(), dist.cpu().numpy()))
    for p, x in got[1:]:
        assert np.array_equal(got[0][0], p)
        assert np.array_equal(got[0][1].view(np.uint32), x.view(np.uint32))
    r.close()
    return got[0][0]


def _soup(t, seed, scale=1.0):
    g = np.random.default_rng(seed)
    c = g.uniform(-1, 1, (t, 1, 3))
    size = 2.0 * t ** (-1 / 3) * np.exp(g.normal(size=(t, 1, 1)) * 0.7)
    return ((c + g.normal(size=(t, 3, 3)) * size) * scale).astype(np.float32).reshape(-1, 3)


@pytest.mark.parametrize("t", [1, 2, 3, 4, 5, 8, 9, 17, 63, 64, 65, 255, 256, 257, 1023, 1024, 1025, 4097, 65536,
                               262144, 262145])
def test_sizes(gpu, t):
    v = _soup(t, t)
    hit = _check(v, random_rays(v, 2000 if t > 5000 else 20000, seed=t)) >= 0
    assert hit.any()


@pytest.mark.parametrize("kind", ["repeated", "huge"])
def test_hard_soups(gpu, kind):
    if kind == "repeated":  # every triangle four times: the lowest index wins
        v = np.tile(_soup(700, 2).reshape(-1, 9), (4, 1)).reshape(-1, 3)
    else:
        v = _soup(2000, 4, 1e15)
    v = np.ascontiguousarray(v, np.float32)
    rays = random_rays(v, 20000, seed=7)
    assert (_check(v, rays) >= 0).any()
