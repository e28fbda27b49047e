"""The work that users of lisa_gb300 have it do, through its public entry points.

Renders (reference and physically based estimator, plain and guided, one
scene and many, first frame and next frame), closest-hit queries over a soup
that changes every call, and training of the guide network on its own.

Rendered images have no value in ``exact``: which surface a path meets next
depends on every rounding before it, so a render in 64 bits follows other
paths.  Closest hits and the guide network have one.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

import lisa_gb300 as L
from lisa_gb300 import scenes as S

N = L._native

# scene family -> mean rays of a path, as a share of its bounce limit (the
# boxes are closed, a path ends early only at the light; most paths of the
# open soup leave it after a few bounces)
SEGMENTS = {"cornell": 0.9, "icosphere": 0.9, "hard_indirect": 0.95, "soup": 0.3, "batch": 0.5}


def listed():
    return [
        # a viewer redrawing a small pane, one sample a pixel per call: launches and host time
        dict(name="preview", kind="render", scene="cornell", size=0, width=160, height=90, spp=1, bounces=5, out="rgba8"),
        # the default Cornell scene, a whole small frame
        dict(name="cornell_frame", kind="render", scene="cornell", size=0, width=256, height=256, spp=64, bounces=7,
             out="image"),
        # one step of the headline frame: 1.31 M triangles, dielectric
        dict(name="icosphere_step", kind="render", scene="icosphere", size=8, width=1024, height=1024, spp=16, bounces=8,
             out="image"),
        # a new scene of that size: upload, BVH build, a short render, the PPM payload
        dict(name="icosphere_new", kind="new", scene="icosphere", size=8, width=512, height=512, spp=4, bounces=8,
             out="ppm"),
        # 4.48 M triangles, 20,000 materials, 2,000 emitters: divergent rays
        dict(name="soup_frame", kind="render", scene="soup", size=20000, width=1920, height=1080, spp=4, bounces=12,
             out="image"),
        # the reference's one random stream per pixel, a thin lens, an odd frame, FP64 mean and variance
        dict(name="pixel_stream_lens", kind="render", scene="icosphere", size=5, width=333, height=217, spp=8, bounces=6,
             out="moments", rng=1, aperture=0.02),
        # physically based estimator, plain sampling, a wide frame
        dict(name="physical_plain", kind="render", scene="hard_indirect", size=7, width=640, height=360, spp=16, bounces=8,
             out="image", estimator=1),
        # physically based, bounces drawn from a trained guide (training is over)
        dict(name="physical_guided", kind="render", scene="hard_indirect", size=8, width=1024, height=1024, spp=16,
             bounces=8, out="image", estimator=1, guide="fixed"),
        # the first waves of a guided render: the guide is trained, not yet sampled
        dict(name="guide_warmup", kind="render", scene="hard_indirect", size=7, width=512, height=512, spp=16, bounces=8,
             out="image", estimator=1, guide="warmup"),
        # several uneven scenes served by one renderer
        dict(name="batch", kind="render", scene="batch", size=12, width=0, height=256, spp=32, bounces=0, out="images"),
        # closest hits against a soup that is new on every call (no allocation, BVH built in place)
        dict(name="soup_query", kind="query", triangles=30001, rays=50003),
        # the guide network by itself: Adam steps and a forward pass on host arrays
        dict(name="guide_train", kind="guide", chunk=2048, steps=16, forward=10007),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["preview", "frame", "frame", "new", "soup", "lens", "physical", "guided", "batch", "query", "guide"])
    if kind == "query":
        return dict(kind="query", triangles=_log_int(rng, 2, 65536), rays=_log_int(rng, 1, 400000))
    if kind == "guide":
        return dict(kind="guide", chunk=128 * _log_int(rng, 1, 40), steps=rng.randint(1, 20), forward=_log_int(rng, 1, 40000))
    if kind == "batch":
        return dict(kind="render", scene="batch", size=rng.randint(2, 14), width=0, height=_log_int(rng, 130, 300),
                    spp=rng.choice([8, 16, 32]), bounces=0, out="images", estimator=rng.choice([0, 1]))
    w, h = _log_int(rng, 200, 1100), _log_int(rng, 150, 1024)
    c = dict(kind="render", width=w, height=h, bounces=rng.randint(2, 9), out="image", estimator=rng.choice([0, 0, 1]))
    spp = max(1, min(64, int(rng.uniform(0.1, 1.0) * (1 << 24) / (w * h))))
    if kind == "preview":
        return dict(c, scene="cornell", size=0, width=_log_int(rng, 17, 320), height=_log_int(rng, 17, 200), spp=1, out="rgba8")
    if kind == "frame":
        s = rng.choice(["cornell", "icosphere", "hard_indirect"])
        return dict(c, scene=s, size=0 if s == "cornell" else rng.randint(3, 8), spp=spp)
    if kind == "new":
        return dict(c, kind="new", scene="icosphere", size=rng.randint(3, 8), spp=min(spp, 8), out="ppm")
    if kind == "soup":
        return dict(c, scene="soup", size=_log_int(rng, 200, 20000), spp=min(spp, 4))
    if kind == "lens":
        return dict(c, scene="icosphere", size=rng.randint(3, 6), width=min(w, 400), height=min(h, 300), spp=rng.randint(1, 8),
                    rng=1, aperture=round(rng.uniform(0.0, 0.05), 3), estimator=0, out="moments")
    if kind == "physical":
        return dict(c, scene=rng.choice(["cornell", "hard_indirect"]), size=rng.randint(3, 7), spp=spp, estimator=1)
    return dict(c, scene="hard_indirect", size=rng.randint(3, 8), spp=min(spp, 16), guide=rng.choice(["fixed", "warmup"]))


# ----------------------------------------------------------------------------
# inputs


@functools.lru_cache(maxsize=12)
def _base_scene(family, size):
    """Meshes of a scene family; what the seed changes is applied afterwards."""
    if family == "cornell":
        return S.cornell_box()
    if family == "icosphere":
        return S.icosphere_box(level=size)
    if family == "hard_indirect":
        return S.hard_indirect(level=size)
    ext = 100.0 * (size / 20000) ** (1 / 3)
    sc = S.sphere_soup(n_spheres=size, extent=ext)
    sc.eye, sc.look_at = (ext / 2, ext / 2, ext * 1.75), (ext / 2, ext / 2, ext / 2)
    return sc


@functools.lru_cache(maxsize=12)
def _base_soup(family, size):
    sc = _base_scene(family, size)
    v, n, mi = sc.soup()
    # what turns with the seed: the noisy ball of a box, every sphere of a soup
    names = [m.name for m in sc.meshes]
    if family == "soup":
        first, last, centre = 0, v.shape[0], sc.look_at
    else:
        name = "sphere" if family == "cornell" else "icosphere"
        at = names.index(name)
        ends = np.cumsum([0] + [m.vertices.reshape(-1, 3).shape[0] for m in sc.meshes])
        first, last = int(ends[at]), int(ends[at + 1])
        centre = (-0.2, -0.34, 0.22) if family == "cornell" else (0.0, -0.18, 0.0)
    return v, n, mi, sc.material_table(), first, last, np.asarray(centre, np.float32)


def _params(case, seed):
    """RendererParams of a family, its round parts turned by the seed about the vertical through their centre."""
    sc = _base_scene(case["scene"], case["size"])
    v, n, mi, mats, first, last, centre = _base_soup(case["scene"], case["size"])
    a = np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi)
    turn = np.array([[math.cos(a), 0, -math.sin(a)], [0, 1, 0], [math.sin(a), 0, math.cos(a)]], np.float32)
    v, n = v.copy(), n.copy()
    v[first:last] = (v[first:last] - centre) @ turn + centre
    n[first:last] = n[first:last] @ turn
    return L.params_from_arrays(v, n, mi, mats, case["width"], case["height"], sc.eye, sc.look_at, sc.fov,
                                case["spp"], case["bounces"])


@functools.lru_cache(maxsize=2)
def _batch_base(n, max_res):
    return S.batch_scenes(n=n, seed=5, max_res=max_res)


def _options(case, seed):
    o = L.default_options(seed=seed % (1 << 31), estimator=case.get("estimator", 0), rng=case.get("rng", 0),
                          aperture=case.get("aperture", 0.0))
    if case["out"] == "moments":
        o.accum_fp64 = 1
    guide = case.get("guide")
    if guide:
        o.mode, o.guide_min_spp = N.LISA_MODE_GUIDED, 1
        if guide == "fixed":  # the budget of training steps is spent before the passes
            o.guide_warmup_waves, o.guide_train_steps = 0, 1
        else:
            o.guide_warmup_waves, o.guide_train_steps = 1 << 30, 0
    return o


def _network(seed, scale=1.0):
    """Guide parameters: He-uniform hidden layers, a small output layer, kappa starting at 2."""
    g = np.random.default_rng(seed)
    a = math.sqrt(6.0 / 64.0)
    w = [g.uniform(-a, a, (64, 64)) for _ in range(4)]
    w5 = g.uniform(-0.1, 0.1, (40, 64)) * scale
    b5 = np.zeros(40)
    b5[3::5] = math.log(2.0)
    return w, w5, np.zeros((4, 64)), b5


def _normal_following(seed):
    """A guide like a trained one: its lobes spread around the surface normal (features 39..41 are
    carried through the layers as positive and negative parts), with a part that varies with position."""
    w, w5, b, b5 = _network(seed, 0.5)
    g = np.random.default_rng(seed + 1)
    for layer in range(4):
        w[layer][:6] = 0.0
        w[layer][6:] *= 0.5
        for k in range(3):
            if layer == 0:
                w[0][2 * k, 39 + k], w[0][2 * k + 1, 39 + k] = 1.0, -1.0
            else:
                w[layer][2 * k, 2 * k] = w[layer][2 * k + 1, 2 * k + 1] = 1.0
    for lobe in range(8):
        for k in range(3):
            w5[5 * lobe + k, 2 * k], w5[5 * lobe + k, 2 * k + 1] = 1.0, -1.0
            b5[5 * lobe + k] = g.uniform(-0.5, 0.5)
        b5[5 * lobe + 3] = g.uniform(0.0, 2.0)
    return w, w5, b, b5


def _flat(net):
    w, w5, b, b5 = net
    return np.concatenate([np.concatenate([x.ravel() for x in w]), w5.ravel(), b.ravel(), b5]).astype(np.float32)


def _prepare_render(case, seed):
    o = _options(case, seed)
    if case["scene"] == "batch":
        g = np.random.default_rng(seed)
        ps = []
        for sc in _batch_base(case["size"], case["height"]):
            eye = tuple(np.asarray(sc.eye) + 0.02 * g.uniform(-1, 1, 3))
            ps.append(L.params_from_scene(sc, num_samples=min(sc.num_samples, case["spp"]), eye=eye))
        return {"case": case, "renderer": L.Renderer(ps, o), "scenes": len(ps)}
    p = _params(case, seed)
    if case["kind"] == "new":
        return {"case": case, "params": p, "options": o}
    r = L.Renderer(p, o)
    if case.get("guide") == "fixed":
        r.render_progressive(1)  # spends the training step
        r.guide().set_params(_flat(_normal_following(seed)))
        r.reset()
    return {"case": case, "renderer": r, "scenes": 1}


def _query_arrays(case, seed):
    """A closed room with small random triangles in it (every ray hits something), rays from points inside it."""
    g = np.random.default_rng(seed)
    t = case["triangles"]
    room, _ = S.box((-1.0, -1.0, -1.0), (1.0, 1.0, 1.0))
    inside = max(0, t - 12)
    c = g.uniform(-0.95, 0.95, (inside, 1, 3))
    tri = np.concatenate([room, c + g.normal(size=(inside, 3, 3)) * 0.6 / max(1, inside) ** (1 / 3)])[:t].astype(np.float32)
    tri[12:] = np.clip(tri[12:], -0.999, 0.999)
    rays = np.empty((case["rays"], 8), np.float32)
    rays[:, 0:3] = g.uniform(-0.9, 0.9, (case["rays"], 3))
    d = g.normal(size=(case["rays"], 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 3], rays[:, 7] = 1e-4, 1e16
    return tri.reshape(-1, 9), rays


def _guide_arrays(case, seed):
    """Encoded positions, normals and view directions, light directions around the normal and their weights."""
    g = np.random.default_rng(seed)
    n = case["chunk"] * case["steps"]
    u = g.uniform(0, 1, (n, 3))
    unit = lambda x: x / np.linalg.norm(x, axis=1, keepdims=True)  # noqa: E731
    nrm, view = unit(g.normal(size=(n, 3))), unit(g.normal(size=(n, 3)))
    f = np.zeros((n, 64), np.float32)
    for k in range(12):
        f[:, 3 * k:3 * k + 3] = np.sin(2.0 ** (k - 3) * math.pi * u)
    f[:, 36:39], f[:, 39:42], f[:, 42:45] = 2 * u - 1, nrm, view
    f[:, 45] = (nrm * view).sum(1)
    dirs = unit(nrm + 0.7 * g.normal(size=(n, 3))).astype(np.float32)
    weights = np.exp(g.normal(size=n)).astype(np.float32)
    return f, dirs, weights


def prepare(case, seed):
    if case["kind"] == "query":
        tri, rays = _query_arrays(case, seed)
        dev = {"device": "cuda"}
        return {"case": case, "tri": torch.from_numpy(tri).cuda(), "rays": torch.from_numpy(rays).cuda(),
                "prim": torch.empty(case["rays"], dtype=torch.int32, **dev),
                "t": torch.empty(case["rays"], dtype=torch.float32, **dev)}
    if case["kind"] == "guide":
        f, dirs, weights = _guide_arrays(case, seed)
        g = L.Guide(seed=1)
        g.set_params(_flat(_network(seed + 7)))
        return {"case": case, "guide": g, "features": f, "dirs": dirs, "weights": weights,
                "ask": np.resize(f, (case["forward"], 64))}
    return _prepare_render(case, seed)


# ----------------------------------------------------------------------------
# one pass


def _counts(st):
    return [int(st.rays_primary), int(st.rays_bounce), int(st.rays_shadow)]


def run(state):
    case = state["case"]
    if case["kind"] == "query":
        torch.cuda.current_stream().synchronize()  # the library reads the tensors on the default stream
        p = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
        N.check(N.lib().lisa_trace_soup_noalloc(p(state["tri"]), case["triangles"], p(state["rays"]), case["rays"],
                                                p(state["prim"]), p(state["t"]), None))
        return {"prim": state["prim"], "t": state["t"]}
    if case["kind"] == "guide":
        g = state["guide"]
        loss = g.train_steps(state["features"], state["dirs"], state["weights"], case["chunk"], case["steps"], 1e-3)
        return {"loss": loss, "params": g.params(), "out": g.forward(state["ask"])}
    if case["kind"] == "new":
        r = L.Renderer(state["params"], state["options"])
        st = r.render()
        out = {"rays": _counts(st), "ppm": r.ppm_rgb8(), "image": r.image()}
        r.close()
        return out
    r = state["renderer"]
    if case["out"] == "images":
        r.reset()
        st = r.render()
        return {"rays": _counts(st), "images": [r.image(k) for k in range(state["scenes"])]}
    st = r.render_progressive(case["spp"])
    out = {"rays": _counts(st)}
    if case["out"] == "rgba8":
        out["rgba8"] = r.rgba8()
    elif case["out"] == "moments":
        out["image"], out["variance"], out["mean64"] = r.image(variance=True, fp64=True)
    else:
        out["image"] = r.image()
    return out


# ----------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    if case["kind"] == "query":
        t, n = case["triangles"], case["rays"]
        # each ray descends to one leaf: eight boxes a level, one triangle test
        return {"bytes": 36.0 * t + 40.0 * n, "flops": n * (192.0 * max(1.0, math.log(t, 8)) + 60.0)}
    if case["kind"] == "guide":
        n = case["chunk"] * case["steps"]
        net = 2.0 * (4 * 64 * 64 + 64 * 40)
        return {"bytes": 4.0 * (68 * n + (64 + 40) * case["forward"] + 2 * 19240),
                "flops": net * (3.0 * n + case["forward"])}
    if case["scene"] == "batch":
        paths = tris = pixels = rays = 0
        for sc in _batch_base(case["size"], case["height"]):
            k = min(sc.num_samples, case["spp"])
            pixels += sc.width * sc.height
            paths += sc.width * sc.height * k
            rays += sc.width * sc.height * k * sc.num_bounces * SEGMENTS["batch"]
            tris += sc.num_triangles
    else:
        sc = _base_scene(case["scene"], case["size"])
        pixels = case["width"] * case["height"]
        paths, tris = pixels * case["spp"], sc.num_triangles
        rays = paths * max(1.0, case["bounces"] * SEGMENTS[case["scene"]])
    # the soup (vertices, normals, material), the accumulators in and out, the image out
    data = 76.0 * tris + pixels * (2 * 56.0 + 12.0)
    # a ray: one descent and one triangle test; a vertex: one shadow draw and one bounce
    flops = rays * (192.0 * max(1.0, math.log(max(tris, 8), 8)) + 60.0 + 60.0)
    if case.get("guide"):
        net = 2.0 * (4 * 64 * 64 + 64 * 40)
        flops += rays * net
        if case["guide"] == "warmup":
            flops += 3.0 * net * 128 * 19456 * max(1.0, paths / (1 << 22))
    return {"bytes": data, "flops": flops}


# ----------------------------------------------------------------------------
# the same in 64 bits


def _exact_query(case, seed):
    """Nearest hit by scanning every triangle (Moeller-Trumbore)."""
    if case["triangles"] * case["rays"] > 4e9:
        return None
    tri, rays = _query_arrays(case, seed)
    v = torch.from_numpy(tri).cuda().double().reshape(-1, 3, 3)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    r = torch.from_numpy(rays).cuda().double()
    out = torch.empty(r.shape[0], dtype=torch.float64, device="cuda")
    nrm = torch.linalg.cross(e1, e2)
    step = max(1, (1 << 24) // v.shape[0])
    for k in range(0, r.shape[0], step):
        o, d = r[k:k + step, 0:3], r[k:k + step, 4:7]
        # with s = o - v0 and n = e1 x e2: t = -(s.n)/(d.n), u and v from d . (s x e)
        det = -(d @ nrm.T)
        tn = o @ nrm.T - (v[:, 0] * nrm).sum(1)
        m = torch.linalg.cross(o, d)  # d . (o x e) = -(o x d) . e
        a = torch.linalg.cross(v[:, 0], e2)
        b = torch.linalg.cross(v[:, 0], e1)
        u = -(m @ e2.T) - d @ a.T  # d . ((o - v0) x e2)
        w = m @ e1.T + d @ b.T  # -d . ((o - v0) x e1)
        # u, w and det share a sign convention: u/det, w/det are the barycentrics
        u, w, t = -u / det, -w / det, tn / det
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-4) & (det != 0)
        out[k:k + step] = torch.where(ok, t, torch.full_like(t, math.inf)).min(1).values
    return {"prim": None, "t": out}


def _exact_guide(case, seed):
    f, dirs, weights = (torch.from_numpy(x).cuda().double() for x in _guide_arrays(case, seed))
    p = torch.from_numpy(_flat(_network(seed + 7))).cuda().double()

    def forward(p, x):
        for k in range(4):
            x = torch.relu(x @ p[4096 * k:4096 * (k + 1)].reshape(64, 64).T + p[18944 + 64 * k:18944 + 64 * (k + 1)])
        return x @ p[16384:18944].reshape(40, 64).T + p[19200:19240]

    def loss_of(p, x, d, w):
        o = forward(p, x).reshape(-1, 8, 5)
        mu = o[..., 0:3] / o[..., 0:3].norm(dim=2, keepdim=True).clamp_min(1e-6)
        kappa = torch.exp(o[..., 3].clamp(-4.0, 8.0))
        mix = torch.softmax(o[..., 4], 1)
        c = (mu * d[:, None, :]).sum(2)
        pdf = kappa / (2 * math.pi * -torch.expm1(-2 * kappa)) * torch.exp(kappa * (c - 1))
        return -(w * torch.log((mix * pdf).sum(1).clamp_min(1e-30))).mean()

    m, v, loss = torch.zeros_like(p), torch.zeros_like(p), None
    for k in range(case["steps"]):
        at = slice(k * case["chunk"], (k + 1) * case["chunk"])
        q = p.clone().requires_grad_(True)
        loss = loss_of(q, f[at], dirs[at], weights[at])
        (g,) = torch.autograd.grad(loss, q)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
    ask = torch.from_numpy(np.resize(_guide_arrays(case, seed)[0], (case["forward"], 64))).cuda().double()
    return {"loss": float(loss.detach()), "params": p, "out": forward(p, ask)}


def exact(case, seed):
    if case["kind"] == "query":
        return _exact_query(case, seed)
    if case["kind"] == "guide":
        return _exact_guide(case, seed)
    return None
