"""Performance cases of the renderer.

Each case is one piece of work that a program using this package asks for
through its public entry points: ray queries, scene configuration, a forward
image, a render + gradient step, a batch of views, an inverse-rendering step,
a batch of served requests. `listed` holds the sizes that the package's own
configurations use, from the smallest call to the largest; `draw` gives others
from the same ranges.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tensorray_b200 import api, autograd, scenes, serve

# rays traced per path sample by each term, of the order that the work
# counters show on the displaced-sphere scene; used by `work` only
RAYS = {"interior": 3.0, "primary": 1.5, "direct": 0.5, "indirect": 3.0, "pixel": 3.0}
TERMS = ("primary", "direct", "indirect", "pixel")


def listed():
    return [
        # a preview while a scene is being set up: launches and host time only
        dict(name="preview", kind="image", scene="ico", tris=1284, w=32, h=24, spp=1, depth=3),
        # a program's own visibility queries: a few, and a whole frame's worth
        dict(name="rays_few", kind="rays", scene="ggx", tris=100_000, n=4099),
        dict(name="rays_frame", kind="rays", scene="ggx", tris=100_000, n=1 << 20),
        # new vertex positions: geometry chain and acceleration structure
        dict(name="configure", kind="configure", scene="ggx", tris=100_000, refit=False),
        # the icosphere configuration: 256 x 256, 16 spp, depth 3, 3 terms
        dict(name="ico_step", kind="step", scene="ico", tris=1284, w=256, h=256, spp=16, depth=3,
             primary=True, direct=True, indirect=False, pixel=False),
        # an image that no tile size divides, an odd spp, all terms
        dict(name="ragged_step", kind="step", scene="ggx", tris=20_000, w=332, h=251, spp=5, depth=7,
             primary=True, direct=True, indirect=True, pixel=True),
        # long paths: above the depth that the smaller path records hold
        dict(name="deep_step", kind="step", scene="ggx", tris=100_000, w=256, h=256, spp=8, depth=12,
             primary=True, direct=True, indirect=True, pixel=True),
        # a final image of the displaced-sphere configuration
        dict(name="ggx_image", kind="image", scene="ggx", tris=100_000, w=512, h=512, spp=64, depth=5),
        # the displaced-sphere configuration: 100K triangles, GGX and texture,
        # 512 x 512, 64 spp, depth 5, all terms, vertex and texel gradients
        dict(name="ggx_step", kind="step", scene="ggx", tris=100_000, w=512, h=512, spp=64, depth=5,
             primary=True, direct=True, indirect=True, pixel=True),
        # multi-view optimisation of the icosphere scene, mixed sizes
        dict(name="views_mixed", kind="views", scene="ico", tris=1284, views=8, res_lo=128, res_hi=512, spp_lo=8,
             spp_hi=64, depth=3, guided=False, refit=False, sigma=0.0, cache=False),
        # a step of the inverse-rendering loop: perturbed start mesh, refit,
        # guided direct boundary, depth 8, few spp
        dict(name="inverse_step", kind="views", scene="served", tris=300_000, views=4, res_lo=512, res_hi=512,
             spp_lo=2, spp_hi=2, depth=8, guided=True, refit=True, sigma=0.004, cache=True),
        # render + gradient requests on two resident scenes, as the server batches them
        dict(name="served", kind="served", scene="served", tris=50_000, requests=8, res_lo=128, res_hi=384, spp_lo=4,
             spp_hi=32, depth=4),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["image", "image", "step", "step", "step", "rays", "configure", "views"])
    scene = rng.choice(["ico", "ggx", "ggx"])
    tris = 1284 if scene == "ico" else log(5_000, 200_000)
    case = dict(kind=kind, scene=scene, tris=tris)
    if kind == "rays":
        case.update(n=log(1_000, 1_500_000))
    elif kind == "configure":
        case.update(refit=rng.random() < 0.5)
    elif kind == "views":
        case.update(views=rng.randint(1, 6), res_lo=log(32, 128), res_hi=log(129, 384), spp_lo=rng.randint(1, 4),
                    spp_hi=rng.randint(4, 16), depth=rng.randint(1, 8), guided=rng.random() < 0.5,
                    refit=rng.random() < 0.5, sigma=rng.choice([0.0, 0.001]), cache=rng.random() < 0.5)
    else:
        # W is a multiple of 4: the pixel term needs W * H * spp divisible by 4
        w, h = 4 * log(8, 128), log(24, 512)
        spp = max(1, min(log(1, 64), 16_000_000 // (w * h)))
        case.update(w=w, h=h, spp=spp, depth=rng.randint(1, 12))
        if kind == "step":
            case.update({t: rng.random() < 0.75 for t in TERMS})
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _mesh_spec(scene, tris):
    """The scene file a program would load (the same for every seed)."""
    if scene == "ico":
        return scenes.config1_scene(64, 64)
    if scene == "ggx":
        return scenes.config2_scene(64, 64, tris=tris)
    return scenes.served_scene(tris, seed=5)


def _spec(scene, tris, w=64, h=64):
    base = _mesh_spec(scene, tris)
    return scenes.SceneSpec(base.meshes, base.bsdfs, base.lights, base.textures,
                            [scenes.CameraSpec((0.0, 0.0, 4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), w, h, 45.0)])


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _positions(sc, gen, sigma):
    """Vertex positions of an optimisation under way: the first shape moved a
    little as a whole, and every vertex of it by N(0, sigma^2)."""
    V = sc._raw_positions.clone()
    s = sc.shapes[0].vertex_slice()
    V[s] += 0.05 * torch.randn(1, 3, generator=gen, device=V.device)
    V[s] += sigma * torch.randn(V[s].shape, generator=gen, device=V.device)
    return V


def _target(h, w, gen):
    """A target image: the scene's range of radiance, smooth."""
    t = torch.rand(1, 3, 5, 5, generator=gen, device="cuda") * 0.5
    return torch.nn.functional.interpolate(t, (h, w), mode="bilinear", align_corners=True)[0].permute(1, 2, 0).contiguous()


def _sigma(case):
    return 0.0 if case["scene"] == "ico" else 0.02 / math.sqrt(case["tris"] / 1000.0)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind in ("image", "step"):
        sc = api.Scene(_spec(case["scene"], case["tris"], case["w"], case["h"]))
        V = _positions(sc, gen, _sigma(case))
        sc.set_vertex_positions(V)
        sc.configure()
        n = {t: case["spp"] if case.get(t) else 0 for t in TERMS}
        opts = api.RenderOptions(seed % 100_003, case["depth"], case["spp"], n["primary"], n["direct"],
                                 n["indirect"], n["pixel"])
        st.update(scene=sc, options=opts)
        if kind == "image":
            st.update(integrator=api.PathTracer())
        else:
            T = torch.rand(sc.num_texels, 3, generator=gen, device="cuda") * 0.6 + 0.2
            st.update(context=autograd.RenderContext(sc, opts), V=V.requires_grad_(True),
                      T=T.requires_grad_(sc.num_texels > 0), target=_target(case["h"], case["w"], gen))
    elif kind == "rays":
        sc = api.Scene(_spec(case["scene"], case["tris"]))
        sc.set_vertex_positions(_positions(sc, gen, _sigma(case)))
        sc.configure()
        st.update(scene=sc, rays=_rays(sc, case["n"], gen))
    elif kind == "configure":
        sc = api.Scene(_spec(case["scene"], case["tris"]))
        sc.configure()
        st.update(scene=sc, V=_positions(sc, gen, _sigma(case)))
    elif kind == "views":
        sc = api.Scene(_spec(case["scene"], case["tris"]))
        sc.configure()
        V = _positions(sc, gen, case["sigma"])
        sc.set_vertex_positions(V)
        sc.configure(refit=case["refit"])
        cams, spps = _views(case, seed)
        vs = api.ViewSet(sc, cams, spps)
        if case["cache"]:
            vs.set_path_cache(64 << 30)
        opts = api.RenderOptions(seed % 100_003, case["depth"], 0, 0, 0, 0, 0)
        opts.g_direct = case["guided"]
        st.update(scene=sc, V=V, views=vs, options=opts, d=torch.empty(vs.npix, 3, device="cuda"),
                  targets=torch.cat([_target(c.height, c.width, gen).reshape(-1, 3) for c in cams]))
    else:
        world = {"small": api.Scene(_spec("ico", 1284)), "large": api.Scene(_spec(case["scene"], case["tris"]))}
        for sc in world.values():
            sc.set_vertex_positions(_positions(sc, gen, 0.0))
            sc.configure()
        server = serve.Server(world)
        server.warmup()
        rng, sizes = np.random.default_rng(seed), np.random.default_rng(0)
        asked = []
        for i in range(case["requests"]):
            res = _between(sizes, case["res_lo"], case["res_hi"])
            asked.append(dict(scene="small" if i % 2 else "large", camera=_camera(rng, res),
                              spp=_between(sizes, case["spp_lo"], case["spp_hi"]), depth=case["depth"],
                              target=_target(res, res, gen).reshape(-1, 3), seed=i + 1))
        st.update(server=server, asked=asked)
    return st


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) if hi > lo else lo


def _camera(rng, res):
    u = rng.normal(size=3)
    p = 4.0 * u / np.linalg.norm(u)
    up = (0.0, 1.0, 0.0) if abs(p[1]) < 3.9 else (1.0, 0.0, 0.0)
    return api.Camera(tuple(float(x) for x in p), (0.0, 0.0, 0.0), up, res, res, 45.0)


def _views(case, seed):
    """Poses on a Fibonacci sphere turned by the seed; resolutions and spp
    spread over their ranges (the same total for every seed)."""
    n = case["views"]
    f = [i / (n - 1) if n > 1 else 1.0 for i in range(n)]
    res = [int(round(case["res_lo"] * (case["res_hi"] / case["res_lo"]) ** x)) for x in f]
    spps = [int(round(case["spp_lo"] * (case["spp_hi"] / case["spp_lo"]) ** (1.0 - x))) for x in f]
    a = 2.0 * math.pi * (seed % 997) / 997.0
    cams = []
    for c, r in zip(scenes.fibonacci_cameras(n, 4.0, [64], seed=2), res):
        x, y, z = c.pos
        p = (x * math.cos(a) - z * math.sin(a), y, x * math.sin(a) + z * math.cos(a))
        cams.append(api.Camera(p, c.target, c.up, r, r, 45.0))
    return cams, spps


def _rays(sc, n, gen):
    """Half camera rays towards the object, half rays leaving surface points
    in every direction, in random order."""
    d = sc.device
    P = sc.geometry()["positions"][sc.shapes[0].vertex_slice()]
    k = n // 2
    pick = torch.randint(len(P), (n,), generator=gen, device=d)
    org = P[pick].clone()
    dirs = torch.randn(n, 3, generator=gen, device=d)
    cam = torch.tensor([0.0, 0.0, 4.0], device=d)
    dirs[:k] = org[:k] * 1.2 + 0.1 * dirs[:k] - cam
    org[:k] = cam
    dirs = dirs / dirs.norm(dim=1, keepdim=True)
    order = torch.randperm(n, generator=gen, device=d)
    org, dirs = org[order].contiguous(), dirs[order].contiguous()
    return org, dirs, torch.full((n,), 1e-2, device=d), torch.full((n,), 1e32, device=d)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "image":
        return st["integrator"].renderC(st["scene"], st["options"])
    if kind == "step":
        st["V"].grad = st["T"].grad = None
        img = autograd.render(st["V"], st["T"], st["context"])
        loss = 0.5 * (img - st["target"]).square().sum()
        loss.backward()
        out = {"image": img.detach(), "loss": loss.detach(), "positions": st["V"].grad}
        if st["T"].requires_grad:
            out["texels"] = st["T"].grad
        return out
    if kind == "rays":
        tri, u, v, t = st["scene"].intersect(*st["rays"])
        vis = st["scene"].occluded(*st["rays"])
        return {"tri": tri, "u": u, "v": v, "t": t, "visible": vis}
    if kind == "configure":
        sc = st["scene"]
        sc.set_vertex_positions(st["V"])
        sc.configure(refit=case["refit"])
        return sc.geometry()
    if kind == "views":
        sc, vs, opts = st["scene"], st["views"], st["options"]
        sc.set_vertex_positions(st["V"])
        sc.configure(refit=case["refit"])
        img = vs.render(api.TRN_PATH_TRACER, opts)
        loss = vs.loss(img, st["targets"], st["d"])
        for term in (api.TRN_PATH_TRACER, api.TRN_PRIMARY_EDGE, api.TRN_DIRECT_EDGE):
            vs.render_grad(term, opts, st["d"])
        return {"image": img, "loss": loss, "positions": sc.get_grads()["positions"]}
    reqs = [serve.RenderRequest(**a) for a in st["asked"]]
    st["server"].run(reqs)
    return {"r%d" % i: {"image": r.image, "loss": r.loss, "positions": r.grad_positions} for i, r in enumerate(reqs)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _sizes(case):
    """(triangles, vertices, edges, texels), close enough for the byte count."""
    t = case["tris"]
    return t, t // 2, 3 * t // 2, 512 * 512 if case["scene"] == "ggx" else 0


def work(case):
    kind = case["kind"]
    T, V, E, X = _sizes(case)
    # one ray: a box pair per level of a balanced tree (2 x 6 multiply-adds
    # and 11 min/max) and one triangle test
    ray = math.log2(T) * 46 + 60
    scene = 12 * V + 12 * T + 36 * T + 12 * X
    if kind == "rays":
        return {"bytes": scene + case["n"] * (2 * 32 + 16 + 4), "flops": 2 * case["n"] * ray}
    if kind == "configure":
        return {"bytes": 12 * V + 12 * T + (12 + 12) * V + 16 * T + 64 * T + 48 * T, "flops": 200 * T}
    shade = 400  # BSDF, light sample and frame at one path vertex
    if kind in ("image", "step"):
        n = case["w"] * case["h"] * case["spp"]
        rays = RAYS["interior"] + sum(RAYS[t] for t in TERMS if case.get(t))
        grad = 12 * V + 12 * X if kind == "step" else 0
        image = 12 * case["w"] * case["h"]
        return {"bytes": scene + image + grad + (scene + image + 112 * T if kind == "step" else 0),
                "flops": n * rays * (ray + shade) * 1.0}
    if kind == "views":
        n = pix = 0
        k = case["views"]
        for i in range(k):
            x = i / (k - 1) if k > 1 else 1.0
            r = case["res_lo"] * (case["res_hi"] / case["res_lo"]) ** x
            pix += r * r
            n += r * r * case["spp_lo"] * (case["spp_hi"] / case["spp_lo"]) ** (1.0 - x)
        rays = RAYS["interior"] + RAYS["primary"] + RAYS["direct"]
        return {"bytes": 2 * scene + 112 * T + 48 * pix + 12 * V, "flops": n * rays * (ray + shade)}
    res2 = case["res_lo"] * case["res_hi"]
    spp = math.sqrt(case["spp_lo"] * case["spp_hi"])
    n = case["requests"] * res2 * spp
    return {"bytes": 2 * scene + case["requests"] * (48 * res2 + 24 * V),
            "flops": n * (2 * RAYS["interior"] + RAYS["primary"] + RAYS["direct"]) * (ray + shade)}


def tolerance(case):
    kind = case["kind"]
    if kind == "rays":
        # every float operation of the hit test is individually rounded and
        # ties go to the smaller triangle index: one result, bit for bit
        return "exact"
    if kind == "configure":
        return {"rel": 1e-6}
    # sums of up to millions of 32-bit contributions in the order the atomics
    # land. Two runs of one build differ by 2e-8 in an image, and by up to
    # 2e-5 in a gradient, whose terms nearly cancel.
    return {"rel": 1e-6 if kind == "image" else 1e-4}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    """64-bit results. Gradients have None: the boundary terms' samples are
    accepted or refused by 32-bit comparisons (which edge, which side, which
    hit), so there is no 64-bit value that belongs to the same samples. Images
    have one where the scene is diffuse and small enough to trace by brute
    force; a path whose 32-bit decision falls the other way is rare there."""
    kind = case["kind"]
    if kind == "configure":
        st = prepare(case, seed)
        return _geometry64(st["scene"].spec, st["V"].double())
    if kind == "rays":
        st = prepare(case, seed)
        if case["n"] * case["tris"] > 2e11:
            return None
        V = st["scene"]._raw_positions.double()
        F = _faces(st["scene"].spec)
        org, d, tmin, tmax = (x.double() for x in st["rays"])
        tri, u, v, t = _closest64(V, F, org, d, 1e-2)
        return {"tri": tri.int(), "u": u, "v": v, "t": t, "visible": (tri < 0).int()}
    if kind in ("image", "step") and case["scene"] == "ico" and case["w"] * case["h"] * case["spp"] <= 1 << 21:
        st = prepare(case, seed)
        sc = st["scene"]
        V = st["V"].detach() if kind == "step" else sc._raw_positions
        img = _render64(sc.spec, V.double(), case, st["options"].seed)
        if kind == "image":
            return img
        return {"image": img, "loss": 0.5 * (img - st["target"].double()).square().sum(), "positions": None}
    return None


def _faces(spec):
    return torch.as_tensor(spec.arrays()["indices"], device="cuda").long()


def _geometry64(spec, V):
    F = _faces(spec)
    c = torch.linalg.cross(V[F[:, 1]] - V[F[:, 0]], V[F[:, 2]] - V[F[:, 0]])
    length = c.norm(dim=1, keepdim=True)
    fn = c / length
    vn = torch.zeros_like(V).index_add_(0, F.reshape(-1), fn.repeat_interleave(3, 0))
    return {"positions": V, "face_normals": fn, "areas": 0.5 * length[:, 0],
            "vertex_normals": vn / vn.norm(dim=1, keepdim=True)}


def _closest64(V, F, org, d, tmin, tmax=None):
    """Closest hit by brute force: (triangle or -1, u, v, t); misses as the
    library reports them (u = v = 0, t = -1)."""
    A, B, C = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    e1, e2 = B - A, C - A
    N = torch.linalg.cross(e1, e2)
    n = len(org)
    tri = torch.full((n,), -1, dtype=torch.long, device=V.device)
    u, v, t = torch.zeros(n, device=V.device).double(), torch.zeros(n, device=V.device).double(), -torch.ones(
        n, device=V.device).double()
    step = max(1, int(1.5e8 // len(F)))
    # det = -d.N, u = (d x e2).(o - A) / det and so on, as matrix products:
    # (o - A).(d x e2) = (o x d).e2 - d.(e2 x A) ... with m = o x d
    e2xA, e1xA, NA = torch.linalg.cross(e2, A), torch.linalg.cross(e1, A), (N * A).sum(1)
    for i in range(0, n, step):
        o, r = org[i:i + step], d[i:i + step]
        m = torch.linalg.cross(o, r)
        det = -(r @ N.T)
        inv = 1.0 / det
        uu = (m @ e2.T - r @ e2xA.T) * inv
        vv = -(m @ e1.T - r @ e1xA.T) * inv
        tt = (o @ N.T - NA) * inv
        ok = (uu >= 0) & (vv >= 0) & (uu + vv <= 1) & (tt > tmin)
        if tmax is not None:
            ok &= tt < tmax[i:i + step, None]
        tt = torch.where(ok, tt, torch.inf)
        best, k = tt.min(1)
        hit = best < torch.inf
        j = k[:, None]
        tri[i:i + step] = torch.where(hit, k, -1)
        u[i:i + step] = torch.where(hit, uu.gather(1, j)[:, 0], 0.0)
        v[i:i + step] = torch.where(hit, vv.gather(1, j)[:, 0], 0.0)
        t[i:i + step] = torch.where(hit, best, -1.0)
    return tri, u, v, t


def _mix32(x):
    m = 0xFFFFFFFF
    x = x ^ (x >> 16)
    x = (x * 0x7FEB352D) & m
    x = x ^ (x >> 15)
    x = (x * 0x846CA68B) & m
    return x ^ (x >> 16)


def _uniform(seed, term, dim, slot):
    """The renderer's counter-based uniform sample of (seed, term, dim, slot)."""
    def one(x):
        return int(_mix32(torch.tensor(x & 0xFFFFFFFF, dtype=torch.int64)))

    s = one(seed * 0x9E3779B9 + 0x632BE5AB)
    s = one(s ^ ((term * 0x85EBCA6B + 0x1B873593) & 0xFFFFFFFF))
    s = one(s ^ ((dim * 0xC2B2AE35 + 0x27D4EB2F) & 0xFFFFFFFF))
    h = _mix32(s ^ _mix32((slot + 0x165667B1) & 0xFFFFFFFF))
    return ((h >> 9).double() + 0.5) / 8388608.0


def _render64(spec, V, case, seed):
    """The diffuse path tracer (next-event estimation with the power
    heuristic, box filter) in float64, by brute-force ray queries."""
    dev = V.device
    a = spec.arrays()
    F = _faces(spec)
    g = _geometry64(spec, V)
    mesh = torch.as_tensor(a["triangle_mesh"], device=dev).long()
    smooth = torch.as_tensor(a["mesh_smooth"], device=dev).bool()[mesh]
    albedo = torch.tensor([spec.bsdfs[m.bsdf].albedo for m in spec.meshes], device=dev).double()[mesh]
    light = torch.as_tensor(a["mesh_light"], device=dev).long()[mesh]
    Le = torch.tensor(spec.lights, device=dev).double()
    lt = torch.nonzero(light >= 0)[:, 0]
    lum = Le[light[lt]] @ torch.tensor([0.212671, 0.715160, 0.072169], device=dev).double()
    func = lum * g["areas"][lt]
    cdf = func.cumsum(0) / func.sum()
    pdf_of = torch.zeros(len(F), device=dev).double()
    pdf_of[lt] = func / func.sum() / g["areas"][lt]
    w, h, spp, depth = case["w"], case["h"], case["spp"], case["depth"]
    cam = spec.cameras[0]
    pos = torch.tensor(cam.pos, device=dev).double()
    slot = torch.arange(w * h * spp, device=dev)
    pix = slot % (w * h)
    stream = (seed * 1000003) & 0xFFFFFFFF

    def S(dim):
        return _uniform(stream, 0, dim, slot)

    def bary(tri, u, v, x):
        f = F[tri]
        return x[f[:, 0]] * (1 - u - v)[:, None] + x[f[:, 1]] * u[:, None] + x[f[:, 2]] * v[:, None]

    def frame(n):
        c = n[:, 0].abs() > n[:, 1].abs()
        z = torch.zeros_like(n[:, 0])
        i0 = (n[:, 0] ** 2 + n[:, 2] ** 2).clamp_min(1e-3).rsqrt()
        i1 = (n[:, 1] ** 2 + n[:, 2] ** 2).clamp_min(1e-3).rsqrt()
        t = torch.where(c[:, None], torch.stack([-n[:, 2] * i0, z, n[:, 0] * i0], 1),
                        torch.stack([z, n[:, 2] * i1, -n[:, 1] * i1], 1))
        return t, torch.linalg.cross(n, t)

    def dot(x, y):
        return (x * y).sum(1)

    # raster x and y both run against the camera axes (right = up x forward)
    fwd = torch.tensor(cam.target, device=dev).double() - pos
    fwd = fwd / fwd.norm()
    right = torch.linalg.cross(torch.tensor(cam.up, device=dev).double(), fwd)
    right = right / right.norm()
    up = torch.linalg.cross(fwd, right)
    half = math.tan(math.radians(cam.fov) / 2)
    sx = 1 - 2 * ((pix % w) + S(0)) / w
    sy = 1 - 2 * ((pix // w) + S(1)) / h
    d = right * (sx * half * w / h)[:, None] + up * (sy * half)[:, None] + fwd
    d = d / d.norm(dim=1, keepdim=True)
    img = torch.zeros(w * h, 3, device=dev).double()
    tri, u, v, t = _closest64(V, F, pos.expand(len(d), 3), d, 1e-2)
    T = torch.ones(len(slot), 3, device=dev).double()
    hit = tri >= 0
    slot, pix, tri, u, v, d, T = (x[hit] for x in (slot, pix, tri, u, v, d, T))
    x = bary(tri, u, v, V)
    ng = g["face_normals"][tri]
    emit = torch.where(((light[tri] >= 0) & (dot(-d, ng) > 0))[:, None], Le[light[tri].clamp_min(0)], 0.0)
    img.index_add_(0, pix, emit)
    for b in range(depth):
        if not len(slot):
            break
        ns = torch.where(smooth[tri][:, None], bary(tri, u, v, g["vertex_normals"]), ng)
        kd = albedo[tri]
        front = dot(ns, -d) > 0
        # next-event estimation
        l0, l1 = S(2 + 5 * b), S(3 + 5 * b)
        e = torch.searchsorted(cdf, l0).clamp_max(len(lt) - 1)
        prev = torch.where(e > 0, cdf[(e - 1).clamp_min(0)], 0.0)
        r = ((l0 - prev) / (cdf[e] - prev)).sqrt()
        y = bary(lt[e], 1 - r, r * l1, V)
        lpdf = pdf_of[lt[e]]
        nl = g["face_normals"][lt[e]]
        wi = y - x
        dist = wi.norm(dim=1)
        wi = wi / dist[:, None]
        cs = dot(ns, wi)
        ok = (dist > 1e-2) & (cs.abs() > 1e-8) & (cs * dot(ng, wi) > 0) & front & (cs > 0) & (dot(-wi, nl) > 0)
        blocked = torch.zeros_like(ok)
        k = torch.nonzero(ok)[:, 0]
        blocked[k] = _closest64(V, F, x[k], wi[k], 1e-2, dist[k] - 1e-2)[0] >= 0
        ok &= ~blocked
        G = dot(nl, wi).abs() / dist ** 2
        bp = cs.abs() / math.pi * G
        mis = lpdf ** 2 / (lpdf ** 2 + bp ** 2)
        c = T * kd / math.pi * (cs.abs() * G / lpdf * mis)[:, None] * Le[light[lt[e]]]
        img.index_add_(0, pix, torch.where(ok[:, None], c, 0.0))
        # cosine-weighted continuation
        r1, r2 = 2 * S(4 + 5 * b) - 1, 2 * S(5 + 5 * b) - 1
        first = r1 ** 2 > r2 ** 2
        rad = torch.where(first, r1, r2)
        phi = torch.where(first, math.pi / 4 * (r2 / r1), math.pi / 2 - math.pi / 4 * (r1 / r2))
        lx, ly = rad * phi.cos(), rad * phi.sin()
        lz = (1 - lx ** 2 - ly ** 2).clamp_min(1e-4).sqrt()
        tx, ty = frame(ns)
        wi = tx * lx[:, None] + ty * ly[:, None] + ns * lz[:, None]
        pdf = lz / math.pi
        ok = front & (dot(ns, wi) > 1e-8) & (dot(ng, wi) > 1e-8)
        keep = torch.nonzero(ok)[:, 0]
        tri2, u2, v2, _ = _closest64(V, F, x[keep], wi[keep], 1e-2)
        keep, tri2, u2, v2 = (q[tri2 >= 0] for q in (keep, tri2, u2, v2))
        xn = bary(tri2, u2, v2, V)
        ngn = g["face_normals"][tri2]
        dn = xn - x[keep]
        dist2 = (dn ** 2).sum(1)
        dn = dn / dist2.sqrt()[:, None]
        G = dot(ngn, dn).abs() / dist2
        bv = kd[keep] / math.pi * (dot(ns[keep], dn).abs() * (dot(ns[keep], dn) > 0))[:, None]
        Tn = T[keep] * bv * (G / (pdf[keep] * G))[:, None]
        pp, pl = pdf[keep] * G, pdf_of[tri2]
        lit = (light[tri2] >= 0) & (dot(-dn, ngn) > 0)
        c = Tn * Le[light[tri2].clamp_min(0)] * (pp ** 2 / (pp ** 2 + pl ** 2))[:, None]
        slot, pix = slot[keep], pix[keep]
        img.index_add_(0, pix, torch.where(lit[:, None], c, 0.0))
        tri, u, v, x, ng, d, T = tri2, u2, v2, xn, ngn, dn, Tn
    return (img / spp).reshape(h, w, 3)
