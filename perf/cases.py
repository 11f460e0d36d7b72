"""Performance cases of the renderer: what users of the package have it do.

Every case goes through the public entry points (``BVH.build_device``,
``Accelerator.trace_*``, the integrators, ``BatchRenderer``, ``DiffRenderer``,
``postprocess``) on seeded synthetic inputs: triangle soups with camera,
bounce and shadow rays, Cornell-style boxes, a procedural city, request
batches and the inverse-rendering scene of the benchmark.  A case is a dict
of plain values; its ``kind`` selects the path.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from zillumgl_gb300 import BVH
from zillumgl_gb300.image import TONE_FILMIC, postprocess
from zillumgl_gb300.scene import BatchRenderer, DiffRenderer, LightIntegrator, PathIntegrator, Scene, TripleIntegrator
from zillumgl_gb300.synthetic import (city_scene, cornell_scene, diff_scene, material_zoo_scene, sphere_box_scene,
                                      textured_scene)

DEV = "cuda"


def listed():
    return [
        # A handful of picking or collision probes against a small mesh: launch latency.
        dict(name="probe_rays", kind="trace", query="closest", family="bounce", tris=2048, rays=997),
        # First hits of a camera over a mid-size mesh (previews, G-buffers): coherent rays.
        dict(name="primary_1m", kind="trace", query="closest", family="primary", tris=1 << 20, rays=1500 * 1100),
        # One diffuse bounce over a mesh whose tables outgrow the L2 cache.
        dict(name="bounce_4m", kind="trace", query="closest", family="bounce", tris=1 << 22, rays=1 << 22),
        # Ambient-occlusion / shadow rays over the largest mesh of the benchmark, full launch.
        dict(name="shadow_16m", kind="trace", query="any", family="bounce", tris=1 << 24, rays=1 << 24),
        # Animated geometry: rebuild the accelerator from device arrays, then cast the camera rays.
        dict(name="rebuild_2m", kind="rebuild", tris=2000003, rays=1024 * 1024),
        # An interactive viewer: one progressive pass of a small film, read back and tone mapped.
        dict(name="cornell_view", kind="view", base="cornell", width=256, height=256, depth=5),
        # An offline render with every material type, an odd film, all passes in one call.
        dict(name="zoo_16spp", kind="passes", base="zoo", width=251, height=187, depth=6, spp=16),
        # A progressive path-tracing pass of a large scene at full HD (the benchmark's city).
        dict(name="city_path", kind="city", integrator="path", grid=64, spheres=2000, width=1920, height=1080, depth=8),
        # A particle-tracing pass at the default 49,152 light paths.
        dict(name="city_light", kind="city", integrator="light", grid=32, spheres=700, width=480, height=270, depth=8),
        # A pass of the combined camera and light integrator.
        dict(name="city_triple", kind="city", integrator="triple", grid=32, spheres=700, width=960, height=540,
             depth=8),
        # A render service's queue: mixed scenes, films and sample counts in one batch.
        dict(name="batch_12", kind="batch", requests=12, max_tris=500000, max_side=1024, max_spp=32),
        # One step of inverse rendering: image, loss and gradient.
        dict(name="diff_step", kind="diff", width=512, height=512, depth=6, spp=32),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "rebuild", "view", "passes", "city", "city", "batch", "diff"])
    if kind == "trace":
        return dict(kind=kind, query=rng.choice(["closest", "any"]), family=rng.choice(["primary", "bounce"]),
                    tris=_logint(rng, 2048, 1 << 24), rays=_logint(rng, 997, 1 << 24))
    if kind == "rebuild":
        return dict(kind=kind, tris=_logint(rng, 5000, 8 << 20), rays=_logint(rng, 10000, 1 << 21))
    if kind == "view":
        return dict(kind=kind, base=rng.choice(["cornell", "zoo", "textured"]), width=_logint(rng, 64, 1024),
                    height=_logint(rng, 64, 1024), depth=rng.randint(2, 8))
    if kind == "passes":
        return dict(kind=kind, base=rng.choice(["cornell", "zoo", "textured"]), width=_logint(rng, 64, 512),
                    height=_logint(rng, 64, 512), depth=rng.randint(2, 8), spp=rng.randint(2, 32))
    if kind == "city":
        return dict(kind=kind, integrator=rng.choice(["path", "light", "triple"]), grid=_logint(rng, 8, 48),
                    spheres=_logint(rng, 50, 1500), width=_logint(rng, 200, 1600), height=_logint(rng, 120, 900),
                    depth=rng.randint(3, 8))
    if kind == "batch":
        return dict(kind=kind, requests=rng.randint(3, 12), max_tris=_logint(rng, 10000, 500000),
                    max_side=_logint(rng, 200, 800), max_spp=rng.randint(4, 24))
    return dict(kind=kind, width=_logint(rng, 64, 512), height=_logint(rng, 64, 512), depth=rng.randint(3, 8),
                spp=rng.randint(2, 32))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _soup(n, seed):
    """n equilateral triangles in the unit cube, edges U(0.001, 0.01), random
    orientation (the benchmark's soup); float32 (3n, 3) vertices and indices."""
    g = _gen(seed)
    c = torch.rand((n, 1, 3), generator=g, device=DEV)
    # smaller meshes get larger triangles, so that as many rays hit as in the 1M one
    grow = max(1.0, (2.0 ** 20 / n) ** (1.0 / 3.0))
    radius = (0.001 + 0.009 * torch.rand((n, 1), generator=g, device=DEV)) * (grow / math.sqrt(3.0))
    u = torch.randn((n, 3), generator=g, device=DEV)
    w = torch.randn((n, 3), generator=g, device=DEV)
    u = u / u.norm(dim=1, keepdim=True)
    w = w - u * (u * w).sum(1, keepdim=True)
    w = w / w.norm(dim=1, keepdim=True)
    v = torch.empty((n, 3, 3), device=DEV)
    for k in range(3):
        a = 2.0 * math.pi * k / 3.0
        v[:, k] = c[:, 0] + radius * (math.cos(a) * u + math.sin(a) * w)
    return v.reshape(-1, 3), torch.arange(3 * n, dtype=torch.int32, device=DEV)


def _primary(n, seed):
    """n pinhole rays, row by row over an image of about 4:3, from one unit in
    front of the cube; the seed moves the camera a little."""
    g = np.random.default_rng(seed)
    pos = torch.tensor([0.5 + g.uniform(-0.1, 0.1), -1.0, 0.5 + g.uniform(-0.1, 0.1)], device=DEV)
    w = max(1, int(math.sqrt(n * 4 / 3)))
    h = -(-n // w)
    i = torch.arange(n, device=DEV)
    t = math.tan(math.radians(22.5))
    x = ((i % w).float() + 0.5) / w * 2 - 1
    y = (torch.div(i, w, rounding_mode="floor").float() + 0.5) / h * 2 - 1
    d = torch.stack([x * (t * w / h), torch.ones_like(x), y * t], 1)
    d = d / d.norm(dim=1, keepdim=True)
    return pos.expand(n, 3).contiguous(), d.contiguous()


def _bounce(acc, vertices, n, seed):
    """Cosine-distributed rays from the camera's hit points; where the camera
    missed, uniform origins in the cube with uniform directions."""
    o, d = _primary(n, seed)
    ids, t = acc.trace_closest(o, d)
    g = _gen(seed + 17)
    r = torch.randn((n, 3), generator=g, device=DEV)
    r = r / r.norm(dim=1, keepdim=True)
    p = torch.rand((n, 3), generator=g, device=DEV)
    hit = (ids >= 0)[:, None]
    tri = vertices.reshape(-1, 3, 3)[ids.clamp(min=0).long()]
    ng = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    ng = ng / ng.norm(dim=1, keepdim=True).clamp(min=1e-20)
    ng = torch.where((ng * d).sum(1, keepdim=True) > 0, -ng, ng)
    out = ng * 1.0001 + r  # the cosine distribution about ng
    out = out / out.norm(dim=1, keepdim=True)
    d2 = torch.where(hit, out, r)
    o2 = torch.where(hit, o + d * t[:, None] + out * 1e-4, p)
    return o2.contiguous(), d2.contiguous()


def _box(case, seed):
    kw = dict(seed=seed, width=case["width"], height=case["height"])
    if case.get("base") == "zoo":
        return material_zoo_scene(**kw)
    if case.get("base") == "textured":
        return textured_scene(**kw)
    return cornell_scene(**kw)


def _city(case, seed):
    return city_scene(seed=seed, width=case["width"], height=case["height"], grid=case["grid"],
                      n_spheres=case["spheres"], env_size=(1024, 512))


def _requests(case, seed):
    """The mix of a request queue: sizes and films spread over their logarithm,
    the same for every seed; the scenes' contents come from the seed."""
    rng = np.random.default_rng(case["requests"])
    out = []
    for r in range(case["requests"]):
        tris = int(np.exp(rng.uniform(np.log(1e3), np.log(case["max_tris"]))))
        side = int(np.exp(rng.uniform(np.log(128), np.log(case["max_side"]))))
        spp = int(rng.integers(4, case["max_spp"] + 1))
        depth = int(rng.integers(4, 9))
        out.append((sphere_box_scene(seed * 1000 + r, tris, side, side), spp, dict(max_depth=depth)))
    return out


# ------------------------------------------------------------------- cases
def prepare(case, seed):
    kind = case["kind"]
    if kind == "trace":
        v, i = _soup(case["tris"], seed)
        acc = BVH(v, i).build_device()
        o, d = _primary(case["rays"], seed) if case["family"] == "primary" else _bounce(acc, v, case["rays"], seed)
        s = dict(case=case, acc=acc, o=o, d=d)
        if case["query"] == "any":
            tm = torch.rand(case["rays"], generator=_gen(seed + 31), device=DEV)
            s["tmax"] = tm + 1.0 if case["family"] == "primary" else tm
        return s
    if kind == "rebuild":
        v, i = _soup(case["tris"], seed)
        o, d = _primary(case["rays"], seed)
        return dict(case=case, v=v, i=i, o=o, d=d)
    if kind in ("view", "passes"):
        W, H = case["width"], case["height"]
        integ = PathIntegrator(Scene(_box(case, seed)), max_depth=case["depth"])
        return dict(case=case, integ=integ, frame=torch.empty((H, W, 4), device=DEV))
    if kind == "city":
        cls = dict(path=PathIntegrator, light=LightIntegrator, triple=TripleIntegrator)[case["integrator"]]
        integ = cls(Scene(_city(case, seed)), max_depth=case["depth"], russian_roulette=1, rr_start_depth=3)
        return dict(case=case, integ=integ, frame=torch.empty((case["height"], case["width"], 4), device=DEV))
    if kind == "batch":
        reqs = []
        for data, spp, params in _requests(case, seed):
            scene = Scene(data)
            W, H = scene.film
            reqs.append((scene, spp, params, torch.zeros((H, W, 4), device=DEV)))
        return dict(case=case, batch=BatchRenderer(reqs), frames=[r[3] for r in reqs])
    W, H = case["width"], case["height"]
    r = DiffRenderer(Scene(diff_scene(seed=seed, width=W, height=H)), case["spp"], max_depth=case["depth"])
    target = torch.rand((H, W, 3), generator=_gen(seed + 5), device=DEV)
    return dict(case=case, diff=r, target=target)


def run(s):
    kind = s["case"]["kind"]
    if kind == "trace":
        if s["case"]["query"] == "any":
            return s["acc"].trace_any(s["o"], s["d"], s["tmax"])
        return s["acc"].trace_closest(s["o"], s["d"])
    if kind == "rebuild":
        acc = BVH(s["v"], s["i"]).build_device()
        return acc.trace_closest(s["o"], s["d"])
    if kind == "view":
        s["integ"].render_one_pass()
        s["integ"].get_frame(s["frame"])
        W, H = s["case"]["width"], s["case"]["height"]
        image = postprocess(s["frame"], W, H, s["integ"].result_scale(), TONE_FILMIC)
        return s["frame"], image
    if kind == "passes":
        s["integ"].render_passes(s["case"]["spp"])
        s["integ"].get_frame(s["frame"])
        return s["frame"]
    if kind == "city":
        s["integ"].render_one_pass()
        s["integ"].get_frame(s["frame"])
        return s["frame"]
    if kind == "batch":
        s["batch"].render()
        return s["frames"]
    image, grad, loss = s["diff"].step_l2(s["target"])
    return image, grad, loss


def work(case):
    """Inputs read once, outputs written once; a ray costs a box test (20
    operations) per level of a binary tree and two triangle tests (50), a path
    vertex two rays and about 500 operations of shading."""
    kind = case["kind"]

    def ray(tris):
        return 40.0 * math.log2(max(tris, 2)) + 100.0

    if kind == "trace":
        io = 32 if case["query"] == "closest" else 29
        return dict(bytes=io * case["rays"] + 36 * case["tris"], flops=case["rays"] * ray(case["tris"]))
    if kind == "rebuild":
        n = case["tris"]
        return dict(bytes=48 * n + 32 * case["rays"], flops=n * 16.0 * math.log2(n) + case["rays"] * ray(n))
    if kind == "batch":
        px = vertices = tris = 0.0
        rng = np.random.default_rng(case["requests"])
        for _ in range(case["requests"]):
            t = int(np.exp(rng.uniform(np.log(1e3), np.log(case["max_tris"]))))
            side = int(np.exp(rng.uniform(np.log(128), np.log(case["max_side"]))))
            spp = int(rng.integers(4, case["max_spp"] + 1))
            depth = int(rng.integers(4, 9))
            px += side * side
            tris += t
            vertices += side * side * spp * 0.5 * depth * (2 * ray(t) + 500)
        return dict(bytes=36 * tris + 16 * px, flops=vertices)
    px = case["width"] * case["height"]
    tris, spp, paths = 2000, case.get("spp", 1), px
    if kind == "city":
        tris = 1920 * case["spheres"] + 12 * case["grid"] ** 2
        paths = 49152 if case["integrator"] == "light" else px
        if case["integrator"] == "triple":
            paths += 2 * 49152
    vertices = paths * spp * 0.5 * case["depth"]
    flops = vertices * (2 * ray(tris) + 500) * (2 if kind == "diff" else 1)
    io = 24 if kind == "diff" else 48 if kind == "view" else 32
    return dict(bytes=36 * tris + io * px, flops=flops)


def exact(case, seed):
    """The small trace cases' hit distances by brute force in 64 bits; the
    other outputs are Monte Carlo images or would take too long."""
    if case["kind"] != "trace" or case["query"] != "closest" or case["tris"] * case["rays"] > 1 << 28:
        return None
    s = prepare(case, seed)
    v, _ = _soup(case["tris"], seed)
    a, b, c = v.double().reshape(-1, 3, 3).unbind(1)
    ab, ac = b - a, c - a
    out = []
    for o, d in zip(s["o"].double().split(4096), s["d"].double().split(4096)):
        best = torch.full((o.shape[0],), 1e8, dtype=torch.float64, device=DEV)
        for lo in range(0, a.shape[0], 1024):
            A, AB, AC = a[lo:lo + 1024], ab[lo:lo + 1024], ac[lo:lo + 1024]
            p = torch.linalg.cross(d[:, None].expand(-1, A.shape[0], -1), AC[None].expand(d.shape[0], -1, -1))
            det = (AB[None] * p).sum(-1)
            ao = o[:, None] - A[None]
            q = torch.linalg.cross(ao, AB[None].expand_as(ao))
            u = (ao * p).sum(-1) / det
            w = (d[:, None] * q).sum(-1) / det
            t = (AC[None] * q).sum(-1) / det
            ok = (det.abs() >= 1e-6) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0)
            best = torch.minimum(best, torch.where(ok, t, torch.full_like(t, 1e8)).min(1).values)
        out.append(best)
    return None, torch.cat(out)
