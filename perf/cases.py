"""The work the framework is measured on, as its users call it.

Each case is one call sequence through the public entry points
(``pathguidingdissertation_gb300.api`` and, for ray batches that already live
on the GPU, the C ABI's ``_device`` calls):

* ``render``  progressive path tracing: clear, n samples per pixel in one
  call or frame by frame, read the film (what ``RayTracer.render`` /
  ``saveHDR`` users do);
* ``guided``  the QuadTree guide's recipe: a recorded training render that
  builds the radiance cache, a guided render on it, the film;
* ``learned`` a render guided by the MLP, the film;
* ``mlp``     the learned guide's training gradient on one batch of radiance
  samples;
* ``rays``    closest-hit or any-hit queries of a device ray batch;
* ``bvh``     building a scene's BVH, and the hit distances of a small ray
              batch on it;
* ``cache``   building the radiance cache from records, then k-nearest and
  guide-density queries on it;
* ``diff``    differentiable rendering: the primal image and its adjoint;
* ``batch``   many scenes of uneven size rendered by one batched call.

Geometry is procedural with a fixed seed per size (the generators are memoised
per process, as a program keeps its loaded scene); cameras, random streams,
rays, records, parameters and samples come from the case's seed.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from pathguidingdissertation_gb300 import abi, scenes
from pathguidingdissertation_gb300.api import Batch, Context

FLT_MAX = float(np.finfo(np.float32).max)
MLP_DIMS = [(80, 64), (64, 64), (64, 64), (64, 64), (64, 64), (64, 40)]  # (inputs, outputs) per layer
MODES = {"plain": abi.MODE_PLAIN, "guided_li": abi.MODE_GUIDED_LI}


def listed():
    return [
        # One progressive frame of a thumbnail view with every material kind:
        # the smallest call, an interactive viewer's step.
        dict(name="frame_zoo_64", kind="render", scene="zoo", tris=0, width=64, height=64, frames=1, spp=1, depth=8,
             mode="plain", mitchell=False),
        # The plain path-tracing configuration: the box at 256 x 256, 16 samples, depth 8.
        dict(name="box_256_16spp", kind="render", scene="box", tris=0, width=256, height=256, frames=1, spp=16,
             depth=8, mode="plain", mitchell=False),
        # One full-resolution frame of the 200k-triangle interior: the
        # reference's one-frame-per-call shape.
        dict(name="interior_720p_frame", kind="render", scene="interior", tris=200_000, width=1280, height=720,
             frames=1, spp=1, depth=10, mode="plain", mitchell=False),
        # The same interior rendered offline, 32 samples per pixel in one call: the benchmark's step.
        dict(name="interior_720p_32spp", kind="render", scene="interior", tris=200_000, width=1280, height=720,
             frames=1, spp=32, depth=10, mode="plain", mitchell=False),
        # QuadTree-guided rendering with its training pass, 16,384-record regions (the measured recipe's size).
        dict(name="guided_box_quadtree", kind="guided", tris=20_000, width=400, height=300, train=8, spp=16, depth=8,
             region=16384),
        # A frame batch guided by the network: inference between traversal and shading at every depth.
        dict(name="learned_interior", kind="learned", tris=200_000, width=640, height=360, spp=4, depth=10),
        # One training batch of the learned guide (2^18 samples): forward, loss and backward.
        dict(name="mlp_gradient_262144", kind="mlp", n=262_144),
        # Incoherent secondary rays on two million triangles.
        dict(name="rays_2m_closest", kind="rays", tris=2_000_000, n=4_000_000, any=False),
        # Scene set-up: the BVH of a two-million-triangle terrain (1024 x 1024 heightfield).
        dict(name="bvh_terrain_2m", kind="bvh", grid=1024, n=65_536),
        # The radiance cache of about a million path vertices, and queries on it.
        dict(name="cache_900k", kind="cache", n=900_001, queries=16_384, k=8, region=1024),
        # An optimisation step of inverse rendering on a half-million-triangle terrain.
        dict(name="diff_terrain", kind="diff", grid=512, width=256, height=256, spp=16, depth=8),
        # A batch of uneven scenes, triangle counts log-uniform, resolutions mixed.
        dict(name="batch_12", kind="batch", scenes=12, max_tris=200_000, max_res=512, spp=8, depth=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, sizes log-uniform over the ranges the listed
    cases stand for (odd ones included)."""
    kind = rng.choice(["render", "render", "render", "guided", "learned", "mlp", "rays", "rays", "bvh", "cache",
                       "diff", "batch"])
    if kind == "render":
        scene = rng.choice(["zoo", "box", "interior"])
        width, height = _log(rng, 33, 1280), _log(rng, 33, 720)
        frames = rng.choice([1, 1, 2, 3])
        spp = max(1, min(_log(rng, 1, 32), 29_000_000 // (width * height * frames)))
        tris = {"zoo": 0, "box": _log(rng, 36, 500_000), "interior": 200_000}[scene]
        return dict(kind=kind, scene=scene, tris=tris, width=width, height=height, frames=frames, spp=spp,
                    depth=rng.randint(1, 10), mode=rng.choice(["plain", "plain", "plain", "guided_li"]),
                    mitchell=rng.random() < 0.2)
    if kind == "guided":
        return dict(kind=kind, tris=_log(rng, 36, 200_000), width=_log(rng, 100, 640), height=_log(rng, 100, 360),
                    train=rng.randint(2, 8), spp=rng.randint(8, 24), depth=rng.randint(4, 10),
                    region=rng.choice([1024, 4096, 16384]))
    if kind == "learned":
        return dict(kind=kind, tris=200_000, width=_log(rng, 64, 640), height=_log(rng, 64, 360),
                    spp=rng.randint(1, 4), depth=rng.randint(2, 10))
    if kind == "mlp":
        return dict(kind=kind, n=_log(rng, 1_000, 262_144))
    if kind == "rays":
        return dict(kind=kind, tris=_log(rng, 1_000, 2_000_000), n=_log(rng, 1_000, 6_000_000),
                    any=rng.random() < 0.5)
    if kind == "bvh":
        return dict(kind=kind, grid=_log(rng, 24, 1000), n=_log(rng, 1_000, 65_536))
    if kind == "cache":
        return dict(kind=kind, n=_log(rng, 1_000, 2_000_000), queries=_log(rng, 100, 16_384), k=rng.randint(1, 32),
                    region=rng.choice([1024, 4096, 16384]))
    if kind == "diff":
        return dict(kind=kind, grid=_log(rng, 48, 700), width=_log(rng, 64, 400), height=_log(rng, 64, 400),
                    spp=rng.randint(2, 16), depth=rng.randint(2, 10))
    return dict(kind=kind, scenes=rng.randint(2, 16), max_tris=_log(rng, 1_000, 200_000),
                max_res=rng.choice([128, 256, 512]), spp=rng.randint(1, 12), depth=rng.randint(3, 8))


# ---- inputs ------------------------------------------------------------------------


@functools.lru_cache(maxsize=8)
def _geometry(scene, tris):
    if scene == "interior":
        # The furniture stands a millimetre off the floor: where a box's
        # bottom lies in the floor's plane, the hit is whichever triangle the
        # tree's leaf order gives first.
        g = scenes.interior(target_tris=tris)
        g.triangles["v"]["p"][..., 1] += np.where(g.triangles["material"] > 2, np.float32(1e-3), np.float32(0))[:, None]
        return g
    if scene == "zoo":
        return scenes.material_zoo(env=True)
    if scene == "terrain":
        return scenes.terrain(tris)
    return scenes.cornell_box(target_tris=tris if tris > 36 else None)


@functools.lru_cache(maxsize=4)
def _soup(tris):
    return scenes.triangle_soup(tris, seed=3, extent=10.0, size=max(0.02, 6.0 / tris ** (1.0 / 3.0)))


def _scene(scene, tris, width, height, rng):
    """The scene seen by a slightly moved camera (a user's viewpoint)."""
    g = _geometry(scene, tris)
    cam = dict(g.camera, width=width, height=height)
    cam["from_"] = tuple(float(x) for x in np.asarray(cam["from_"]) + rng.uniform(-0.05, 0.05, 3))
    return scenes.SceneDesc(g.triangles, g.materials, cam, env=g.env, textures=g.textures, name=g.name)


def _context(desc):
    """A scene with its tree in hand, as a program that keeps built trees
    imports it: every leaf's triangles in ascending order (the builder leaves
    their order open, and a ray through a shared edge hits the first one)."""
    ctx = Context(0)
    ctx.upload(desc)
    ctx.bvh_build()
    nodes, idx = ctx.bvh_export()
    starts = np.sort(nodes["left_first"][nodes["used"] > 0])
    leaf = np.searchsorted(starts, np.arange(len(idx)), side="right").astype(np.int64)
    idx = (np.sort((leaf << 32) | idx.astype(np.int64)) & 0x7FFFFFFF).astype(np.int32)
    ctx.bvh_import(nodes, idx)
    return ctx


def _records(n, rng):
    """Path vertices on the surfaces of a room: positions on six walls and a
    few objects, directions about the normals, heavy-tailed radiance."""
    r = np.zeros(n, abi.PATH_VERTEX)
    half = np.array([4.0, 2.0, 3.0])
    pos = rng.uniform(-1.0, 1.0, (n, 3)) * half
    axis = rng.integers(0, 3, n)
    side = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    wall = rng.random(n) < 0.6
    rows = np.arange(n)
    pos[rows[wall], axis[wall]] = (side * half[axis])[wall] * (1.0 - 1e-3 * rng.random(n)[wall])
    normal = np.zeros((n, 3))
    normal[rows, axis] = -side
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d = normal + 0.98 * d
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r["position"] = pos
    r["normal"] = normal
    r["wi"] = d
    r["Li"] = rng.lognormal(-0.5, 1.0, (n, 1)) * rng.uniform(0.5, 1.0, (n, 3))
    return r


def _unit(rng, n):
    v = rng.standard_normal((n, 3))
    return (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)


def _mlp_inputs(case, seed):
    rng = np.random.default_rng(seed)
    lo, hi = np.array([-4.0, 0.0, -3.0], np.float32), np.array([4.0, 4.0, 3.0], np.float32)
    params = np.concatenate([np.concatenate([rng.uniform(-1, 1, n * k) * math.sqrt(6.0 / k) * (0.5 if n == 40 else 1.0),
                                             rng.uniform(-0.1, 0.1, n)]) for k, n in MLP_DIMS]).astype(np.float32)
    s = np.zeros(case["n"], abi.RADIANCE_SAMPLE)
    s["position"] = rng.uniform(lo, hi, (case["n"], 3))
    s["normal"], s["wo"], s["wi"] = _unit(rng, case["n"]), _unit(rng, case["n"]), _unit(rng, case["n"])
    s["weight"] = rng.lognormal(-1.0, 1.0, case["n"])
    return lo, hi, params, s


def _device_rays(n, lo, hi, tmax, seed):
    """Origins in the inner 90 % of the box, uniform directions (32-byte pgx_ray rows)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo = torch.tensor(lo, dtype=torch.float32, device="cuda")
    hi = torch.tensor(hi, dtype=torch.float32, device="cuda")
    u = torch.rand((n, 3), generator=g, device="cuda")
    d = torch.randn((n, 3), generator=g, device="cuda")
    rays = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
    rays[:, :3] = 0.5 * (lo + hi) + (u - 0.5) * (hi - lo) * 0.9
    rays[:, 3] = tmax
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    torch.cuda.synchronize()
    return rays


def _batch_scenes(case, rng):
    """Tessellated boxes, triangle counts log-uniform, three resolutions."""
    out = []
    geo = np.random.default_rng(11)
    for i in range(case["scenes"]):
        tris = int(math.exp(geo.uniform(math.log(36), math.log(case["max_tris"]))))
        res = case["max_res"] >> int(geo.integers(0, 3))
        out.append(_scene("box", tris, res, max(16, res - 7 * (i % 3)), rng))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = dict(case, seed=int(seed))
    if kind == "render":
        s["ctx"] = _context(_scene(case["scene"], case["tris"], case["width"], case["height"], rng))
    elif kind == "guided":
        s["ctx"] = _context(_scene("box", case["tris"], case["width"], case["height"], rng))
        s["ctx"].guide_configure(region_records=case["region"], clamp_median=20.0, glossy_alpha=2.0)
    elif kind == "learned":
        s["ctx"] = _context(_scene("interior", case["tris"], case["width"], case["height"], rng))
        s["ctx"].mlp_init(seed=1 + int(seed) % 1000)
    elif kind == "mlp":
        lo, hi, params, s["samples"] = _mlp_inputs(case, seed)
        s["ctx"] = Context(0)
        s["ctx"].mlp_init(1, lo, hi)
        s["ctx"].mlp_set_params(params)
    elif kind == "rays":
        desc = _soup(case["tris"])
        lo, hi = desc.bounds()
        s["ctx"] = _context(desc)
        s["rays"] = _device_rays(case["n"], lo, hi, 4.0 if case["any"] else FLT_MAX, seed)
        s["out"] = torch.zeros(case["n"], dtype=torch.uint8, device="cuda") if case["any"] else \
            torch.zeros((case["n"], 4), dtype=torch.int32, device="cuda")
    elif kind == "bvh":
        desc = _scene("terrain", case["grid"], 512, 512, rng)
        s["ctx"] = Context(0)
        s["ctx"].upload(desc)
        lo, hi = desc.bounds()
        s["rays"] = _device_rays(case["n"], lo, hi, FLT_MAX, seed)
        s["out"] = torch.zeros((case["n"], 4), dtype=torch.int32, device="cuda")
    elif kind == "cache":
        s["records"] = _records(case["n"], rng)
        s["queries"] = s["records"]["position"][rng.integers(0, case["n"], case["queries"])] + \
            rng.normal(0.0, 0.02, (case["queries"], 3)).astype(np.float32)
        s["dirs"] = _unit(rng, case["queries"])
        s["ctx"] = Context(0)
        s["ctx"].guide_configure(region_records=case["region"])
    elif kind == "diff":
        s["ctx"] = _context(_scene("terrain", case["grid"], case["width"], case["height"], rng))
        s["dimg"] = rng.normal(0.0, 0.1, (case["height"], case["width"], 3)).astype(np.float32)
    else:
        s["ctxs"] = [_context(d) for d in _batch_scenes(case, rng)]
        s["batch"] = Batch(s["ctxs"])
    torch.cuda.synchronize()
    return s


# ---- one pass ----------------------------------------------------------------------


def _trace_device(s):
    ctx = s["ctx"]
    fn = ctx.lib.pgx_trace_any_device if s.get("any") else ctx.lib.pgx_trace_closest_device
    ctx.check(fn(ctx.h, C.c_void_p(s["rays"].data_ptr()), s["n"], C.c_void_p(s["out"].data_ptr()), None))
    if s.get("any"):
        return s["out"]
    return {"id": s["out"][:, 0], "tuv": s["out"][:, 1:].view(torch.float32)}


def run(state):
    s = state
    kind = s["kind"]
    if kind == "render":
        ctx = s["ctx"]
        ctx.clear()
        for _ in range(s["frames"]):
            ctx.render(s["spp"], mode=MODES[s["mode"]], seed=s["seed"] + 1, max_depth=s["depth"],
                       mitchell=s["mitchell"])
        return ctx.film()[0]
    if kind == "guided":
        ctx = s["ctx"]
        ctx.clear()
        ctx.render(s["train"], mode=abi.MODE_PLAIN, seed=s["seed"] + 1, max_depth=s["depth"], record_paths=s["train"])
        ctx.render(s["spp"], mode=abi.MODE_GUIDED_QUADTREE, seed=s["seed"] + 2, max_depth=s["depth"],
                   guide_fraction=0.7)
        return ctx.film()[0]
    if kind == "learned":
        ctx = s["ctx"]
        ctx.clear()
        ctx.render(s["spp"], mode=abi.MODE_GUIDED_MLP, seed=s["seed"] + 1, max_depth=s["depth"], guide_fraction=0.75)
        return ctx.film()[0]
    if kind == "mlp":
        grad, loss = s["ctx"].mlp_gradient(s["samples"])
        return {"grad": grad, "loss": loss}
    if kind == "rays":
        return _trace_device(s)
    if kind == "bvh":
        s["ctx"].bvh_build()
        # distances, and the nodes and triangles all rays visited: what the
        # tree determines whatever order its leaves keep their triangles in
        return {"t": _trace_device(s)["tuv"][:, 0], "visits": list(s["ctx"].trace_counters())}
    if kind == "cache":
        ctx = s["ctx"]
        ctx.cache_build(s["records"])
        # the indexes follow the cache's own record order: distances are compared
        return {"d2": ctx.cache_knn(s["queries"], s["k"])[1], "pdf": ctx.guide_pdf(s["queries"], s["dirs"])}
    if kind == "diff":
        ctx = s["ctx"]
        img = ctx.diff_render(s["spp"], seed=s["seed"] + 1, max_depth=s["depth"])
        env, albedo, rough = ctx.diff_adjoint(s["dimg"], s["spp"], seed=s["seed"] + 1, max_depth=s["depth"])
        return {"image": img, "env": env, "albedo": albedo, "roughness": rough}
    for c in s["ctxs"]:
        c.clear()
    s["batch"].render(s["spp"], seed=s["seed"] + 1, max_depth=s["depth"])
    return [c.film()[0] for c in s["ctxs"]]


# ---- what a pass cannot do without ------------------------------------------------------


def _trace_work(rays, tris):
    """One root-to-leaf descent per ray (two 18-operation slab tests a level)
    and one triangle test of about 45 operations."""
    return rays * (math.log2(max(tris, 4)) * 36.0 + 45.0)


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: an
    estimate from the numbers of rays (a path has about two rays per vertex
    and about 2.5 vertices, fewer at small depths), records and samples."""
    kind = case["kind"]
    vertices = min(2.5, 1.0 + case.get("depth", 8) * 0.5)
    if kind in ("render", "guided", "learned"):
        tris = max(case["tris"], 132)
        pix = case["width"] * case["height"]
        paths = pix * (case["spp"] * case.get("frames", 1) + case.get("train", 0))
        flops = _trace_work(2 * vertices * paths, tris) + 300.0 * vertices * paths
        if kind == "learned":
            flops += 48_128.0 * vertices * paths
        return dict(bytes=tris * 240.0 + pix * 12.0, flops=flops)
    if kind == "mlp":
        return dict(bytes=case["n"] * 52.0 + 2 * 24_424 * 4.0, flops=case["n"] * 3 * 2.0 * sum(k * n for k, n in MLP_DIMS))
    if kind == "rays":
        return dict(bytes=case["n"] * (33.0 if case["any"] else 48.0) + case["tris"] * 100.0,
                    flops=_trace_work(case["n"], case["tris"]))
    if kind == "bvh":
        tris = 2 * (case["grid"] - 1) ** 2
        return dict(bytes=tris * (36.0 + 48.0 + 32.0) + case["n"] * 48.0, flops=tris * math.log2(tris) * 20.0)
    if kind == "cache":
        return dict(bytes=case["n"] * (48.0 + 48.0 + 10.0), flops=case["n"] * math.log2(case["n"]) * 10.0 +
                    case["queries"] * (math.log2(case["n"]) * 20.0 + case["k"] * 50.0))
    if kind == "diff":
        tris = 2 * (case["grid"] - 1) ** 2
        paths = case["width"] * case["height"] * case["spp"]
        return dict(bytes=tris * 240.0 + case["width"] * case["height"] * 36.0 + 512 * 256 * 24.0,
                    flops=2 * (_trace_work(2 * vertices * paths, tris) + 300.0 * vertices * paths))
    geo = np.random.default_rng(11)
    total, paths = 0.0, 0.0
    for i in range(case["scenes"]):
        tris = math.exp(geo.uniform(math.log(36), math.log(case["max_tris"])))
        res = case["max_res"] >> int(geo.integers(0, 3))
        pix = res * max(16, res - 7 * (i % 3))
        total += tris * 240.0 + pix * 12.0
        paths += pix * case["spp"]
    return dict(bytes=total, flops=_trace_work(2 * vertices * paths, max(case["max_tris"] // 4, 36)) + 300.0 * vertices * paths)


# ---- outputs in 64 bits ----------------------------------------------------------------


def _exact_mlp(case, seed):
    """Loss and gradient of the mixture network, float64 autograd."""
    lo, hi, params, s = _mlp_inputs(case, seed)
    dev = "cuda"
    p = torch.tensor(params, dtype=torch.float64, device=dev, requires_grad=True)
    t64 = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    lo_t, hi_t = t64(lo), t64(hi)
    wgt_all = t64(s["weight"])
    scale = 1.0 / wgt_all.sum()
    loss_sum = 0.0
    for a in range(0, case["n"], 65_536):
        b = slice(a, a + 65_536)
        x = ((t64(s["position"][b]) - lo_t) / (hi_t - lo_t)).clamp(0.0, 1.0)
        ang = math.pi * x[:, :, None] * torch.tensor([2.0 ** j for j in range(12)], dtype=torch.float64, device=dev)
        enc = torch.stack([ang.sin(), ang.cos()], -1).reshape(len(x), 72)
        h = torch.cat([enc, t64(s["normal"][b]), t64(s["wo"][b]), torch.zeros((len(x), 2), dtype=torch.float64, device=dev)], 1)
        at = 0
        for i, (k, n) in enumerate(MLP_DIMS):
            w, c = p[at:at + n * k].reshape(n, k), p[at + n * k:at + n * k + n]
            at += n * k + n
            h = h @ w.T + c
            if i < len(MLP_DIMS) - 1:
                h = h.relu()
        logw = torch.log_softmax(h[:, :8], 1)
        m = h[:, 8:32].reshape(-1, 8, 3)
        mu = m / m.norm(dim=2, keepdim=True)
        kappa = torch.nn.functional.softplus(h[:, 32:40]) + 0.01
        cos = (mu * t64(s["wi"][b])[:, None, :]).sum(2)
        logv = torch.log(kappa / (2.0 * math.pi * -torch.expm1(-2.0 * kappa))) + kappa * (cos - 1.0)
        loss = -(wgt_all[b] * scale * torch.logsumexp(logw + logv, 1)).sum()
        loss.backward()
        loss_sum += float(loss.detach())
    return {"grad": p.grad.detach(), "loss": loss_sum}


def _exact_cache(case, seed):
    """Squared distances of the k nearest records by brute force; the guide's
    density has no closed form to state."""
    rng = np.random.default_rng(seed)
    rec = _records(case["n"], rng)
    q = rec["position"][rng.integers(0, case["n"], case["queries"])] + \
        rng.normal(0.0, 0.02, (case["queries"], 3)).astype(np.float32)
    p = torch.tensor(np.ascontiguousarray(rec["position"]), device="cuda").double()
    qd = torch.tensor(np.ascontiguousarray(q), device="cuda").double()
    out = torch.full((case["queries"], case["k"]), math.inf, dtype=torch.float64, device="cuda")
    step = max(1, 40_000_000 // case["n"])
    for a in range(0, case["queries"], step):
        d2 = torch.zeros((len(qd[a:a + step]), case["n"]), dtype=torch.float64, device="cuda")
        for c in range(3):
            d2 += (qd[a:a + step, c:c + 1] - p[None, :, c]) ** 2
        k = min(case["k"], case["n"])
        out[a:a + step, :k] = torch.topk(d2, k, dim=1, largest=False, sorted=True).values
    return {"d2": out, "pdf": None}


def exact(case, seed):
    """Paths, hits and their sums are float32 decisions with no 64-bit value
    to state; the network's gradient and the distances have one."""
    if case["kind"] == "mlp":
        return _exact_mlp(case, seed)
    if case["kind"] == "cache":
        return _exact_cache(case, seed)
    return None
