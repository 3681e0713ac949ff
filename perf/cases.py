"""Measured cases: what a user of the renderer has it do, through the
package's public entry points (``psychopath_cpp_b200.api``).

Three families of use, each over its range of sizes:

* ray streams: ``Tracer.trace_device`` / ``Tracer.trace`` on closest-hit and
  shadow rays, from a few hundred rays of one bucket to millions, on flat,
  patch and instanced scenes, with few or all Intersection fields;
* light samples: ``LightTree.sample`` on scenes of one to 10,000 lights;
* renders: ``PathTraceIntegrator``, ``BatchRenderer`` and ``DiffRenderer``,
  from a thumbnail at one sample per pixel to a 720p frame of the many-light
  scene, over every kind of object, light and closure.

Scenes and rays are made from the seed by the generators of
``psychopath_cpp_b200.scenes`` with the sizes of the repository's benchmark
and tests, or by the ray generators below.  All floats are 32 bits (the
renderer has no other type).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from psychopath_cpp_b200 import api, scenes

# Intersection fields a caller asks for: the hit itself, or all that shading
# needs (what the reference's integrator reads).
HIT_FIELDS = ("hit", "id", "t", "uv")
SHADING_FIELDS = ("hit", "id", "t", "uv", "p", "n", "dpdu", "dpdv", "backfacing", "light_pdf", "offset", "space",
                  "closure", "closure_color")
_TORCH = {np.uint8: torch.uint8, np.uint64: torch.int64, np.float32: torch.float32}


def listed():
    return [
        # one bucket's camera rays against a small flat scene: the smallest
        # call, where launch and latency count
        {"name": "rays_bucket", "path": "trace", "scene": "plain", "prims": 64, "lights": 1, "rays": 1021,
         "fields": "hit", "host": False},
        # the trace microbenchmark of the repository: a 4M-ray stream against
        # a 256x256 bilinear heightfield
        {"name": "rays_heightfield", "path": "trace", "scene": "heightfield", "prims": 256, "lights": 0,
         "rays": 4194304, "fields": "hit", "host": False},
        # an integrator's mixed stream (camera, bounce and shadow rays) against
        # instanced geometry with motion, all the fields shading needs
        {"name": "rays_instanced", "path": "trace", "scene": "many_light", "prims": 800, "lights": 500, "rays": 300007,
         "fields": "shading", "host": False},
        # the drop-in for the reference's Tracer::trace: host arrays in and out
        {"name": "rays_host", "path": "trace", "scene": "flat", "prims": 5000, "lights": 10, "rays": 65536,
         "fields": "shading", "host": True},
        # next-event queries of one bounce against the benchmark's light count
        {"name": "lights_10k", "path": "lights", "prims": 8, "lights": 10000, "queries": 65536},
        # a thumbnail at one sample per pixel and its 8-bit image: what an
        # interactive preview asks for
        {"name": "preview", "path": "render", "scene": "plain", "prims": 64, "lights": 1, "width": 80, "height": 60,
         "spp": 1, "length": 4, "image": True},
        # the plain renderer workload of the repository
        {"name": "render_plain", "path": "render", "scene": "plain", "prims": 64, "lights": 1, "width": 320,
         "height": 240, "spp": 16, "length": 4, "image": False},
        # microfacet closures on most objects, an odd frame
        {"name": "render_gtr", "path": "render", "scene": "gtr", "prims": 24, "lights": 1, "width": 193, "height": 109,
         "spp": 8, "length": 4, "image": False},
        # the largest scene of the batch workload on its own
        {"name": "render_flat_50k", "path": "render", "scene": "flat", "prims": 50000, "lights": 100, "width": 512,
         "height": 384, "spp": 16, "length": 4, "image": False},
        # the headline scene and resolution, at the samples of one progressive
        # pass of its 64
        {"name": "render_many_light", "path": "render", "scene": "many_light", "prims": 2000, "lights": 10000,
         "width": 1280, "height": 720, "spp": 4, "length": 6, "image": False},
        # many small renders of different scenes in one call
        {"name": "batch_small", "path": "batch", "scene": "flat", "renders": 16, "prims": 2000, "lights": 19,
         "width": 192, "height": 160, "spp": 8},
        # one optimisation step: forward render, image loss, adjoint
        {"name": "diff_step", "path": "diff", "scene": "adjoint", "prims": 64, "lights": 8, "width": 256,
         "height": 256, "spp": 32, "length": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["trace", "trace", "trace", "lights", "render", "render", "render", "render", "batch", "diff"])
    if path == "trace":
        scene = rng.choice(["plain", "heightfield", "many_light", "flat", "motion"])
        prims = {"plain": (8, 256), "heightfield": (8, 200), "many_light": (50, 1500), "flat": (20, 20000),
                 "motion": (2, 12)}[scene]
        host = rng.random() < 0.3
        return {"path": path, "scene": scene, "prims": _log(rng, *prims),
                "lights": 0 if scene == "heightfield" else 1 if scene in ("plain", "motion") else _log(rng, 1, 1000),
                "rays": _log(rng, 200, 400000 if host else 2000000), "fields": rng.choice(["hit", "shading"]),
                "host": host}
    if path == "lights":
        return {"path": path, "prims": 8, "lights": _log(rng, 1, 10000), "queries": _log(rng, 200, 400000)}
    if path == "batch":
        return {"path": path, "scene": "flat", "renders": rng.randint(2, 24), "prims": _log(rng, 20, 2000),
                "lights": rng.randint(1, 19), "width": rng.randint(33, 200), "height": rng.randint(33, 160),
                "spp": rng.randint(1, 16)}
    scene = "adjoint" if path == "diff" else rng.choice(["plain", "gtr", "rect", "motion", "flat", "many_light"])
    prims = {"adjoint": (8, 64), "plain": (8, 256), "gtr": (8, 64), "rect": (8, 64), "motion": (2, 12),
             "flat": (20, 50000), "many_light": (50, 2000)}[scene]
    width = _log(rng, 40, 640)
    height = max(17, int(width * rng.uniform(0.5, 1.0)))
    return {"path": path, "scene": scene, "prims": _log(rng, *prims),
            "lights": {"adjoint": 8, "flat": _log(rng, 1, 100), "many_light": _log(rng, 10, 10000)}.get(scene, 1),
            "width": width, "height": height,
            # at most a million paths, so that no drawn frame outweighs the listed ones
            "spp": max(1, min(_log(rng, 1, 32), 1000000 // (width * height))),
            "length": rng.randint(2, 6), "image": False}


# --------------------------------------------------------------------------
# Scenes
# --------------------------------------------------------------------------

def _scene(kind, prims, lights, seed, res=(64, 48), spp=1):
    if kind == "plain":
        return scenes.plain_scene(seed, res=res, spp=spp, n_spheres=prims)
    if kind == "heightfield":
        return scenes.heightfield_scene(prims, seed=seed)
    if kind == "flat":
        return scenes.batch_scene(seed, res, spp, prims, lights)
    if kind == "motion":
        return scenes.motion_patch_scene(seed, res=res, spp=spp, n=prims)
    if kind == "gtr":
        return scenes.gtr_scene(seed, res=res, spp=spp, n_spheres=prims)
    if kind == "rect":
        return scenes.rect_light_scene(seed, res=res, spp=spp, n_spheres=prims)
    if kind == "adjoint":
        return scenes.adjoint_scene(seed, res=res, spp=spp, n_spheres=prims, n_lights=lights)
    # the many-light scene keeps its proportions: a group of instanced spheres
    # for every four ground patches
    return scenes.many_light_scene(seed, res=res, spp=spp, n_patches=prims, n_groups=max(5, prims // 4),
                                   n_lights=lights)


# Where each scene's geometry lies, and where its camera looks from.
def _extent(kind, prims):
    if kind == "heightfield":
        return (0.0, 0.0, -0.5), (float(prims), float(prims), 4.0), (prims / 2, -prims / 2, prims / 2)
    if kind == "many_light":
        side = math.sqrt(prims * 1.25) / 2
        return (-side, -side, -0.5), (side, side, 5.0), (0.0, -32.0, 14.0)
    return (-5.0, -5.0, 0.0), (5.0, 5.0, 2.0), (0.0, -15.0, 7.0)


# --------------------------------------------------------------------------
# Ray streams
# --------------------------------------------------------------------------

def _heightfield_rays(n, size, g):
    """The stream of scenes.heightfield_rays (cosine about -z from a box above
    the field, constant ray width, half ordered and half shuffled), drawn on
    the device."""
    dev = g.device
    ox, oy = torch.rand(n, generator=g, device=dev) * size, torch.rand(n, generator=g, device=dev) * size
    oz = 2.0 + 2.0 * torch.rand(n, generator=g, device=dev)
    u, phi = torch.rand(n, generator=g, device=dev), 2 * math.pi * torch.rand(n, generator=g, device=dev)
    r = u.sqrt()
    d = torch.stack([r * phi.cos(), r * phi.sin(), -(1 - u).clamp_min(0).sqrt()], 1)
    o = torch.stack([ox, oy, oz], 1)
    h = n // 2
    # the ordered half: by direction quadrant, then along a Z-curve of 1x1 cells
    cell = torch.zeros(h, dtype=torch.int64, device=dev)
    for b in range(9):
        cell |= ((ox[:h].long() >> b) & 1) << (2 * b)
        cell |= ((oy[:h].long() >> b) & 1) << (2 * b + 1)
    order = (((d[:h, 0] > 0).long() + 2 * (d[:h, 1] > 0).long()) << 20 | cell).argsort(stable=True)
    o[:h], d[:h] = o[order], d[order]
    z = torch.zeros(n, 3, device=dev)
    wx, wy = z.clone(), z.clone()
    wx[:, 0], wy[:, 1] = 0.6, 0.6
    return {"o": o, "d": d, "odx": wx, "ody": wy, "ddx": z, "ddy": z.clone(),
            "time": torch.zeros(n, device=dev), "type": torch.ones(n, dtype=torch.int16, device=dev)}


def _mixed_rays(n, lo, hi, eye, g):
    """An integrator's stream: the first half camera rays in scanline order,
    a quarter bounce rays (random directions, the wide direction
    differentials of a diffuse bounce), a quarter shadow rays (type 32, the
    direction reaching to the light)."""
    dev = g.device
    lo, hi, eye = (torch.tensor(v, dtype=torch.float32, device=dev) for v in (lo, hi, eye))
    target = lo + (hi - lo) * torch.rand(n, 3, generator=g, device=dev)
    start = lo + (hi - lo) * torch.rand(n, 3, generator=g, device=dev)
    cam = n // 2
    shadow = n - n // 4
    # camera rays: a jittered grid on the ground plane, row by row
    side = max(1, int(math.sqrt(cam)))
    k = torch.arange(cam, device=dev)
    grid = torch.stack([(k % side).float(), (k // side).float()], 1) + torch.rand(cam, 2, generator=g, device=dev)
    target[:cam, :2] = lo[:2] + (hi - lo)[:2] * (grid / (side + 1))
    target[:cam, 2] = lo[2]
    start[:cam] = eye
    d = target - start
    aim = torch.randn(n, 3, generator=g, device=dev)
    d[cam:shadow] = aim[cam:shadow]
    d[shadow:, 2] += 6.0  # towards the lights above
    unit = d / d.norm(dim=1, keepdim=True).clamp_min(1e-6)
    d[:shadow] = unit[:shadow]
    x = torch.cross(unit, torch.tensor([[0.3, 0.5, 0.8]], device=dev).expand_as(unit), dim=1)
    x = x / x.norm(dim=1, keepdim=True).clamp_min(1e-6)
    y = torch.cross(unit, x, dim=1)
    spread = torch.full((n, 1), 0.15, device=dev)
    spread[:cam] = 0.002
    width = torch.full((n, 1), 0.02, device=dev)
    width[:cam] = 0.0
    kind = torch.ones(n, dtype=torch.int16, device=dev)
    kind[shadow:] = 32
    return {"o": start, "d": d, "odx": x * width, "ody": y * width, "ddx": x * spread, "ddy": y * spread,
            "time": torch.rand(n, generator=g, device=dev), "type": kind}


# --------------------------------------------------------------------------
# prepare / run
# --------------------------------------------------------------------------

def _context(scene):
    ctx = api.Context(0)
    ctx.upload(scene)
    return ctx


def _rays(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["scene"] == "heightfield":
        return _heightfield_rays(case["rays"], case["prims"], g)
    return _mixed_rays(case["rays"], *_extent(case["scene"], case["prims"]), g)


def _light_queries(case, seed):
    """Rows n u v pos nor d wavelength time pad, as LightTree.sample takes
    them: points near the ground, normals about +z, incoming directions from
    above."""
    rng = np.random.default_rng(seed)
    k = case["queries"]
    q = np.zeros((k, 15), np.float32)
    q[:, 0:3] = rng.random((k, 3))
    q[:, 3:6] = rng.uniform((-4.5, -4.5, 0.0), (4.5, 4.5, 1.5), (k, 3))
    nor = rng.normal(0.0, 0.4, (k, 3)) + (0.0, 0.0, 1.0)
    q[:, 6:9] = nor / np.linalg.norm(nor, axis=1, keepdims=True)
    d = rng.normal(0.0, 0.5, (k, 3)) + (0.0, 0.0, -1.0)
    q[:, 9:12] = d / np.linalg.norm(d, axis=1, keepdims=True)
    q[:, 12] = rng.uniform(380.0, 700.0, k)
    return q


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    path = case["path"]
    if path == "trace":
        ctx = _context(_scene(case["scene"], case["prims"], case["lights"], seed))
        rays = _rays(case, seed)
        fields = SHADING_FIELDS if case["fields"] == "shading" else HIT_FIELDS
        if case["host"]:
            rays = {k: v.cpu().numpy() for k, v in rays.items()}
            hits = None
        else:
            rays = {k: v.contiguous() for k, v in rays.items()}
            hits = {}
            for f in fields:
                dtype, width = api.HIT_FIELDS[f]
                hits[f] = torch.zeros((case["rays"], width) if width > 1 else case["rays"], dtype=_TORCH[dtype],
                                      device=dev)
        return {"path": path, "tracer": api.Tracer(ctx), "rays": rays, "hits": hits, "fields": fields}
    if path == "lights":
        return {"path": path, "tree": api.LightTree(_context(_scene("flat", case["prims"], case["lights"], seed))),
                "queries": _light_queries(case, seed)}
    if path == "batch":
        # renders of differing sizes and scenes, at most the case's own; the
        # frames are the job's, the scenes in them the seed's
        rng = np.random.default_rng(case["renders"])
        entries = []
        for k in range(case["renders"]):
            w, h = (int(rng.integers(max(16, case[a] // 3), case[a] + 1)) for a in ("width", "height"))
            sc = _scene("flat", int(rng.integers(max(10, case["prims"] // 10), case["prims"] + 1)),
                        int(rng.integers(1, case["lights"] + 1)), 64 * seed + k)
            entries.append({"scene": _context(sc), "width": w, "height": h,
                            "spp": int(rng.integers(max(1, case["spp"] // 4), case["spp"] + 1)), "seed": seed + k})
        return {"path": path, "batch": api.BatchRenderer(api.Context(0), entries)}
    w, h = case["width"], case["height"]
    scene = _scene(case["scene"], case["prims"], case["lights"], seed, (w, h), case["spp"])
    ctx = _context(scene)
    xyz = torch.zeros(h * w * 3, dtype=torch.float32, device=dev)
    counts = torch.zeros(h * w, dtype=torch.int32, device=dev)
    state = {"path": path, "xyz": xyz, "counts": counts}
    if path == "render":
        state["integrator"] = api.PathTraceIntegrator(ctx, w, h, case["spp"], seed=seed & 0x7fffffff,
                                                      path_length=case["length"])
        state["film"] = api.Film(ctx, xyz, counts, w, h) if case["image"] else None
        return state
    # differentiable render: four albedo weights a sphere, one emission scale a light
    shaders, objects, ns, no = api.flat_indices(scene)
    shader_param, object_param, init = np.full(ns, -1, np.int32), np.full(no, -1, np.int32), []
    for name, sh in scene.root.shaders.items():
        if name.startswith("mat"):
            shader_param[shaders[id(sh)]] = len(init)
            init += [0.8 * float(sh.color[0])] * 4
    for name in scene.root.objects:
        if name.startswith("light"):
            object_param[objects[(0, name)]] = len(init)
            init.append(1.0)
    g = torch.Generator(device="cuda").manual_seed(seed)
    state["params"] = torch.tensor(init, dtype=torch.float32, device=dev)
    state["target"] = 0.2 * torch.rand(h * w, 3, generator=g, device=dev)
    state["renderer"] = api.DiffRenderer(ctx, w, h, case["spp"], shader_param, object_param, len(init),
                                         seed=seed & 0x7fffffff, path_length=case["length"])
    return state


def run(state):
    path = state["path"]
    if path == "trace":
        if state["hits"] is None:
            return state["tracer"].trace(state["rays"], fields=state["fields"])
        state["tracer"].trace_device(state["rays"], state["hits"])
        return state["hits"]
    if path == "lights":
        rows, ids = state["tree"].sample(state["queries"])
        return {"samples": rows, "ids": ids.view(np.int64)}
    if path == "batch":
        b = state["batch"]
        b.zero()
        b.render(with_stats=False)
        return {"films": b.films, "counts": b.counts}
    xyz, counts = state["xyz"], state["counts"]
    xyz.zero_()
    counts.zero_()
    if path == "render":
        state["integrator"].integrate_device(xyz, counts, with_stats=False)
        out = {"xyz": xyz, "counts": counts}
        if state["film"] is not None:
            out["image"] = state["film"].srgb8()
        return out
    r, params = state["renderer"], state["params"]
    r.forward(params, xyz, counts)
    n = counts.view(-1, 1).float()
    dl = 2.0 * (xyz.view(-1, 3) / n - state["target"]) / n
    return {"xyz": xyz, "counts": counts, "grad": r.adjoint(params, dl.reshape(-1))}


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------

# Reading a ray (o, d, four differentials, time, type) and the bytes of a
# primitive (its geometry and its instance record) in the scene.
RAY_BYTES = 6 * 12 + 4 + 2
PRIM_BYTES = {"plain": 48, "flat": 56, "heightfield": 80, "motion": 240, "gtr": 48, "rect": 48, "adjoint": 48,
              "many_light": 224}
# Operations: a slab test of four boxes per tree level, and one primitive
# test, for every ray; a light sample (a level of the light tree: two node
# estimates), one closure evaluation and a spectral upsampling for every
# path vertex.
BOX4_FLOPS, PRIM_FLOPS, LIGHT_LEVEL_FLOPS, VERTEX_FLOPS = 4 * 18, 30, 2 * 60, 400


def _count(case):
    n = case["prims"]
    return n * n if case["scene"] in ("heightfield", "motion") else n


def _ray_flops(prims):
    return BOX4_FLOPS * (1 + math.log(max(prims, 1), 4)) + PRIM_FLOPS


def _vertex_flops(prims, lights):
    return 2 * _ray_flops(prims) + LIGHT_LEVEL_FLOPS * math.log2(max(lights, 1) + 1) + VERTEX_FLOPS


def work(case):
    path = case["path"]
    if path == "trace":
        n, prims = case["rays"], _count(case)
        fields = SHADING_FIELDS if case["fields"] == "shading" else HIT_FIELDS
        out = sum(np.dtype(api.HIT_FIELDS[f][0]).itemsize * api.HIT_FIELDS[f][1] for f in fields)
        return {"bytes": n * (RAY_BYTES + out) + prims * PRIM_BYTES[case["scene"]], "flops": n * _ray_flops(prims)}
    if path == "lights":
        return {"bytes": case["queries"] * (15 * 4 + 14 * 4 + 8) + case["lights"] * 48,
                "flops": case["queries"] * (LIGHT_LEVEL_FLOPS * math.log2(case["lights"] + 1) + 100)}
    if path == "batch":
        # sides, samples and scenes are spread evenly below the case's own
        pixels = case["renders"] * (case["width"] * 2 / 3) * (case["height"] * 2 / 3)
        return {"bytes": 2 * 16 * pixels + case["renders"] * 0.55 * case["prims"] * PRIM_BYTES["flat"],
                "flops": pixels * 0.63 * case["spp"] * 4 * _vertex_flops(0.55 * case["prims"], 0.5 * case["lights"])}
    pixels, prims = case["width"] * case["height"], _count(case)
    # the film is read and written; most paths end before their last vertex
    vertices = pixels * case["spp"] * (1 + 0.5 * (case["length"] - 1))
    passes = 2 if path == "diff" else 1
    return {"bytes": passes * (2 * 16 * pixels + prims * PRIM_BYTES[case["scene"]] + case["lights"] * 48),
            "flops": passes * vertices * _vertex_flops(prims, case["lights"])}


# --------------------------------------------------------------------------
# 64-bit results
# --------------------------------------------------------------------------

def exact(case, seed):
    """The distance to the closest hit of each ray against the plain scene
    (spheres, the light's sphere and the flat ground square), solved in 64
    bits.  The other outputs have no such value: ids and flags are whole
    numbers, patch hits elsewhere are defined by the renderer's own dicing,
    and a film is a sum over paths whose every turn depends on rounding."""
    if case["path"] != "trace" or case["scene"] != "plain" or case["rays"] > 500000:
        return None
    rays = _rays(case, seed)
    fields = SHADING_FIELDS if case["fields"] == "shading" else HIT_FIELDS
    scene = _scene("plain", case["prims"], case["lights"], seed).root
    o, d = rays["o"].double(), rays["d"].double()
    inf = torch.tensor(math.inf, dtype=torch.float64, device=o.device)
    best = torch.full_like(o[:, 0], math.inf)
    for name, ob in scene.objects.items():
        if name == "ground":
            t = -o[:, 2] / d[:, 2]
            p = o + d * t[:, None]
            inside = (p[:, 0].abs() <= 10) & (p[:, 1].abs() <= 10) & (t > 0)
            best = torch.minimum(best, torch.where(inside, t, inf))
            continue
        centre, radius = (ob.locations[0], ob.radii[0]) if name == "light" else (ob.location, ob.radius)
        oc = o - torch.tensor(np.asarray(centre, np.float32).astype(np.float64), device=o.device)
        a, b = (d * d).sum(1), 2 * (d * oc).sum(1)
        c = (oc * oc).sum(1) - float(np.float32(radius)) ** 2
        disc = b * b - 4 * a * c
        root = disc.clamp_min(0).sqrt()
        q = -0.5 * torch.where(b < 0, b - root, b + root)
        t0, t1 = q / a, c / q
        t0, t1 = torch.minimum(t0, t1), torch.maximum(t0, t1)
        t = torch.where(t0 >= 1e-4, t0, torch.where(t1 >= 1e-4, t1, inf))
        best = torch.minimum(best, torch.where(disc >= 0, t, inf))
    best = torch.where(rays["type"] == 32, inf, best)  # a shadow ray reports no distance
    return {f: best if f == "t" else None for f in fields}
