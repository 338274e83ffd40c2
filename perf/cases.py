"""The framework's work as its users call it, as cases that can be timed.

listed() and draw() give cases, prepare() makes what a program has in hand
before the call, run() is one pass through the public entry points
(math_b200.painter), work() what that pass cannot do without and exact() its
outputs in 64 bits where they can be had without a renderer.

Kinds:
  render  a new painter of a resident scene, its passes, the images read back
          (an interactive or offline render of one scene)
  batch   renders of several resident scenes through a job server that the
          program keeps, all submitted at once, their images read back
  open    a scene built from host arrays (mesh ingestion, copies, BVH, facet
          records) and its first image
  trace   ray queries from host arrays against a resident scene

Sizes are those of the repository's own workloads (the 3- and 4-space Cornell
boxes, the noisy 4-space sphere, the members of the mixed 3/4/5-space batch)
and smaller ones of the same kinds.  A mesh is a hull of points on the sphere
(in 3-space an icosphere) computed once per process and turned by a rotation
drawn from the seed, so every seed gives another scene and other streams.
"""

from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from math_b200 import painter as P
from math_b200 import scenes


def _render(name, n, edge, spp, depth, points, precision, spectrum=False, integrator="bpt", scene="box",
            passes=1, flat=False):
    return {"name": name, "kind": "render", "n": n, "edge": edge, "spp": spp, "depth": depth, "points": points,
            "precision": precision, "spectrum": spectrum, "integrator": integrator, "scene": scene,
            "passes": passes, "flat": flat}


def listed():
    return [
        # an interactive preview: a small window at one sample per pixel, all latency
        _render("preview_3d_f32", 3, 32, 1, 5, 642, "float"),
        # the 3-space Cornell box (256^2, 16 samples, 20,480 triangles) in the
        # precision that follows the reference bit for bit
        _render("cornell_3d_f64", 3, 256, 16, 5, 10242, "double"),
        # the 4-space Cornell box in 64 spectral bands (64^3 voxels, 27 samples)
        _render("cornell_4d_spectrum_f32", 4, 64, 16, 6, 20000, "float", spectrum=True, scene="box_solid"),
        # an object alone, many materials, ball light, parallel projection: short paths
        _render("sphere_4d_f32", 4, 61, 8, 8, 40000, "float", scene="sphere"),
        # a 4-space member of the mixed batch in double precision, an odd screen
        _render("mixed_4d_f64", 4, 37, 8, 7, 12000, "double"),
        # a 5-space member of the mixed batch, the longest work of the list
        _render("mixed_5d_f32", 5, 18, 16, 8, 6000, "float"),
        # a small 5-space render in double precision, an odd screen
        _render("mixed_5d_f64", 5, 9, 16, 6, 3000, "double"),
        # path tracing in 64 bands, and two accumulated passes of it in double precision
        _render("pt_4d_spectrum_f32", 4, 48, 16, 6, 20000, "float", spectrum=True, integrator="pt", scene="box_solid"),
        _render("pt_3d_f64", 3, 255, 16, 5, 10242, "double", integrator="pt", passes=2),
        # twelve renders of mixed dimension through the job server at once
        {"name": "batch_f32", "kind": "batch", "jobs": 12, "scale": 0.35, "precision": "float"},
        # opening a 4-space scene from host arrays, to its first low-sample image
        {"name": "open_4d_f32", "kind": "open", "n": 4, "edge": 24, "spp": 1, "depth": 5, "points": 20000,
         "precision": "float"},
        # closest hits of rays from host arrays (picking, probes)
        {"name": "trace_4d_f64", "kind": "trace", "n": 4, "rays": 65536, "points": 8000, "precision": "double",
         "any": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# the largest screen edge of a drawn render per dimension: at 16 samples it
# costs less than the largest listed case
_EDGES = {3: (16, 320), 4: (8, 48), 5: (5, 15)}
_POINTS = {3: (162, 10242), 4: (500, 20000), 5: (200, 6000)}


def draw(rng):
    kind = rng.choice(["render"] * 7 + ["batch", "open", "trace"])
    precision = rng.choice(["float", "double"])
    n = rng.choice([3, 4, 5])
    points = _log(rng, *_POINTS[n])
    if kind == "batch":
        return {"kind": "batch", "jobs": rng.randint(2, 14), "scale": round(rng.uniform(0.1, 0.3), 3),
                "precision": precision}
    if kind == "open":
        return {"kind": "open", "n": n, "edge": _log(rng, 4, _EDGES[n][1] // 2), "spp": rng.choice([1, 2, 4]),
                "depth": rng.randint(2, 8), "points": points, "precision": precision}
    if kind == "trace":
        return {"kind": "trace", "n": n, "rays": _log(rng, 100, 100000), "points": min(points, 8000 if n < 5 else 1000),
                "precision": precision, "any": rng.random() < 0.5}
    c = _render("", n, _log(rng, *_EDGES[n]), _log(rng, 1, 16), rng.randint(1, 8), points, precision,
                spectrum=rng.random() < 0.35, integrator=rng.choice(["bpt", "bpt", "pt"]),
                scene=rng.choice(["box", "box", "box_solid"] + (["sphere"] if n == 4 else [])),
                passes=1, flat=rng.random() < 0.15)
    del c["name"]
    return c


# --------------------------------------------------------------------------
# inputs


@functools.lru_cache(maxsize=None)
def _mesh(n, points, noise=0.0):
    """Unit sphere mesh: in 3-space the icosphere with the nearest number of vertices, else a convex hull."""
    if n == 3:
        level = min(range(1, 7), key=lambda k: abs(math.log((10 * 4 ** k + 2) / points)))
        return scenes.icosphere(level)
    return scenes.convex_hull_mesh(scenes.sphere_points(n, points, 7, noise=noise))


def _turned(n, points, seed, noise=0.0):
    p, f = _mesh(n, points, noise)
    rot = scenes.random_rotation(n, seed % (1 << 31))
    return (p.astype(np.float64) @ rot.T).astype(np.float32), f


def _box(n, points, edge, seed, solid=False):
    """The Cornell box of the mixed batch: walls open towards the camera, a
    ceiling light and the mesh; `solid`: a rotated parallelotope beside it."""
    colors = {"default": (0.7, 0.7, 0.7), (0, -1): (0.75, 0.15, 0.15), (0, 1): (0.15, 0.75, 0.15)}
    shapes = scenes.box_walls(n, 1.0, colors, open_axis=n - 1, open_side=-1)
    carrier, light = scenes.ceiling_light(n, 1.0, 0.5, up_axis=1, radiance=float(10 * 2 ** (n - 3)))
    shapes.append(carrier)
    light["shape"] = len(shapes) - 1
    if solid:
        vectors = (scenes.random_rotation(n, (seed + 1) % (1 << 31)) * 0.5).T
        center = np.array([0.45, -0.55] + [0.3] * (n - 2))
        shapes.append({"type": "parallelotope", "metalness": 0.0, "roughness": 0.2, "color": [0.8, 0.5, 0.3],
                       "alpha": 1.0, "org": (center - 0.5 * vectors.sum(axis=0)).tolist(),
                       "vectors": vectors.tolist()})
    p, f = _turned(n, points, seed)
    middle = [-0.35 if solid else 0.0, -0.55] + [-0.1] * (n - 2)
    shapes.append({"type": "mesh", "objects": [{
        "points": p, "facets": f, "matrix": scenes.transform_matrix(n, 0.4, middle), "metalness": 0.0,
        "roughness": 0.3, "color": [0.8, 0.8, 0.8], "alpha": 1.0}]})
    return {"n": n, "shapes": shapes, "lights": [light], "projector": scenes.camera(n, 3.0, [edge] * (n - 1)),
            "background": [0.0, 0.0, 0.0]}


def _sphere(n, points, edge, seed):
    """A noisy sphere of 16 mesh objects of different roughness, a ball light and a parallel projection."""
    p, f = _turned(n, points, seed, noise=0.002)
    level = np.random.default_rng(seed).integers(0, 16, size=len(f))
    objects = [{"points": p, "facets": f[level == k], "matrix": scenes.transform_matrix(n, 1.0, [0] * n),
                "metalness": 0.0, "roughness": 0.1 + 0.03 * k, "color": [0.8, 0.6, 0.4], "alpha": 1.0}
               for k in range(16) if np.any(level == k)]
    d = np.zeros(n)
    d[1], d[n - 1] = -1.0, 0.6
    center = [0.0] * n
    center[1], center[n - 1] = 1.7, -1.0
    light = {"type": "ball", "center": center, "direction": (d / np.linalg.norm(d)).tolist(), "radius": 0.3,
             "radiance": [30.0] * 3}
    axes = np.eye(n)
    projector = {"type": "parallel", "org": (-3.0 * axes[n - 1]).tolist(), "dir": axes[n - 1].tolist(),
                 "axes": axes[:n - 1].tolist(), "units_per_pixel": 2.4 / edge, "size": [edge] * (n - 1)}
    return {"n": n, "shapes": [{"type": "mesh", "objects": objects}], "lights": [light], "projector": projector,
            "background": [0.0, 0.0, 0.0]}


def _description(case, seed):
    if case.get("scene") == "sphere":
        return _sphere(case["n"], case["points"], case["edge"], seed)
    return _box(case["n"], case["points"], case.get("edge", 8), seed, solid=case.get("scene") == "box_solid")


def _jobs(case):
    """Dimension, screen edge, samples, depth and mesh points of the jobs of a batch, as the mixed batch draws them."""
    rng = random.Random(case["jobs"])
    jobs = []
    for k in range(case["jobs"]):
        n = 3 + k % 3
        lo, hi = scenes.MIXED_SCREENS[n]
        edge = max(4, int(round(rng.uniform(lo, hi) * case["scale"])))
        jobs.append((n, edge, _log(rng, 4, 64), rng.randint(5, 8), {3: 2562, 4: 3000, 5: 1000}[n]))
    return jobs


def _rays(case, seed):
    """Rays from inside the box (and from the camera's side of it) in all directions."""
    rng = np.random.default_rng(seed)
    n, count = case["n"], case["rays"]
    org = rng.uniform(-0.95, 0.95, size=(count, n))
    org[: count // 4, n - 1] = -3.0
    d = rng.normal(size=(count, n))
    # half of them towards the mesh, as probes of an object are
    aimed = slice(0, count // 2)
    d[aimed] = np.array([0.0, -0.55] + [-0.1] * (n - 2)) + 0.25 * d[aimed] - org[aimed]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.ascontiguousarray(np.concatenate([org, d], axis=1))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        jobs = _jobs(case)
        resident = [P.Scene(_box(n, points, edge, seed + k), case["precision"]) for k, (n, edge, _, _, points) in enumerate(jobs)]
        return {"case": case, "seed": seed, "jobs": jobs, "scenes": resident, "server": P.Server(16, 48 << 30)}
    desc = _description(case, seed)
    if kind == "open":
        return {"case": case, "seed": seed, "desc": desc}
    scene = P.Scene(desc, case["precision"], case.get("spectrum", False))
    if kind == "trace":
        return {"case": case, "scene": scene, "rays": _rays(case, seed)}
    return {"case": case, "seed": seed, "scene": scene}


def _images(scene, case, seed):
    painter = scene.painter(case["spp"], case["depth"], seed=seed & 0xffffffff,
                            integrator=case.get("integrator", "bpt"), flat_shading=case.get("flat", False))
    painter.run(case.get("passes", 1))
    rgb, rgba = painter.images()
    painter.close()
    return {"rgb": rgb, "rgba": rgba}


def run(state):
    case = state["case"]
    if case["kind"] == "render":
        return _images(state["scene"], case, state["seed"])
    if case["kind"] == "batch":
        server = state["server"]
        ids = [server.submit_render(scene, spp, depth, seed=(state["seed"] + k) & 0xffffffff)
               for k, (scene, (_, _, spp, depth, _)) in enumerate(zip(state["scenes"], state["jobs"]))]
        out = []
        for scene, job in zip(state["scenes"], ids):
            server.wait(job)
            rgb, rgba = server.images(job, scene.pixels)
            server.release(job)
            out.append({"rgb": rgb, "rgba": rgba})
        return out
    if case["kind"] == "open":
        scene = P.Scene(state["desc"], case["precision"])
        out = _images(scene, case, state["seed"])
        scene.close()
        return out
    hits = state["scene"].trace(state["rays"], any_hit=case["any"])
    if case["any"]:
        return {"hit": hits}
    kind, index, t, point = hits
    return {"kind": kind, "index": index, "t": t, "point": point}


# --------------------------------------------------------------------------
# floors


# facets per mesh point of a hull on the sphere, measured on the hulls above
_FACETS = {3: 2.0, 4: 6.7, 5: 29.5}


def _query_flops(n, points):
    """One ray query: the 2n flat shapes, a root-to-leaf descent of the BVH and two facets."""
    facets = max(2.0, _FACETS[n] * points)
    return 2 * n * 2 * (2 * n + 1) + math.log2(facets) * 6 * n + 2 * 2 * n * (n + 1)


def _scene_bytes(n, points, size):
    """Facet records and BVH nodes, once."""
    facets = _FACETS[n] * points
    return facets * ((n * (n + 1)) * size + 4 * (n + 3)) + facets * 0.7 * (2 * n * size + 8)


def _render_work(n, edge, spp, depth, points, precision, integrator="bpt", passes=1):
    """Paths of two subpaths of half the depth on average and one connection
    per pair of vertices (path tracing: one subpath, one light ray per
    vertex); about 300 operations of shading and sampling per vertex."""
    size = 8 if precision == "double" else 4
    pixels = edge ** (n - 1)
    paths = passes * pixels * scenes.stratified_spp(spp, n - 1)
    k = max(1.0, depth / 2)
    queries = 2 * k + k * k / 2 if integrator == "bpt" else 2 * k
    vertices = 2 * k if integrator == "bpt" else k
    return {"bytes": _scene_bytes(n, points, size) + 28 * pixels,
            "flops": paths * (queries * _query_flops(n, points) + vertices * 300.0)}


def work(case):
    if case["kind"] == "batch":
        parts = [_render_work(n, edge, spp, depth, points, case["precision"]) for n, edge, spp, depth, points in _jobs(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, points = case["n"], case["points"]
    size = 8 if case["precision"] == "double" else 4
    if case["kind"] == "trace":
        out = 4 if case["any"] else 8 + 8 + 8 * n
        return {"bytes": case["rays"] * (16 * n + out) + _scene_bytes(n, points, size),
                "flops": case["rays"] * _query_flops(n, points)}
    w = _render_work(n, case["edge"], case["spp"], case["depth"], points, case["precision"],
                     case.get("integrator", "bpt"), case.get("passes", 1))
    if case["kind"] == "open":
        # the host arrays in, the records out once more, an n x n elimination per facet
        facets = _FACETS[n] * points
        w["bytes"] += points * 4 * n + facets * 4 * n
        w["flops"] += facets * n * 2 * n ** 3 / 3
    return w


# --------------------------------------------------------------------------
# 64 bits


def _complement(v):
    """Normals of the hyperplanes spanned by [F, n - 1, n] vectors, by cofactors."""
    n = v.shape[-1]
    cols = torch.arange(n, device=v.device)
    return torch.stack([(-1) ** i * torch.linalg.det(v[:, :, cols[cols != i]]) for i in range(n)], dim=-1)


def _flat_hits(org, d, corner, vectors, simplex):
    """Distances [R, F] (inf: none) of rays to flat (n-1)-simplices or
    parallelotopes given by a corner and n - 1 edge vectors."""
    normal = _complement(vectors)
    normal = normal / normal.norm(dim=-1, keepdim=True)
    t = ((corner * normal).sum(-1) - org @ normal.T) / (d @ normal.T)
    ok = t > 0
    # dual vectors of the edges within the hyperplane: coordinates of the hit
    dual = torch.linalg.inv(torch.cat([vectors, normal[:, None, :]], dim=1)).transpose(1, 2)
    total = torch.zeros_like(t)
    for i in range(vectors.shape[1]):
        w = dual[:, i]
        x = org @ w.T + t * (d @ w.T) - (corner * w).sum(-1)
        ok &= (x > 0) & (x < 1)
        total += x
    if simplex:
        ok &= total < 1
    return torch.where(ok, t, torch.full_like(t, math.inf))


def exact(case, seed):
    """Ray queries by brute force in double precision.  The images have no
    value here: they are Monte-Carlo estimates on given random streams, for
    which a plain double-precision renderer would take minutes."""
    if case["kind"] != "trace" or case["any"] or case["rays"] * case["points"] * _FACETS[case["n"]] > 8e9:
        return None
    n = case["n"]
    at = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    rays = torch.from_numpy(_rays(case, seed)).to(at)
    groups = []
    for s in _description(case, seed)["shapes"]:
        if s["type"] == "mesh":
            for o in s["objects"]:
                m = torch.tensor(o["matrix"], dtype=torch.float64)
                v = torch.from_numpy(o["points"].astype(np.float64)) @ m[:n, :n].T + m[:n, n]
                f = v[torch.from_numpy(o["facets"].astype(np.int64))].to(at)
                groups.append((f[:, -1], f[:, :-1] - f[:, -1:], True))
        else:
            groups.append((torch.tensor([s["org"]], dtype=torch.float64, device=at),
                           torch.tensor([s["vectors"]], dtype=torch.float64, device=at), False))
    best = torch.full((len(rays),), math.inf, dtype=torch.float64, device=at)
    for b in range(0, len(rays), 1024):
        org, d = rays[b: b + 1024, :n], rays[b: b + 1024, n:]
        for corner, vectors, simplex in groups:
            best[b: b + 1024] = torch.minimum(best[b: b + 1024], _flat_hits(org, d, corner, vectors, simplex).amin(1))
    hit = torch.isfinite(best)
    t = torch.where(hit, best, torch.zeros_like(best))
    point = torch.where(hit[:, None], rays[:, :n] + t[:, None] * rays[:, n:], torch.zeros_like(rays[:, :n]))
    return {"kind": None, "index": None, "t": t.cpu().numpy(), "point": point.cpu().numpy()}
