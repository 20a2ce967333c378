"""The work that programs have this library do, as cases that can be timed.

A case names a scene generator, its size, the build parameters and what one
pass does:

  build    triangles on the device -> CWBVH -> its nodes and primitive order on
           the host (the drop-in for the reference's builder)
  frame    triangles on the device -> CWBVH -> closest hits of a camera's rays,
           as for geometry that changes from frame to frame
  batch    many scenes of uneven size in one segmented build, then the rays of
           all of them in one multi-BVH traversal
  trace    rays against a resident CWBVH: closest hits, occlusion, or closest
           hits on the 24-byte compressed triangles
  serve    a host ray batch against a resident CWBVH, hits on the host
  tlas     rays through instances: a TLAS over resident BLAS
  dynamic  moved objects of a resident BVH2: new leaf boxes, refit, box queries

Scenes and rays are the repository's benchmark generators (uniform soup,
Gaussian clusters, architectural), drawn on the GPU from the case's seed.
Every output is an id, a bit pattern, an offset or bytes of a tree, so equal
results are equal words and there is nothing to compare in 64 bits.
"""
import math

import numpy as np
import torch

import obvhs_gb300 as G
from obvhs_gb300.params import PRESETS, BvhBuildParams

#: Build parameters by name: the six presets, and the plain PLOC -> CWBVH
#: builds (radius, passes at distance 1) without reinsertion or pre-splits.
PLAIN = {"ploc_r16": (16, 0), "ploc_r14": (14, 3)}


def params_of(name):
    if name in PLAIN:
        radius, threshold = PLAIN[name]
        return BvhBuildParams(False, radius, threshold, 0.0, 0.0, 0, 3, 3.0)
    return PRESETS[name]()


def listed():
    return [
        # one small object of a scene rebuilt, the tree taken back to the host
        {"name": "build-2k-fast", "op": "build", "scene": "soup", "n": 2_000, "params": "fast"},
        # the smallest benchmark configuration: 10k triangles, a 256 x 256 view
        {"name": "frame-10k", "op": "frame", "scene": "soup", "n": 10_000, "params": "ploc_r16",
         "rays": "view", "w": 256, "h": 256},
        # a mid-sized asset imported with the default preset; odd sizes
        {"name": "build-100k-medium", "op": "build", "scene": "clusters", "n": 100_003, "params": "medium"},
        # a quality build (pre-splits, U128 codes, reinsertion) and its full-HD view
        {"name": "frame-1m-slow", "op": "frame", "scene": "clusters", "n": 1_000_000, "params": "slow",
         "rays": "view", "w": 1920, "h": 1080},
        # the headline build at its full size, viewed once
        {"name": "frame-8m", "op": "frame", "scene": "arch", "n": 8_000_000, "params": "ploc_r14",
         "rays": "view", "w": 1280, "h": 720},
        # a level's worth of objects built and traced together
        {"name": "batch-96", "op": "batch", "scene": "clusters", "n": 96, "low": 1_000, "high": 200_000,
         "params": "medium"},
        # path tracing on a resident quality tree: camera rays, then incoherent ones
        {"name": "trace-1m-view", "op": "trace", "scene": "clusters", "n": 1_000_000, "params": "slow",
         "rays": "view", "w": 1920, "h": 1080, "mode": "closest"},
        {"name": "trace-8m-incoherent", "op": "trace", "scene": "arch", "n": 8_000_000, "params": "ploc_r14",
         "rays": "inside", "w": 16_000_000, "h": 1, "mode": "closest"},
        # shadow rays of the same kind of scene
        {"name": "trace-2m-shadow", "op": "trace", "scene": "arch", "n": 2_000_000, "params": "medium",
         "rays": "shadow", "w": 4_000_000, "h": 1, "mode": "miss"},
        # the smallest request of a ray service
        {"name": "serve-1k", "op": "serve", "scene": "soup", "n": 10_000, "params": "medium",
         "rays": "inside", "w": 1_000, "h": 1},
        # instances under a TLAS
        {"name": "tlas-64", "op": "tlas", "scene": "soup", "n": 64, "low": 5_000, "high": 20_000, "params": "medium",
         "rays": "inside", "w": 1_000_000, "h": 1},
        # a physics step over moving objects
        {"name": "dynamic-60k", "op": "dynamic", "scene": "clusters", "n": 60_000, "params": "fast", "moved": 6_000,
         "queries": 1_024},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    op = rng.choice(["build", "frame", "frame", "batch", "trace", "trace", "trace", "serve", "tlas", "dynamic"])
    scene = rng.choice(["soup", "clusters", "arch"])
    c = {"op": op, "scene": scene}
    if op == "build":
        c.update(n=_log_int(rng, 1_000, 300_000), params=rng.choice(["fastest", "very_fast", "fast", "medium"]))
    elif op == "frame":
        params = rng.choice(list(PRESETS) + list(PLAIN))
        c.update(n=_log_int(rng, 3_000, 2_000_000 if params in PRESETS else 8_000_000), params=params, rays="view",
                 w=rng.randint(160, 1920), h=rng.randint(90, 1080))
    elif op == "batch":
        c.update(n=_log_int(rng, 8, 160), low=rng.randint(1_000, 4_000), high=rng.randint(20_000, 150_000),
                 params=rng.choice(["very_fast", "fast", "medium", "ploc_r14"]))
    elif op == "trace":
        mode = rng.choice(["closest", "closest", "miss", "compressed"])
        c.update(n=_log_int(rng, 10_000, 4_000_000), params=rng.choice(["fast", "medium", "slow", "ploc_r14"]), mode=mode)
        rays = "shadow" if mode == "miss" else rng.choice(["view", "inside"])
        c["rays"] = rays
        if rays == "view":
            c.update(w=rng.randint(160, 2560), h=rng.randint(90, 1440))
        else:
            c.update(w=_log_int(rng, 30_000, 8_000_000), h=1)
    elif op == "serve":
        c.update(n=_log_int(rng, 10_000, 500_000), params="medium", rays="inside", w=_log_int(rng, 1_000, 100_000), h=1)
    elif op == "tlas":
        c.update(scene="soup", n=_log_int(rng, 8, 200), low=rng.randint(500, 5_000), high=rng.randint(8_000, 30_000),
                 params=rng.choice(["fast", "medium"]), rays="inside", w=_log_int(rng, 50_000, 2_000_000), h=1)
    else:
        n = _log_int(rng, 5_000, 300_000)
        c.update(n=n, params=rng.choice(["fast", "medium"]), moved=rng.randint(1, n // 4),
                 queries=_log_int(rng, 64, 4_096))
    return c


# --- scenes (obvhs_gb300/scenes.py, drawn on the GPU) -------------------------


class Rand:
    """Seeded draws on the GPU."""

    def __init__(self, seed, stream):
        self.g = torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + stream)

    def uniform(self, lo, hi, *shape):
        return torch.rand(shape, generator=self.g, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    def normal(self, *shape):
        return torch.randn(shape, generator=self.g, device="cuda", dtype=torch.float64)

    def integers(self, n, *shape):
        return torch.randint(0, n, shape, generator=self.g, device="cuda")

    def permutation(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _directions(r, n):
    z = 1 - 2 * r.uniform(0, 1, n)
    phi = r.uniform(0, 2 * math.pi, n)
    s = (1 - z * z).clamp(min=0).sqrt()
    return torch.stack([s * phi.cos(), s * phi.sin(), z], 1)


def _equilateral(r, centres, edge):
    """Equilateral triangles of the given edge in random orientation."""
    n = len(centres)
    normal = _unit(r.normal(n, 3))
    t = r.normal(n, 3)
    t = _unit(t - (t * normal).sum(1, keepdim=True) * normal)
    b = torch.linalg.cross(normal, t)
    phi = r.uniform(0, 2 * math.pi, n, 1)
    rad = (edge / math.sqrt(3))[:, None]
    return torch.cat([centres + rad * ((phi + 2 * math.pi * k / 3).cos() * t + (phi + 2 * math.pi * k / 3).sin() * b)
                      for k in range(3)], 1).float()


def _soup(r, n):
    """Centroids in [-1, 1]^3, vertices within 0.02 of them."""
    c = r.uniform(-1, 1, n, 1, 3)
    return (c + r.uniform(-0.02, 0.02, n, 3, 3)).reshape(n, 9).float(), (0.0, 0.0, -3.0)


def _clusters(r, n):
    """64 Gaussian clusters in [-10, 10]^3, log-normal edges around 0.01; the
    view is three sigmas in front of the densest cluster."""
    centre = r.uniform(-10, 10, 64, 3)
    sigma = r.uniform(math.log(0.1), math.log(2.0), 64).exp()
    which = r.integers(64, n)
    cen = centre[which] + r.normal(n, 3) * sigma[which, None]
    tris = _equilateral(r, cen, (math.log(0.01) + 0.7 * r.normal(n)).exp())
    k = int(sigma.argmin())
    x, y, z = centre[k].tolist()
    return tris, (x, y, z - 3.0 * float(sigma[k]))


ARCH_LO, ARCH_HI = (-10.0, -3.0, -10.0), (10.0, 3.0, 10.0)


def _arch_box(r, n):
    lo = torch.tensor(ARCH_LO, device="cuda", dtype=torch.float64)
    hi = torch.tensor(ARCH_HI, device="cuda", dtype=torch.float64)
    return lo + r.uniform(0, 1, n, 3) * (hi - lo)


def _arch(r, n):
    """40 % of the triangles from 200 tessellated axis-aligned quads, the rest
    clutter of edge 0.002-0.02, in a 20 x 6 x 20 box."""
    quads = 200
    walls = max(quads, int(n * 0.4))
    per = -(-walls // quads)
    axis = r.integers(3, quads)
    size = r.uniform(0.05, 0.5, quads)
    origin = _arch_box(r, quads)
    k = torch.arange(walls, device="cuda")
    q, cell, half = k // per, (k % per) // 2, (k % per) % 2
    side = max(1, math.ceil(math.sqrt((per + 1) // 2)))
    axes = torch.tensor([[1, 2], [0, 2], [0, 1]], device="cuda")[axis]
    unit = torch.eye(3, device="cuda", dtype=torch.float64)
    du = (unit[axes[:, 0]] * size[:, None])[q]
    dv = (unit[axes[:, 1]] * size[:, None])[q]
    a = origin[q] + (cell % side).double()[:, None] * du + (cell // side).double()[:, None] * dv
    first = (half == 0)[:, None]
    wall = torch.cat([a, torch.where(first, a + du, a + du + dv), torch.where(first, a + du + dv, a + dv)], 1).float()
    rest = n - walls
    if rest <= 0:
        return wall[:n].contiguous(), (0.0, 0.0, -9.0)
    clutter = _equilateral(r, _arch_box(r, rest), r.uniform(0.002, 0.02, rest))
    return torch.cat([wall, clutter])[r.permutation(n)].contiguous(), (0.0, 0.0, -9.0)


SCENES = {"soup": _soup, "clusters": _clusters, "arch": _arch}


def _ray_array(o, d, tmax):
    rays = torch.zeros((len(d), 8), device="cuda", dtype=torch.float32)
    rays[:, 0:3] = o
    rays[:, 4:7] = d
    rays[:, 7] = tmax
    return rays


def _view(camera, w, h):
    """Pixel-centre rays of a 60-degree pinhole looking along +z."""
    th = math.tan(math.radians(30))
    x = ((torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w * 2 - 1) * th * w / h
    y = (1 - (torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h * 2) * th
    d = torch.stack([x[None].expand(h, w), y[:, None].expand(h, w), torch.ones(h, w, device="cuda").double()], 2)
    o = torch.tensor(camera, device="cuda", dtype=torch.float32)
    return _ray_array(o, _unit(d.reshape(-1, 3)).float(), math.inf)


def _bounds(tris):
    v = tris.reshape(-1, 3)
    return v.amin(0).double(), v.amax(0).double()


def _rays(case, r, tris, camera):
    n = case["w"] * case["h"]
    if case["rays"] == "view":
        return _view(camera, case["w"], case["h"])
    lo, hi = _bounds(tris)
    if case["scene"] == "arch":  # the room; its walls reach beyond it
        lo, hi = (torch.tensor(v, device="cuda", dtype=torch.float64) for v in (ARCH_LO, ARCH_HI))
    o = lo + r.uniform(0, 1, n, 3) * (hi - lo)
    if case["rays"] == "inside":
        return _ray_array(o.float(), _directions(r, n).float(), math.inf)
    # shadow rays toward four lights near the top, ending just before them
    light = (lo + hi) / 2 + (hi - lo) * torch.cat([r.uniform(-0.45, 0.45, 4, 1), r.uniform(0.33, 0.48, 4, 1),
                                                   r.uniform(-0.45, 0.45, 4, 1)], 1)
    to = light[r.integers(4, n)] - o
    dist = to.norm(dim=1)
    return _ray_array(o.float(), (to / dist[:, None]).float(), (dist * (1 - 1e-4)).float())


def _sizes(case):
    """Triangle counts of a batch: log-uniform over [low, high], large and small ones mixed."""
    n = case["n"]
    at = [(i * 0.6180339887498949) % 1.0 for i in range(n)]
    return [int(case["low"] * (case["high"] / case["low"]) ** x) for x in at]


def _tri_boxes(tris):
    v = tris.reshape(-1, 3, 3)
    return torch.cat([v.amin(1), v.amax(1)], 1).contiguous()


# --- what a program holds before the call, and the call ------------------------


def prepare(case, seed):
    r = Rand(seed, 1)
    op = case["op"]
    s = {"op": op, "params": params_of(case["params"])}
    if op in ("batch", "tlas"):
        tris, rays, owner, shift = [], [], [], []
        for i, n in enumerate(_sizes(case)):
            t, _ = SCENES[case["scene"]](r, n)
            if op == "tlas":  # the instances apart, partly overlapping
                t = (t + r.uniform(-5, 5, 1, 3).float().repeat(1, 3)).contiguous()
            else:
                k = int(4096 + n)
                lo, hi = _bounds(t)
                rays.append(_ray_array((lo + r.uniform(0, 1, k, 3) * (hi - lo)).float(), _directions(r, k).float(),
                                       math.inf))
                owner.append(torch.full((k,), i, dtype=torch.int32, device="cuda"))
            tris.append(t)
        s["tris"] = tris
        if op == "batch":
            s["rays"], s["owner"] = torch.cat(rays), torch.cat(owner)
        else:
            s["blas"] = G.build_cwbvh_from_tris_segmented(tris, s["params"])
            boxes = torch.stack([torch.cat(_bounds(t)) for t in tris]).float().contiguous()
            s["tlas"] = G.build_cwbvh(boxes, BvhBuildParams(False, 6, 0, 0.0, 0.0, 0, 1, 3.0))
            s["rays"] = _ray_array(r.uniform(-7, 7, case["w"], 3).float(), _directions(r, case["w"]).float(), math.inf)
        return s
    tris, camera = SCENES[case["scene"]](r, case["n"])
    if op == "dynamic":
        boxes = _tri_boxes(tris)
        s["bvh"] = G.build_bvh2(boxes, s["params"])
        nodes, _ = s["bvh"].download()
        leaf = np.nonzero(nodes[:, 12:16].copy().view(np.uint32).ravel())[0]
        g = np.random.default_rng(seed)
        moved = np.sort(g.choice(leaf, size=min(case["moved"], len(leaf)), replace=False))
        new = nodes[moved].view(np.float32).reshape(-1, 8)[:, [0, 1, 2, 4, 5, 6]]
        new = new + np.tile(g.normal(scale=0.02, size=(len(moved), 3)).astype(np.float32), (1, 2))
        s["ids"] = torch.from_numpy(moved.astype(np.int32)).cuda()
        s["boxes"] = torch.from_numpy(np.ascontiguousarray(new, dtype=np.float32)).cuda()
        at = boxes[r.integers(len(boxes), case["queries"])].double()
        c, half = (at[:, :3] + at[:, 3:]) / 2, r.uniform(0.005, 0.05, case["queries"], 1)
        s["query"] = torch.cat([c - half, c + half], 1).float().cpu().numpy()
        s["contacts"] = np.zeros(64 * case["queries"], np.uint32)
        return s
    if op in ("build", "frame"):
        s["tris"] = tris
        if op == "frame":
            s["rays"] = _rays(case, r, tris, camera)
        else:
            s["nodes"] = np.zeros((case["n"], 80), np.uint8)
        return s
    s["bvh"] = G.build_cwbvh_from_tris(tris, s["params"])
    s["rays"] = _rays(case, r, tris, camera)
    if op == "serve":
        s["rays"] = s["rays"].cpu().numpy()
    else:
        s["mode"] = case["mode"]
        if case["mode"] == "compressed":
            s["bvh"].set_triangles_compressed(tris)
    return s


def run(state):
    op = state["op"]
    if op == "build":
        # into the program's own node array, as large as any tree of n triangles
        nodes, order = G.build_cwbvh_from_tris(state["tris"], state["params"]).download()
        state["nodes"][:len(nodes)] = nodes
        return {"nodes": state["nodes"], "used": len(nodes), "order": order}
    if op == "frame":
        return {"hits": G.build_cwbvh_from_tris(state["tris"], state["params"]).ray_traverse(state["rays"])}
    if op == "batch":
        bvhs = G.build_cwbvh_from_tris_segmented(state["tris"], state["params"])
        return {"hits": G.ray_traverse_multi(bvhs, state["owner"], state["rays"])}
    if op == "trace":
        b = state["bvh"]
        call = {"closest": b.ray_traverse, "miss": b.ray_traverse_miss, "compressed": b.ray_traverse_compressed}
        return {"hits": call[state["mode"]](state["rays"])}
    if op == "serve":
        ids, t = state["bvh"].ray_traverse(state["rays"])
        return {"ids": ids, "t": t.view(np.uint32)}
    if op == "tlas":
        return {"hits": state["tlas"].ray_traverse_tlas_blas(state["blas"], state["rays"])}
    b = state["bvh"]
    b.set_node_aabbs(state["ids"], state["boxes"])
    b.refit_all()
    # the contact list of the step, as long as the program has room for
    found = b.aabb_query(state["query"])
    ids = np.concatenate(found)[:len(state["contacts"])]
    state["contacts"][:len(ids)] = ids
    return {"ids": state["contacts"], "counts": np.array([len(f) for f in found])}


def work(case):
    """Bytes: triangles (36 B) or boxes in, rays in (32 B) and hits out (8 B;
    16 B through a TLAS, 1 B for occlusion), the tree that the pass writes for
    its caller or reads (about 0.12 nodes of 80 B and one index a primitive).
    Operations: the radius search of the builds (13 a pair, 2r pairs, about 2
    clusters a primitive) and, a ray, some 12 nodes of 8 children at 20
    operations and 4 triangles at 45."""
    op, p = case["op"], params_of(case["params"])
    rays = case.get("w", 0) * case.get("h", 0)
    n = case["n"]
    if op in ("batch", "tlas"):
        n = sum(_sizes(case))
        if op == "batch":
            rays = n + 4096 * case["n"]
    tree = 14 * n
    search = 2.0 * n * 2 * int(p.ploc_search_distance) * 13
    hit = 16 if op == "tlas" else 1 if case.get("mode") == "miss" else 8
    trace = rays * (12 * 8 * 20 + 4 * 45)
    if op == "build":
        return {"bytes": 36 * n + tree, "flops": search}
    if op in ("frame", "batch"):
        return {"bytes": 36 * n + rays * (32 + hit), "flops": search + trace}
    if op == "dynamic":
        return {"bytes": case["moved"] * 28 + 2 * n * 32 + case["queries"] * 24, "flops": 6.0 * n}
    return {"bytes": tree + 36 * n + rays * (32 + hit), "flops": trace}


def exact(case, seed):
    """No output is a rounded number: ids, bit patterns, counts and bytes."""
    return None
