"""Performance cases of the LBVH and the path tracer, through their public entry points.

A case is a dict of plain values; its "kind" says which path it takes:

  trace      ray queries against a resident triangle BVH (closest hit or any hit)
  rebuild    a per-frame hierarchy rebuild over moved triangles, then closest hits
  refit      a per-frame refit of an unchanged topology, then closest hits of segments
  overlap    broad phase: the boxes' hierarchy rebuilt, then every overlapping pair
  render     one film of a resident scene
  frame      one displayed frame of an animated scene: new vertices from the host, the
             scene refitted, rendered, tone mapped and read back as bytes
  serve      a batch of requests submitted to the render server and waited for

Ray queries and hierarchy builds take device memory, as a renderer or a simulation that
keeps its geometry on the GPU does.  Rebuild and refit return hits and not nodes: the
library keeps the nodes to itself, and callers see them through their queries.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import lux_b200 as L
from lux_b200 import scene as S
from lux_b200 import scenes as SC
from lux_b200 import server as V

# A program keeps one context (and its scratch memory and path pools) for its lifetime,
# on the stream that its own device work is queued on.
_shared: dict = {}


def _context():
    if not _shared:
        _shared["stream"] = torch.cuda.Stream()
        _shared["ctx"] = L.Context(0, stream=_shared["stream"].cuda_stream)
    return _shared["ctx"]


# ------------------------------------------------------------------------ the cases

def listed():
    return [
        # Picking and probe queries: a few rays at one mesh, where latency counts.
        {"name": "trace_probe", "kind": "trace", "geometry": "terrain", "tris": 20480,
         "rays": 2048, "pattern": "uniform", "any": False},
        # A small dynamic object rebuilt every frame: launches and latency count.
        {"name": "rebuild_small", "kind": "rebuild", "geometry": "terrain", "tris": 5001,
         "rays": 1000, "bits": 30},
        # The hierarchy microbenchmark's build: a million triangles a frame, some rays.
        {"name": "rebuild_1m", "kind": "rebuild", "geometry": "soup", "tris": 1 << 20,
         "rays": 65536, "bits": 30},
        # The microbenchmark's refit after a jitter, with bounded queries.
        {"name": "refit_1m", "kind": "refit", "geometry": "soup", "tris": 1 << 20,
         "rays": 65536, "bits": 30},
        # The microbenchmark's ray batch: the largest query.
        {"name": "trace_4m", "kind": "trace", "geometry": "soup", "tris": 1 << 20,
         "rays": 1 << 22, "pattern": "uniform", "any": False},
        # Shadow segments over a terrain, an odd count of each.
        {"name": "shadow_terrain", "kind": "trace", "geometry": "terrain", "tris": 777777,
         "rays": 1000003, "pattern": "segment", "any": True},
        # Collision broad phase over boxes with 63-bit codes, an odd count.
        {"name": "broadphase_63", "kind": "overlap", "boxes": 300007, "bits": 63},
        # The Cornell box at its stated size: tiny scene, ordinary film.
        {"name": "render_cornell", "kind": "render", "scene": "cornell", "width": 256,
         "height": 256, "spp": 64, "depth": 4, "sampler": S.SAMPLER_POWER},
        # The heavy scene (333k triangles, GGX and glass), depth 8.
        {"name": "render_heavy", "kind": "render", "scene": "heavy", "width": 512,
         "height": 512, "spp": 16, "depth": 8, "sampler": S.SAMPLER_POWER},
        # Instances and pass-through materials, light tree, an odd film.
        {"name": "render_grid", "kind": "render", "scene": "grid", "width": 401,
         "height": 301, "spp": 7, "depth": 6, "sampler": S.SAMPLER_TREE},
        # An interactive preview of a deforming mesh: one sample a pixel, bytes out.
        {"name": "preview_frame", "kind": "frame", "subdivisions": 5, "width": 320,
         "height": 240, "spp": 1, "depth": 4},
        # The render service: a mixed batch over four resident scenes.
        {"name": "serve_batch", "kind": "serve", "requests": 8, "side": 512, "spp": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "rebuild", "refit", "overlap", "render", "render",
                       "frame", "serve"])
    geometry = rng.choice(["soup", "terrain"])
    if kind == "trace":
        return {"kind": kind, "geometry": geometry, "tris": _log(rng, 1000, 1 << 20),
                "rays": _log(rng, 1000, 1 << 22),
                "pattern": rng.choice(["uniform", "segment", "camera"]),
                "any": rng.random() < 0.5}
    if kind in ("rebuild", "refit"):
        return {"kind": kind, "geometry": geometry, "tris": _log(rng, 1000, 1 << 21),
                "rays": _log(rng, 1000, 1 << 17), "bits": rng.choice([30, 30, 63])}
    if kind == "overlap":
        return {"kind": kind, "boxes": _log(rng, 1000, 1 << 20), "bits": rng.choice([30, 63])}
    if kind == "render":
        return {"kind": kind, "scene": rng.choice(["cornell", "heavy", "grid", "soup"]),
                "width": _log(rng, 64, 640), "height": _log(rng, 64, 640),
                "spp": _log(rng, 1, 24), "depth": rng.randint(2, 10),
                "sampler": rng.choice([S.SAMPLER_UNIFORM, S.SAMPLER_POWER, S.SAMPLER_TREE])}
    if kind == "frame":
        return {"kind": kind, "subdivisions": rng.randint(3, 6), "width": _log(rng, 160, 640),
                "height": _log(rng, 120, 480), "spp": rng.randint(1, 4),
                "depth": rng.randint(2, 6)}
    return {"kind": kind, "requests": rng.randint(2, 8), "side": _log(rng, 128, 512),
            "spp": _log(rng, 4, 32)}


# ------------------------------------------------------------------------ inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float32)


def _sphere(gen, n):
    z = 1 - 2 * _uniform(gen, n)
    phi = 2 * math.pi * _uniform(gen, n)
    r = torch.sqrt(torch.clamp(1 - z * z, min=0))
    return torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], 1)


def _triangles(case, gen):
    """n x 9 triangles in the unit cube.  soup: the microbenchmark's distribution (edges
    log-normal about a fifth of the mean spacing) in random order; terrain: a height field
    of smooth waves, row after row, as meshes come from files and generators."""
    n = case["tris"]
    if case["geometry"] == "soup":
        c = _uniform(gen, n, 1, 3)
        length = torch.exp(0.5 * torch.randn(n, 3, 1, generator=gen, device="cuda"))
        length = length * (2e-3 * ((1 << 20) / n) ** (1 / 3))
        return (c + _sphere(gen, 3 * n).view(n, 3, 3) * length).reshape(n, 9).contiguous()
    cells = (n + 1) // 2
    cols = max(1, int(math.sqrt(cells)))
    rows = (cells + cols - 1) // cols
    x = torch.linspace(0, 1, cols + 1, device="cuda")
    y = torch.linspace(0, 1, rows + 1, device="cuda")
    gy, gx = torch.meshgrid(y, x, indexing="ij")
    z = torch.full_like(gx, 0.3)
    for octave in range(5):
        k = 2.0 ** octave * 3
        a = 2 * math.pi * _uniform(gen, 3)
        z = z + 0.08 / 2 ** octave * torch.sin(k * (gx * torch.cos(a[0]) + gy * torch.sin(a[0]))
                                               * 2 + a[1]) * torch.cos(k * gy + a[2])
    p = torch.stack([gx, gy, z], 2)
    a, b, c, d = p[:-1, :-1], p[:-1, 1:], p[1:, 1:], p[1:, :-1]
    tris = torch.stack([torch.stack([a, b, c], 2), torch.stack([a, c, d], 2)], 2)
    return tris.reshape(-1, 9)[:n].contiguous()


def _rays(count, pattern, gen):
    """count x 8 rays.  uniform: origins in the cube, directions on the sphere, unbounded;
    segment: between two points of the cube, as shadow and visibility queries are; camera:
    a pinhole view in raster order."""
    out = torch.empty(count, 8, device="cuda")
    if pattern == "camera":
        width = max(1, int(math.sqrt(count * 4 / 3)))
        i = torch.arange(count, device="cuda")
        jitter = _uniform(gen, count, 2)
        height = max(1, (count + width - 1) // width)
        u = ((i % width) + jitter[:, 0]) / width - 0.5
        v = ((i // width) + jitter[:, 1]) / height - 0.5
        out[:, 0:3] = torch.tensor([0.5, -0.9, 1.1], device="cuda")
        d = torch.stack([u * 0.9, torch.ones_like(u), v * 0.7 - 0.5], 1)
        out[:, 4:7] = d / d.norm(dim=1, keepdim=True)
        out[:, 3] = 0.0
        out[:, 7] = math.inf
        return out
    o = _uniform(gen, count, 3)
    out[:, 0:3] = o
    if pattern == "segment":
        d = _uniform(gen, count, 3) - o
        length = d.norm(dim=1, keepdim=True).clamp(min=1e-6)
        out[:, 4:7] = d / length
        out[:, 3] = 1e-4
        out[:, 7] = length[:, 0]
    else:
        out[:, 4:7] = _sphere(gen, count)
        out[:, 3] = 0.0
        out[:, 7] = math.inf
    return out


def _boxes(case, gen):
    """Boxes of mixed extents, on average about half a neighbour each (a broad phase)."""
    n = case["boxes"]
    c = _uniform(gen, n, 3)
    h = 0.18 * n ** (-1 / 3) * torch.exp(0.4 * torch.randn(n, 3, generator=gen, device="cuda"))
    return torch.cat([c - h, c + h], 1).contiguous()


def _scene_builder(name, width, height, seed):
    if name == "cornell":
        b = S.make_cornell_scene(width, height)
        # The box's light a little brighter or dimmer by seed: the inputs differ.
        f = 1.0 + 0.02 * (seed % 50)
        b.materials[3] = S.emissive((15.0 * f, 14.0 * f, 12.0 * f))
        return b
    if name == "heavy":
        return SC.heavy_render_scene(width, height, seed=seed)
    if name == "soup":
        return SC.soup_scene(width, height, n_tris=1 << 18, seed=seed)
    b = SC.sphere_grid_scene(width, height)
    f = 1.0 + 0.02 * (seed % 50)
    b.materials[1] = S.emissive((10.0 * f, 10.0 * f, 9.0 * f))
    return b


def _sphere_frame(subdivisions, seed):
    """Vertices of a displaced sphere (the deforming mesh of a preview) and its faces."""
    return SC.displaced_sphere(subdivisions, (-0.4, 1.25, 0.6), 0.35, 0.08, seed)


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    st = {"case": case, "ctx": ctx}
    if kind in ("trace", "rebuild", "refit"):
        gen = _generator(seed)
        tris = _triangles(case, gen)
        rays = _rays(case["rays"], case.get("pattern", "segment" if kind == "refit" else "uniform"),
                     gen)
        torch.cuda.synchronize()
        st["bvh"] = ctx.build_lbvh(tris, L.PRIM_TRIANGLES, case.get("bits", 30))
        if kind != "trace":
            # The frame's geometry: the built one jittered (refit) or swept by a wave.
            if kind == "refit":
                move = 1e-4 * torch.randn(tris.shape, generator=gen, device="cuda")
            else:
                move = 0.01 * torch.sin(9.0 * tris.view(-1, 3).roll(1, 1) + _uniform(gen, 1))
            tris = (tris + move.view(tris.shape)).contiguous()
        st["tris"], st["rays"] = tris, rays
        st["hit_id"] = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
        st["hit_t"] = torch.empty(case["rays"], device="cuda")
    elif kind == "overlap":
        boxes = _boxes(case, _generator(seed))
        torch.cuda.synchronize()
        st["bvh"] = ctx.build_lbvh(boxes, L.PRIM_AABBS, case["bits"])
        st["boxes"] = boxes
        st["pairs"] = torch.empty(4 * case["boxes"], 2, dtype=torch.int32, device="cuda")
        st["keys"] = torch.empty(4 * case["boxes"], dtype=torch.int64, device="cuda")
    elif kind == "render":
        st["scene"] = S.Scene(ctx, _scene_builder(case["scene"], case["width"], case["height"], seed))
        st["req"] = S.request(case["width"], case["height"], case["spp"], case["depth"], seed=seed,
                              light_sampler=case["sampler"])
        st["film"] = torch.empty(case["height"], case["width"], 3, device="cuda")
    elif kind == "frame":
        b = S.make_cornell_scene(case["width"], case["height"])
        rough = b.add_material(S.ggx((0.8, 0.55, 0.35), 0.3, 0.0))
        v, idx = _sphere_frame(case["subdivisions"], seed)
        st["mesh"] = b.add_mesh(S.Mesh(v, idx, np.full(len(idx), rough, np.int32)))
        b.add_instance(st["mesh"])
        st["scene"] = S.Scene(ctx, b)
        st["vertices"], _ = _sphere_frame(case["subdivisions"], seed + 1)
        st["req"] = S.request(case["width"], case["height"], case["spp"], case["depth"], seed=seed)
        st["film"] = torch.empty(case["height"], case["width"], 3, device="cuda")
        st["image"] = np.empty((case["height"], case["width"], 3), np.uint8)
    else:
        side = case["side"]
        scenes = [S.Scene(ctx, _scene_builder(n, side, side, seed))
                  for n in ("cornell", "heavy", "soup", "grid")]
        st["server"] = V.Server(scenes, pool_paths=1 << 21)
        st["requests"] = []
        for k, r in enumerate(SC.batched_requests(case["requests"])):
            # The batched workload's requests, their sizes scaled to the case's side.
            w = max(32, r["width"] * side // 1024)
            h = max(32, r["height"] * side // 1024 - 3)
            spp = max(1, r["spp"] * case["spp"] // 256)
            st["requests"].append((r["scene"], S.request(w, h, spp, r["max_depth"], seed=100 * seed + k),
                                   np.zeros((h, w, 3), np.float32)))
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------------ one pass

def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind in ("trace", "rebuild", "refit"):
        bvh = st["bvh"]
        if kind == "rebuild":
            bvh.rebuild(st["tris"])
        elif kind == "refit":
            bvh.refit(st["tris"])
        if case.get("any"):
            return {"hit_id": bvh.trace_any(st["rays"], st["hit_id"])}
        hit_id, hit_t = bvh.trace_closest(st["rays"], st["hit_id"], st["hit_t"])
        return {"hit_id": hit_id, "hit_t": hit_t}
    if kind == "overlap":
        bvh = st["bvh"]
        bvh.rebuild(st["boxes"])
        found = bvh.overlap_self(len(st["pairs"]), st["pairs"])
        # Pairs come in no fixed order; a solver that has to be reproducible sorts them
        # (into a list of fixed room, its rest marked unused).
        with torch.cuda.stream(_shared["stream"]):
            keys = torch.sort(found.pairs.view(torch.int64).view(-1)).values
            st["keys"][:len(keys)] = keys
            st["keys"][len(keys):] = -1
        return {"pairs": st["keys"], "found": found.found_count}
    if kind == "render":
        return {"film": S.render(ctx, st["scene"], st["req"], st["film"])}
    if kind == "frame":
        st["scene"].update_mesh(st["mesh"], st["vertices"])
        S.render(ctx, st["scene"], st["req"], st["film"])
        L._check(ctx._lib.lux_film_encode(ctx.handle, L._ptr(st["film"]), case["width"],
                                          case["height"], case["spp"], 0, L._ptr(st["image"])))
        return {"film": st["film"], "image": st["image"]}
    server = st["server"]
    ids = [server.submit(scene, req, film)[0] for scene, req, film in st["requests"]]
    server.wait_all()
    assert all(server.poll(i) == V.DONE for i in ids)
    return {"films": [film for _, _, film in st["requests"]]}


# ------------------------------------------------------------------------ its work

# Floating-point operations of one box test and one triangle test, and the tests a ray
# makes on average in the library's defined visit order (counted by its own statistics
# calls on these scenes): per extension ray and per shadow segment alike.
_BOX_FLOPS, _TRI_FLOPS, _SHADE_FLOPS = 20, 50, 300
_SCENE_BOXES = {"cornell": 30, "heavy": 67, "grid": 70, "soup": 250}
_SCENE_TRIS = {"cornell": 6, "heavy": 2.5, "grid": 3, "soup": 3}
_SCENE_BYTES = {"cornell": 36 * 36, "heavy": 333000 * 36, "grid": 20480 * 36 + 257 * 64,
                "soup": (1 << 18) * 36}


def _render_work(scene, width, height, spp, depth):
    paths = width * height * spp
    rays = paths * min(depth + 1, 6) * 1.4     # extension rays and shadow segments
    per_ray = (_BOX_FLOPS * _SCENE_BOXES[scene] + _TRI_FLOPS * _SCENE_TRIS[scene] + _SHADE_FLOPS)
    return 12 * width * height + _SCENE_BYTES[scene], rays * per_ray


def work(case):
    kind = case["kind"]
    if kind in ("trace", "rebuild", "refit"):
        n, r = case["tris"], case["rays"]
        boxes = (18 if case["geometry"] == "soup" else 6) * math.log2(n)
        out = 4 if case.get("any") else 8
        return {"bytes": 36 * n + (32 + out) * r,
                "flops": r * (_BOX_FLOPS * boxes + _TRI_FLOPS * 3.4)}
    if kind == "overlap":
        n = case["boxes"]
        return {"bytes": 24 * n + 8 * n, "flops": n * 6 * 4 * math.log2(n)}
    if kind == "render":
        b, f = _render_work(case["scene"], case["width"], case["height"], case["spp"], case["depth"])
        return {"bytes": b, "flops": f}
    if kind == "frame":
        b, f = _render_work("heavy", case["width"], case["height"], case["spp"], case["depth"])
        tris = 20 * 4 ** case["subdivisions"]
        return {"bytes": 15 * case["width"] * case["height"] + 36 * tris, "flops": f}
    total_b = total_f = 0
    for k in range(case["requests"]):
        s = ("cornell", "heavy", "soup", "grid")[k % 4]
        b, f = _render_work(s, case["side"] * 2 // 5, case["side"] * 2 // 5,
                            max(1, case["spp"] // 4), 8)
        total_b, total_f = total_b + b, total_f + f
    return {"bytes": total_b, "flops": total_f}


def tolerance(case):
    """Hits, pairs and bytes are defined exactly (the reference's order of visits and of
    rounded operations), t included.  Films are sums of samples that are defined exactly
    too: the sums may be taken in another order (float32, a few to some hundred terms)."""
    if case["kind"] in ("render", "serve"):
        return {"rel": 1e-5}
    if case["kind"] == "frame":
        return {"rel": 1e-5, "differ": 0.0}
    return "exact"


# ------------------------------------------------------------------------ in 64 bits

def exact(case, seed):
    """Closest-hit distances by testing every ray against every triangle in float64 (hit
    ids have no value here: equal distances are told apart by the order of visits).  None
    for the other paths (Monte Carlo films follow 32-bit random walks) and where the
    pairs are too many."""
    if case["kind"] not in ("trace", "rebuild", "refit") or case.get("any"):
        return None
    n, r = case["tris"], case["rays"]
    if n * r > 1 << 33:
        return None
    st = prepare(case, seed)
    tri = st["tris"].double().view(n, 3, 3)
    rays = st["rays"].double()
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    out = torch.empty(r, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 25) // n)
    for i in range(0, r, step):
        o, d = rays[i:i + step, None, 0:3], rays[i:i + step, None, 4:7]
        h = torch.linalg.cross(d.expand(-1, n, 3), e2[None].expand(d.shape[0], -1, -1))
        a = (e1 * h).sum(2)
        f = 1.0 / a
        s = o - v0
        u = f * (s * h).sum(2)
        q = torch.linalg.cross(s, e1[None].expand(d.shape[0], -1, -1))
        w = f * (d * q).sum(2)
        t = f * (e2 * q).sum(2)
        ok = (a.abs() >= 1e-7) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1)
        ok &= (t > rays[i:i + step, 3:4]) & (t < rays[i:i + step, 7:8])
        out[i:i + step] = torch.where(ok, t, math.inf).amin(1)
    return {"hit_id": None, "hit_t": out}
