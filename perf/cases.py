"""What a program that uses this framework has it do: the calls whose time matters.

A case is a session (scene, image size, samples, depth, launch fields) and one pass through its
public calls: a rendered frame with its readback, a pick, a block of ray queries, a batched
frame, a mesh swapped in. Scenes are the generated configurations 0-3 (Cornell box, spheres,
environment-lit mesh, slit room) at the sizes this repository's configurations, tests and
benchmark use; `level` is the icosphere level of a scene's mesh (20 * 4^level triangles).

Launch fields of a case ("width" ... "fuse_camera") are those that pt_autotune chooses and a
program then keeps; a case without them runs the library's defaults.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("gpu-pathed_b200"))
import pathed  # noqa: E402

# Camera + continuation + contributing shadow rays per path at the configurations' own depths
# (device counters): what an estimate of a frame's work is scaled by.
RAYS_PER_PATH = {0: 6.0, 1: 2.8, 2: 1.6, 3: 13.4}
DEPTH = {0: 5, 1: 8, 2: 6, 3: 10}

LAUNCH = ("block", "sort_materials", "sort_rays", "speculate", "split_shade", "shadow_order", "fuse_camera")


def listed():
    return [
        # a cursor dragged over the image: one pick per mouse event (the reference GUI's hitTest)
        {"name": "pick_drag", "kind": "pick", "config": 1, "level": -1, "w": 400, "h": 400, "n": 16},
        # the GUI's interactive view: camera moved, one sample per pixel, the display buffer read
        {"name": "preview_cornell", "kind": "preview", "config": 0, "level": -1, "w": 400, "h": 400, "spp": 1, "depth": 5},
        # configuration 0 as it stands, default launch fields
        {"name": "cornell_512", "kind": "frame", "config": 0, "level": -1, "w": 512, "h": 512, "spp": 16, "depth": 5},
        # configuration 1, the benchmark's workload, with the fields the autotuner picks for it
        {"name": "spheres_1024", "kind": "frame", "config": 1, "level": -1, "w": 1024, "h": 1024, "spp": 64, "depth": 8,
         "width": 4, "leaf": 8, "builder": 2, "sort_materials": 1, "split_shade": 2, "shadow_order": 1, "fuse_camera": 1},
        # configuration 2, the 1.31M-triangle mesh under the environment map, tuned
        {"name": "mesh_1080p", "kind": "frame", "config": 2, "level": 8, "w": 1920, "h": 1080, "spp": 32, "depth": 6,
         "width": 4, "leaf": 8, "block": 256, "split_shade": 3, "speculate": 3},
        # configuration 3, the slit room, tuned: the largest frame
        {"name": "slit_room_1024", "kind": "frame", "config": 3, "level": 8, "w": 1024, "h": 1024, "spp": 16, "depth": 10,
         "width": 4, "leaf": 2, "block": 256, "sort_materials": 1, "sort_rays": 1, "split_shade": 1, "speculate": 3},
        # progressive refinement at a ragged window size, without emitter sampling, defaults
        {"name": "progressive_odd", "kind": "frame", "config": 3, "level": 5, "w": 777, "h": 431, "spp": 3, "depth": 7,
         "nee": False, "frames": 2},
        # one guided frame of a running render: guide inference, sample collection, training
        {"name": "guided_slit", "kind": "guided", "config": 3, "level": 6, "w": 1024, "h": 1024, "spp": 1, "depth": 10},
        # closest-hit queries of a host program against a large mesh
        {"name": "trace_1m", "kind": "trace", "config": 2, "level": 7, "n": 1000003},
        # visibility queries in a closed room
        {"name": "occluded_200k", "kind": "occluded", "config": 3, "level": 6, "n": 200000},
        # several scenes of uneven size in one frame
        {"name": "batch_6", "kind": "batch", "scenes": 6, "draw": 11, "max_level": 6, "max_res": 512, "max_spp": 16},
        # a mesh replaced in a running session (device-built tree) and its first image
        {"name": "swap_mesh", "kind": "swap", "config": 0, "level": 6, "w": 512, "h": 512, "spp": 1, "depth": 5, "builder": 1},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _frame_size(rng, cost, most):
    """A ragged image size and spp whose paths times `cost` stay within `most`."""
    while True:
        w, h, spp = _log(rng, 64, 1920), _log(rng, 64, 1080), _log(rng, 1, 64)
        if w * h * spp * cost <= most:
            return w, h, spp


def draw(rng):
    kind = rng.choice(["frame"] * 8 + ["preview", "pick", "guided", "trace", "trace", "occluded", "batch", "swap"])
    config = rng.randrange(4)
    level = rng.randint(3, 8) if config >= 2 else -1
    if kind == "frame":
        depth = rng.randint(1, 10)
        w, h, spp = _frame_size(rng, RAYS_PER_PATH[config], 1024 * 1024 * 16 * 13.4 / 2)
        c = {"kind": kind, "config": config, "level": level, "w": w, "h": h, "spp": spp, "depth": depth,
             "nee": rng.random() < 0.85, "frames": rng.choice([1, 1, 2])}
        if rng.random() < 0.6:  # fields the autotuner chooses among
            c.update({"width": rng.choice([2, 4, 4, 8]), "leaf": rng.choice([2, 4, 8, 16]), "builder": rng.choice([0, 0, 1, 2]),
                      "block": rng.choice([128, 256]), "sort_materials": rng.choice([1, 2]), "sort_rays": rng.choice([1, 2]),
                      "speculate": rng.choice([1, 2, 3, 4]), "split_shade": rng.choice([1, 2, 3]),
                      "shadow_order": rng.choice([1, 2]), "fuse_camera": rng.choice([1, 2])})
        option = rng.random()  # the session options that change what a frame runs
        if option < 0.08:
            c["watertight"] = True
        elif option < 0.16:
            c["quantized"] = True
        elif option < 0.24:
            c["normals"] = True
        return c
    if kind == "preview":
        return {"kind": kind, "config": rng.randrange(2), "level": -1, "w": _log(rng, 128, 1280), "h": _log(rng, 128, 1080),
                "spp": rng.choice([1, 1, 2, 3]), "depth": rng.randint(1, 10)}
    if kind == "pick":
        return {"kind": kind, "config": 1, "level": -1, "w": _log(rng, 200, 1920), "h": _log(rng, 200, 1080), "n": rng.randint(8, 40)}
    if kind == "guided":
        return {"kind": kind, "config": rng.choice([2, 3]), "level": rng.randint(3, 6), "w": _log(rng, 256, 1024),
                "h": _log(rng, 256, 1024), "spp": rng.randint(1, 3), "depth": rng.randint(4, 10)}
    if kind == "trace":
        return {"kind": kind, "config": config, "level": min(level, 7), "n": _log(rng, 33, 2000000), "width": rng.choice([2, 4, 4, 8])}
    if kind == "occluded":
        return {"kind": kind, "config": config, "level": min(level, 7), "n": _log(rng, 33, 2000000)}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 8), "draw": rng.randrange(1 << 20), "max_level": 5, "max_res": 512,
                "max_spp": rng.choice([4, 8, 16])}
    return {"kind": kind, "config": rng.randrange(2), "level": rng.randint(3, 6), "w": _log(rng, 128, 1024),
            "h": _log(rng, 128, 1024), "spp": 1, "depth": rng.randint(2, 8), "builder": rng.choice([1, 2])}


def _image(c, channels=3):
    """A page-locked image, as a program that reads every frame back keeps."""
    return torch.empty((c["h"], c["w"], channels), dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()


def _session(c, seed):
    s = pathed.Session(c.get("w", 64), c.get("h", 64))
    if "builder" in c:
        s.set_bvh_builder(c["builder"])
    if "width" in c:
        s.set_bvh(c["width"], c.get("leaf", 4))
    if c.get("quantized"):
        s.set_bvh_quantized(True)
    if c.get("watertight"):
        s.set_watertight(True)
    launch = {k: c[k] for k in LAUNCH if k in c}
    if "block" in launch:
        launch["block_extend"] = launch["block_shadow"] = launch.pop("block")
    if launch:
        s.set_launch(**launch)
    return s


def _scene(c, seed):
    s = _session(c, seed)
    s.load_config(c["config"], 1 + seed, None if c["level"] < 0 else c["level"])
    s.set_seed(1 + seed)
    if "depth" in c:
        s.set_max_depth(c["depth"])
    if "nee" in c:
        s.set_nee(c["nee"])
    if c.get("normals"):
        s.set_renderer(pathed.RENDERER_NORMALS)
    return s


def _look(c, rng):
    """A camera of a user who moves around the scene."""
    r, y, at = ((3.75, 1.0, 1.0) if c["config"] == 0 else (17.0, 6.0, 0.5))
    a = rng.uniform(-0.12, 0.12)
    origin = (r * math.sin(a), y + rng.uniform(-0.2, 0.2), r * math.cos(a))
    return origin, (0.0, at, 0.0), (0.0, 1.0, 0.0), 40.0 / 180.0 * math.pi


def _rays(c, seed):
    """Queries of a host program: from a camera into the scene, and from points inside the
    scene's bounds in all directions, as its secondary rays would leave."""
    g = torch.Generator().manual_seed(seed + 77)
    n = c["n"]
    eye, half = {0: ((0, 1, 3.75), 1.0), 1: ((0, 6, 17), 8.0), 2: ((0, 0.45, 3.1), 1.2), 3: ((0.3, 0.9, 2.3), 2.4)}[c["config"]]
    mid = torch.tensor([0.0, {0: 1.0, 1: 4.0, 2: 0.0, 3: 0.8}[c["config"]], 0.0])
    inside = mid + half * (2 * torch.rand(n, 3, generator=g) - 1)
    primary = (torch.arange(n) % 3 == 0)[:, None]
    eye = torch.tensor(eye).expand(n, 3)
    free = torch.randn(n, 3, generator=g)
    o = torch.where(primary, eye, inside)
    d = torch.where(primary, inside - eye, free)
    return o.float().contiguous().numpy(), torch.nn.functional.normalize(d.float(), dim=1).contiguous().numpy()


def _batch_specs(c, seed):
    specs = pathed.batch_generate(c["draw"], c["scenes"])
    for k, b in enumerate(specs):
        b["seed"] = 1 + seed + 101 * k
        b["level"] = min(b["level"], c["max_level"])
        b["width"] = b["height"] = min(b["width"], c["max_res"])
        b["spp"] = min(b["spp"], c["max_spp"])
        b["guided"] = 0
    return specs


def prepare(case, seed):
    c, kind = case, case["kind"]
    rng = random.Random(seed)
    st = {"case": c}
    if kind == "batch":
        s = pathed.Session(64, 64)
        s.load_batch(_batch_specs(c, seed))
        s.set_seed(1 + seed)
    elif kind == "swap":
        src = pathed.Session(8, 8)
        src.load_config(c["config"], 1 + seed, c["level"])
        a = src.export_scene()
        src.close()
        st["arrays"] = {k: a[k] for k in ("tri_vertices", "tri_normals", "tri_materials", "spheres", "sphere_materials",
                                          "material_types", "material_albedo", "material_emit", "material_ior",
                                          "material_alpha") if a[k].size}
        s = _session(c, seed)
        s.load_config(c["config"], 1 + seed)
        s.set_max_depth(c["depth"])
        st["look"] = _look(c, rng)
        st["out"] = _image(c)
    else:
        s = _scene(c, seed)
    st["session"] = s
    if kind in ("frame", "guided"):
        st["out"] = _image(c)
    if kind in ("preview", "pick"):
        st["look"] = _look(c, rng)
        s.set_camera(*st["look"])
    if kind == "pick":
        x0, y0, x1, y1 = (rng.randrange(v) for v in (c["w"], c["h"], c["w"], c["h"]))
        st["at"] = [(x0 + (x1 - x0) * k // c["n"], y0 + (y1 - y0) * k // c["n"]) for k in range(c["n"])]
    if kind in ("trace", "occluded"):
        st["o"], st["d"] = _rays(c, seed)
        st["tmin"] = np.full(c["n"], 1e-4, np.float32)
        st["tmax"] = np.full(c["n"], 3.4e38 if kind == "trace" else 1.5, np.float32)
    if kind == "guided":
        # a running guided render late in its schedule: sampling from the network, few and small steps
        s.set_guide_options(steps_per_frame=4, lr=1e-4, warmup_steps=0)
        s.set_guiding(True)
        st["params"] = s.guide_params()
    # the session has shown something before the pass that counts: its scene is on the device
    if kind in ("frame", "preview", "guided", "batch", "swap"):
        s.render(1)
    else:
        s.hit_test(0, 0) if kind == "pick" else s.trace_rays(st["o"][:1], st["d"][:1], 1e-4, 3.4e38)
    return st


def run(st):
    c, s = st["case"], st["session"]
    kind = c["kind"]
    if kind == "frame":
        s.reset()
        for _ in range(c.get("frames", 1)):
            s.render(c["spp"])
        return s.readback(st["out"])
    if kind == "preview":
        s.set_camera(*st["look"])
        s.render(c["spp"])
        return s.readback_rgba8()
    if kind == "pick":
        return np.array([s.hit_test(x, y) for x, y in st["at"]], np.int32)
    if kind == "guided":
        s.set_guide_params(st["params"])
        s.reset()
        s.render(c["spp"])
        return {"image": s.readback(st["out"]), "params": s.guide_params()}
    if kind == "trace":
        return s.trace_rays(st["o"], st["d"], st["tmin"], st["tmax"], with_bary=True)
    if kind == "occluded":
        return s.occluded(st["o"], st["d"], st["tmin"], st["tmax"])
    if kind == "batch":
        s.reset()
        s.render(1)
        return [s.batch_readback(k) for k in range(c["scenes"])]
    s.load_arrays(**st["arrays"])
    s.set_camera(*st["look"])
    s.render(c["spp"])
    return s.readback(st["out"])


def _prims(config, level):
    base = {0: 36, 1: 70, 2: 0, 3: 2002}[config]
    return base + (20 * 4 ** level if level >= 0 else 0)


def _query_flops(prims):
    """One query that finds its hit with no detour: a box test per level of a binary tree (two
    children, 13 operations each) and one primitive test."""
    return 26.0 * max(1.0, math.log2(prims)) + 50.0


def work(case):
    """Scene and inputs read once, results written once; per ray a direct descent of the tree
    and the shading of its vertex (about 150 operations)."""
    c, kind = case, case["kind"]
    if kind == "batch":
        by = fl = 0.0
        for b in _batch_specs(c, 0):
            p = _prims(b["config"], b["level"])
            paths = b["width"] * b["height"] * b["spp"]
            rays = paths * RAYS_PER_PATH[b["config"]] * min(1.0, b["max_depth"] / DEPTH[b["config"]])
            by += 72.0 * p + 12.0 * b["width"] * b["height"]
            fl += rays * (_query_flops(p) + 150.0)
        return {"bytes": by, "flops": fl}
    p = _prims(c["config"], c["level"])
    if kind in ("trace", "occluded"):
        return {"bytes": 36.0 * p + c["n"] * (32.0 + (24.0 if kind == "trace" else 4.0)), "flops": c["n"] * _query_flops(p)}
    if kind == "pick":
        return {"bytes": 16.0 * p + 12.0 * c["n"], "flops": c["n"] * _query_flops(p)}
    pixels = c["w"] * c["h"] * c.get("frames", 1)
    rays_per_path = 1.0 if c.get("normals") else max(1.0, RAYS_PER_PATH[c["config"]] * min(1.0, c["depth"] / DEPTH[c["config"]]))
    rays = pixels * (1 if c.get("normals") else c["spp"]) * rays_per_path
    by = 72.0 * p + (4.0 if kind == "preview" else 12.0) * pixels
    fl = rays * (_query_flops(p) + 150.0)
    if kind == "guided":  # network inference per vertex, four training steps of 2^16 samples
        fl += rays / 2 * 31744.0 + 4 * 65536 * 3 * 31744.0
        by += 4 * 4 * 16104.0
    return {"bytes": by, "flops": fl}


def exact(case, seed):
    """Distances and barycentric coordinates of closest-hit queries in 64 bits, every primitive
    against every ray (where that is quick). A path-traced image has no such value: each pixel is
    a sum over random paths whose branches flip with the last bit of a variate. Ids are whole
    numbers, and equal."""
    c = case
    if c["kind"] != "trace" or c["n"] * _prims(c["config"], c["level"]) > 3e10:
        return None
    s = pathed.Session(8, 8)
    s.load_config(c["config"], 1 + seed, None if c["level"] < 0 else c["level"])
    a = s.export_scene()
    s.close()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    o, d = (torch.from_numpy(v).to(dev).double() for v in _rays(c, seed))
    tri = torch.from_numpy(a["tri_vertices"]).to(dev).double().reshape(-1, 3, 3)
    sph = torch.from_numpy(a["spheres"]).to(dev).double().reshape(-1, 4)
    tmin, inf = float(np.float32(1e-4)), float("inf")
    out_t, out_b = torch.zeros(c["n"], device=dev).double(), torch.zeros(c["n"], 2, device=dev).double()
    chunk = max(1, min(c["n"], int(6e7) // max(1, tri.shape[0] + sph.shape[0])))
    for at in range(0, c["n"], chunk):
        ro, rd = o[at:at + chunk, None], d[at:at + chunk, None]
        best = torch.full((ro.shape[0],), inf, device=dev).double()
        bary = torch.zeros(ro.shape[0], 2, device=dev).double()
        if len(tri):
            p0, e1, e2 = tri[None, :, 0], tri[None, :, 1] - tri[None, :, 0], tri[None, :, 2] - tri[None, :, 0]
            dot = lambda x, y: x[..., 0] * y[..., 0] + x[..., 1] * y[..., 1] + x[..., 2] * y[..., 2]  # noqa: E731
            cross = lambda x, y: torch.stack([x[..., 1] * y[..., 2] - x[..., 2] * y[..., 1],  # noqa: E731
                                              x[..., 2] * y[..., 0] - x[..., 0] * y[..., 2],
                                              x[..., 0] * y[..., 1] - x[..., 1] * y[..., 0]], -1)
            s1, r = cross(rd, e2), ro - p0
            inv = 1.0 / dot(s1, e1)
            s2 = cross(r, e1.expand_as(r))
            b1, b2, t = dot(r, s1) * inv, dot(rd, s2) * inv, dot(e2.expand_as(s2), s2) * inv
            t = torch.where((b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= tmin), t, inf)
            best, k = t.min(1)
            bary = torch.stack([b1.gather(1, k[:, None])[:, 0], b2.gather(1, k[:, None])[:, 0]], 1)
            del s1, r, s2, b1, b2, t, inv
        if len(sph):
            oc = ro - sph[None, :, :3]
            b, q = (oc * rd).sum(-1), (oc * oc).sum(-1) - sph[None, :, 3] ** 2
            dd = (rd * rd).sum(-1)
            root = torch.sqrt(torch.clamp(b * b - dd * q, min=0.0))
            near, far = (-b - root) / dd, (-b + root) / dd
            ts = torch.where(near > tmin, near, far)
            ts = torch.where((b * b - dd * q > 0) & (ts > tmin), ts, inf).min(1).values
            bary = torch.where((ts < best)[:, None], torch.zeros_like(bary), bary)
            best = torch.minimum(best, ts)
        hit = torch.isfinite(best)
        out_t[at:at + chunk] = torch.where(hit, best, 0.0)
        out_b[at:at + chunk] = torch.where(hit[:, None], bary, torch.zeros_like(bary))
    return {"prim_type": None, "prim_id": None, "mat_id": None, "t": out_t, "bary": out_b}
