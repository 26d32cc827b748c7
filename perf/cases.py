"""What a program does with this renderer, as cases to be timed.

A case goes through the public interface of ray-tracer_b200/rtg.py: renders (one
pass or progressive), batches, served previews, ray queries and cold scenes. A
program keeps one Context for each way it works, so the contexts here live as long
as the process; a state keeps the scenes it uploaded.

Scenes are those of workloads.py. The seed of a state moves the camera, turns or
shifts some of the objects and seeds the samples, so another seed is another scene
of the same kind and size.
"""
import json
import math
import os
import sys

import numpy as np

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ray-tracer_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import rtg  # noqa: E402
import workloads  # noqa: E402

TUNED_POOL = 1 << 23  # what rtg_autotune picks for large work on a B200


def listed():
    return [
        # Renders on a context as it is created.
        # An interactive preview of a small room: the smallest whole call, image and all.
        _render("preview_128", "cornell", 128, 128, 4, 4, out="image"),
        # The Cornell box of the benchmark (C1), in one pass.
        _render("cornell_256x64", "cornell", 256, 256, 64, 8),
        # A render with the settings a scene file gets by default (640x360, 64 spp, depth 8, progressive passes).
        _render("default_640x360", "spheres", 640, 360, 64, 8, progressive=True),
        # Multiple importance sampling at an odd size, progressive.
        _render("cornell_mis_odd", "cornell", 333, 217, 48, 8, progressive=True, mis=True),
        # The Whitted-style integrator on glass and metal meshes.
        _render("direct_640x360", "mesh", 640, 360, 16, 8, integrator="direct"),
        # Final renders, one at a time, with the pool the autotuner picks: the benchmark's sphere field (C2)
        # and its mesh of 174k triangles (C3).
        _render("spheres_512x128", "spheres", 512, 512, 128, 16, pool="tuned"),
        _render("mesh_1024x64", "mesh", 1024, 1024, 64, 12, pool="tuned"),
        # A batch of uneven scenes (16 of the benchmark's mix), progressive, with their images: the largest case.
        {"name": "batch_mix16", "kind": "batch", "first": 16, "scenes": 16, "pool": "tuned"},
        # A server's previews: 24 requests over 8 resident scenes, submitted together and read back.
        {"name": "serve_previews", "kind": "serve", "scenes": 8, "previews": 24, "size": 128, "spp": 4, "depth": 4},
        # A scene that is not resident: its JSON text in, a preview of it out (time to first picture).
        {"name": "cold_mesh", "kind": "cold", "subdivisions": 6, "segments": 256, "size": 128, "spp": 4, "depth": 4},
        # Ray queries on host arrays: a bake or a visibility study (many rays, a large mesh) and picking or
        # collision queries (a few thousand rays, closest hit and occlusion).
        {"name": "rays_mesh_1m", "kind": "rays", "scene": "mesh", "rays": 1_000_000},
        {"name": "rays_spheres_20k", "kind": "rays", "scene": "spheres", "rays": 20_011},
    ]


def _render(name, scene, width, height, spp, depth, progressive=False, mis=False, integrator="path", pool="default",
            out="mean"):
    return {"name": name, "kind": "render", "scene": scene, "width": width, "height": height, "spp": spp,
            "depth": depth, "progressive": progressive, "mis": mis, "integrator": integrator, "pool": pool,
            "out": out}


def draw(rng):
    """Another case of the same ranges; sizes are odd as often as not."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["render"] * 6 + ["batch", "serve", "cold", "rays", "rays"])
    if kind == "rays":
        scene = rng.choice(["cornell", "spheres", "mesh"])
        return {"kind": "rays", "scene": scene, "rays": log_int(1000, 1_000_000 if scene == "mesh" else 200_000)}
    if kind == "cold":
        return {"kind": "cold", "subdivisions": rng.randint(3, 6), "segments": log_int(24, 256),
                "size": log_int(64, 256), "spp": rng.choice([1, 4, 8]), "depth": rng.randint(3, 8)}
    if kind == "serve":
        return {"kind": "serve", "scenes": rng.randint(2, 8), "previews": rng.randint(4, 48), "size": log_int(64, 192),
                "spp": rng.randint(1, 8), "depth": rng.randint(3, 8)}
    if kind == "batch":
        return {"kind": "batch", "first": rng.randint(17, 29), "scenes": rng.randint(2, 8),
                "pool": rng.choice(["default", "tuned"])}
    scene = rng.choice(["cornell", "spheres", "mesh"])
    width = log_int(64, 1024)
    height = max(16, int(width * rng.uniform(0.5, 1.0)))
    integrator = rng.choice(["path"] * 5 + ["direct", "normals"])
    # A drawn render has at most as many samples as mesh_1024x64.
    spp = min(log_int(1, 256), max(1, (1 << 26) // (width * height)))
    if integrator == "direct":
        spp = min(spp, 16)
    case = _render("", scene, width, height, spp, rng.randint(3, 16), progressive=rng.random() < 0.5,
                   mis=integrator == "path" and rng.random() < 0.2, integrator=integrator,
                   pool=rng.choice(["default", "tuned"]), out=rng.choice(["mean", "image"]))
    del case["name"]
    return case


# ---------------------------------------------------------------------------
# Scenes

def _moved(scene, seed):
    """The same kind of scene with another camera position, other object positions and other samples."""
    rng = np.random.default_rng([seed, 77])
    cam = scene["camera"]
    look_from, look_at = np.array(cam["look_from"], float), np.array(cam["look_at"], float)
    dist = float(np.linalg.norm(look_from - look_at))
    cam["look_from"] = [float(x) for x in look_from + 0.02 * dist * rng.uniform(-1, 1, 3)]
    for o in scene["objects"]:
        if o["type"] in ("box", "mesh"):
            o["rotate_y"] = float(o.get("rotate_y", 0.0) + rng.uniform(-5, 5))
        elif o["type"] == "sphere" and o["radius"] < 0.5:
            o["center"] = [float(o["center"][0] + rng.uniform(-0.02, 0.02)), o["center"][1],
                           float(o["center"][2] + rng.uniform(-0.02, 0.02))]
    scene["render"]["seed"] = int(rng.integers(1, 1 << 30))
    return scene


def _scene(kind, seed, subdivisions=6, segments=256):
    if kind == "cornell":
        return _moved(workloads.cornell(), seed)
    if kind == "spheres":
        return _moved(workloads.sphere_field(), seed)
    mesh = workloads.mesh_stress()
    for o in mesh["objects"]:
        if o.get("source") == "icosphere":
            o["subdivisions"] = subdivisions
        elif o.get("source") == "torus":
            o["segments"], o["segments_v"] = segments, max(3, segments * 180 // 256)
    return _moved(mesh, seed)


_contexts = {}


def _context(pool):
    """The program's context for this way of working, made on first use and kept."""
    if pool not in _contexts:
        c = rtg.Context(0)
        if pool == "tuned":
            c.set_tuning(pool_paths=TUNED_POOL)
        if pool == "serve":
            c.serve_prepare()
        _contexts[pool] = c
    return _contexts[pool]


class _State:
    """A case, its context and the scenes it keeps resident."""

    def __init__(self, case, ctx):
        self.case, self.ctx, self.ids, self.settings, self.options, self.data = case, ctx, [], [], None, None

    def add(self, scene):
        host = rtg.parse_scene(json.dumps(scene), None, "auto")
        self.ids.append(self.ctx.upload(host))
        self.settings.append(self.ctx.scene_settings(self.ids[-1]))

    def __del__(self):
        for i in self.ids:
            self.ctx.release(i)


# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "render":
        st = _State(case, _context(case["pool"]))
        st.add(_scene(case["scene"], seed))
        s = st.settings[0]
        s.width, s.height, s.spp, s.max_depth = case["width"], case["height"], case["spp"], case["depth"]
        s.integrator, s.mis = case["integrator"], case["mis"]
        s.rr_min_depth = min(s.rr_min_depth, s.max_depth)
        st.options = rtg.RenderOptions(progressive=case["progressive"], max_pass_spp=32)
    elif kind == "batch":
        st = _State(case, _context(case["pool"]))
        for k in range(case["first"], case["first"] + case["scenes"]):
            st.add(_moved(workloads.mix_scene(k), seed + k))
        st.options = rtg.RenderOptions(progressive=True, max_pass_spp=32)
    elif kind == "serve":
        st = _State(case, _context("serve"))
        for k in range(case["scenes"]):
            st.add(_moved(workloads.mix_scene(k), seed + k))
        for s in st.settings:
            s.width, s.height, s.spp, s.max_depth = case["size"], case["size"], case["spp"], case["depth"]
            s.rr_min_depth = min(s.rr_min_depth, s.max_depth)
        st.options = rtg.RenderOptions(progressive=False)
    elif kind == "cold":
        st = _State(case, _context("default"))
        scene = _scene("mesh", seed, case["subdivisions"], case["segments"])
        scene["render"] |= {"width": case["size"], "height": case["size"], "spp": case["spp"],
                            "max_depth": case["depth"]}
        st.data = json.dumps(scene)
        st.options = rtg.RenderOptions(progressive=False)
    else:
        st = _State(case, _context("default"))
        scene = _scene(case["scene"], seed)
        st.add(scene)
        st.data = _rays(case, seed)
    return st


#: Bounds of the three scenes that rays start from (1.2 times the objects').
_BOUNDS = {"cornell": ((-50, -50, -50), (610, 610, 610)), "spheres": ((-13, 0.01, -13), (13, 3, 13)),
           "mesh": ((-7, -0.8, -5), (7, 8.8, 7))}


def _rays(case, seed):
    """Random rays over the scene's bounds, 1% of them parallel to an axis: (o, tmin, d, tmax) as float32."""
    rng = np.random.default_rng([seed, 5])
    n = case["rays"]
    lo, hi = (np.array(b, float) for b in _BOUNDS[case["scene"]])
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    axis = np.nonzero(rng.random(n) < 0.01)[0]
    d[axis] = np.eye(3)[rng.integers(0, 3, len(axis))] * rng.choice([-1.0, 1.0], size=(len(axis), 1))
    rays = np.empty((n, 8), np.float32)
    rays[:, 0:3] = rng.uniform(lo, hi, size=(n, 3))
    rays[:, 3] = 1e-6
    rays[:, 4:7] = d
    rays[:, 7] = 3.0e38
    return rays


def run(state):
    case, ctx = state.case, state.ctx
    kind = case["kind"]
    if kind == "render":
        s = state.settings[0]
        r = rtg.Renderer(ctx, state.ids[0], s, state.options)
        r.render()
        return r.image() if case["out"] == "image" else r.framebuffer_mean()
    if kind == "batch":
        ctx.render_batch(state.ids, state.settings, state.options)
        return ctx.images(range(len(state.ids)), [(s.width, s.height) for s in state.settings])
    if kind == "serve":
        open_ = []
        for k in range(case["previews"]):
            j = k % len(state.ids)
            open_.append(ctx.submit(state.ids[j], state.settings[j], state.options, 0))
        images = {}
        while len(images) < len(open_):
            for rid, p in ctx.pump(2.0, return_on_event=True):
                if p.finished:
                    images[rid] = ctx.request_image(rid, case["size"], case["size"])
                    ctx.release_request(rid)
        return [images[rid] for rid in open_]
    if kind == "cold":
        sid = ctx.upload(rtg.parse_scene(state.data, None, "auto"))
        r = rtg.Renderer(ctx, sid, None, state.options)
        r.render()
        image = r.image()
        ctx.release(sid)
        return image
    t, prim, plane, bary = ctx.trace_closest(state.ids[0], state.data)
    return {"t": t, "prim": prim, "plane": plane, "bary": bary, "occluded": ctx.trace_any(state.ids[0], state.data)}


# ---------------------------------------------------------------------------

#: Of each scene: closest-hit and shadow rays a sample, binary tree nodes and primitive tests a ray (measured
#: with the renderer's own counters on workloads.py's scenes), and bytes of its tree and primitives.
_COST = {"cornell": (4.5, 7, 5, 6e3), "spheres": (2.4, 8, 4, 9e4), "mesh": (3.9, 13.9, 6.5, 2.5e7),
         "mix": (2.7, 6.4, 3.9, 1.6e6)}
#: Two slab tests of a node (12 FMAs, 20 minima and maxima), a primitive test, and the rest of a ray's work.
_NODE, _PRIM, _RAY = 44, 60, 120


def _flops(scene, rays):
    _, nodes, prims, _ = _COST[scene]
    return rays * (nodes * _NODE + prims * _PRIM + _RAY)


def work(case):
    kind = case["kind"]
    if kind == "rays":
        n = case["rays"]
        # Both queries read 32 bytes a ray; they return 20 bytes and 1 byte.
        return {"bytes": n * (2 * 32 + 21) + _COST[case["scene"]][3], "flops": _flops(case["scene"], 2 * n)}
    if kind == "cold":
        triangles = 20 * 4 ** case["subdivisions"] + 2 * case["segments"] * max(3, case["segments"] * 180 // 256)
        rays = case["size"] ** 2 * case["spp"] * 2.5
        # Each triangle's record, normals, boxes and nodes are written and read once; about 20 levels of binning.
        return {"bytes": triangles * 2 * 250 + case["size"] ** 2 * 3, "flops": triangles * 20 * 60 + _flops("mesh", rays)}
    if kind == "serve":
        px = case["previews"] * case["size"] ** 2
        return {"bytes": px * 3 + case["scenes"] * _COST["mix"][3], "flops": _flops("mix", px * case["spp"] * 2.2)}
    if kind == "batch":
        px = samples = 0
        for k in range(case["first"], case["first"] + case["scenes"]):
            r = workloads.mix_scene(k)["render"]
            px += r["width"] * r["height"]
            samples += r["width"] * r["height"] * r["spp"]
        return {"bytes": px * 3 + case["scenes"] * _COST["mix"][3],
                "flops": _flops("mix", samples * _COST["mix"][0])}
    px = case["width"] * case["height"]
    rays = 1.0 if case["integrator"] == "normals" else min(_COST[case["scene"]][0], 2.0 * case["depth"])
    return {"bytes": px * (24 if case["out"] == "mean" else 3) + _COST[case["scene"]][3],
            "flops": _flops(case["scene"], px * case["spp"] * rays)}


def exact(case, seed):
    """Distances of the ray queries on the sphere field in 64 bits. The other cases have no such value: a path
    draws its decisions from its own results, so 64-bit paths part from 32-bit ones, images are bytes, and
    rays against the meshes take too long without a tree."""
    if case["kind"] != "rays" or case["scene"] != "spheres":
        return None
    scene = _scene("spheres", seed)
    rays = _rays(case, seed).astype(np.float64)
    spheres = np.array([[*o["center"], o["radius"]] for o in scene["objects"] if o["type"] == "sphere"])
    n = len(rays)
    best = np.full(n, np.inf)
    for at in range(0, n, 4096):
        o, tmin, d = rays[at:at + 4096, 0:3], rays[at:at + 4096, 3], rays[at:at + 4096, 4:7]
        with np.errstate(divide="ignore", invalid="ignore"):
            t = -o[:, 1] / d[:, 1]  # the ground plane y = 0
            near = np.where((np.abs(d[:, 1]) > 1e-12) & (t > tmin), t, np.inf)
            a = np.sum(d * d, 1)[:, None]
            oc = spheres[None, :, :3] - o[:, None, :]
            h = np.einsum("rk,rsk->rs", d, oc)
            r = spheres[None, :, 3]
            perp = oc - (h / a)[..., None] * d[:, None, :]
            disc = a * (r * r - np.sum(perp * perp, 2))
            q = h + np.copysign(np.sqrt(disc), h)
            roots = np.stack([(np.sum(oc * oc, 2) - r * r) / q, q / a])
            roots = np.where((disc >= 0) & (roots > tmin[None, :, None]), roots, np.inf)
            best[at:at + 4096] = np.minimum(near, roots.min(axis=(0, 2)))
    return {"t": np.where(np.isfinite(best), best, 0.0), "prim": None, "plane": None, "bary": None, "occluded": None}
