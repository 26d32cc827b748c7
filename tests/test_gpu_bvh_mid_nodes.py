"""GPU BVH build: nodes that one block builds (33 to 1,024 primitives), and the level
passes above them, give the host build's layout byte for byte at the edges of both
ranges, with teams of warps on a node and without, and down to the depth cap."""
import json

import numpy as np
import pytest

import rtg

pytestmark = pytest.mark.gpu

PARTS = ["roots", "nodes", "nodes4", "prims", "slot_material", "slot_normals", "slot_prim"]


def _points(kind, n):
    rng = np.random.default_rng(n)
    if kind == "uniform":
        return rng.uniform(-5, 5, (n, 3))
    if kind == "sorted":  # 32 neighbours in the input are neighbours in space
        return np.sort(rng.uniform(-5, 5, (n, 1)), axis=0) * [1.0, 0.0, 0.0]
    if kind == "clusters":
        return rng.integers(-2, 3, (n, 3)) * 3.0 + rng.normal(0, 1e-3, (n, 3))
    if kind == "same":
        return np.zeros((n, 3))
    out = []  # chains of which every split peels one off, and a cluster that holds the rest
    for axis, scale in ((0, 1.0), (1, 2.0), (2, 4.0)):
        for k in range(1, 26):
            p = [0.0, 0.0, 0.0]
            p[axis] = scale * 32.0 ** k
            out.append(p)
    return np.concatenate([np.array(out), rng.uniform(0, 1, (n, 3))])


@pytest.mark.parametrize("kind,n", [("uniform", n) for n in (33, 63, 65, 256, 1023, 1024, 1025, 2049, 6000)]
                         + [("sorted", 1024), ("sorted", 4097), ("clusters", 900), ("clusters", 5000),
                            ("same", 1024), ("same", 3000), ("chains", 200), ("chains", 1500)])
def test_layout_matches_host_build(ctx, kind, n):
    rng = np.random.default_rng(n + 1)
    spheres = [{"type": "sphere", "center": [float(x) for x in c], "radius": float(r), "material": "m"}
               for c, r in zip(_points(kind, n), rng.uniform(0.05, 0.4, n + 75))]
    host = rtg.parse_scene(json.dumps({
        "camera": {"look_from": [0, 2, 12], "look_at": [0, 0, 0], "vfov": 40},
        "render": {"width": 16, "height": 16, "spp": 1, "max_depth": 2, "seed": 5},
        "materials": {"m": {"type": "lambertian", "albedo": [0.6, 0.5, 0.4]}}, "objects": spheres,
        "lights": [{"type": "point", "position": [0, 6, 4], "intensity": [20, 20, 20]}]}))
    a, b = ctx.upload(host), ctx.upload_gpu_bvh(host)
    try:
        for part in PARTS:
            x, y = ctx.scene_layout(a, part), ctx.scene_layout(b, part)
            if part == "roots":  # the fourth word says where the tree was built
                x, y = np.delete(x, 3, axis=1), np.delete(y, 3, axis=1)
            assert x.tobytes() == y.tobytes(), part
        ia, ib = ctx.scene_info(a), ctx.scene_info(b)
        for k in ("bvh_nodes", "bvh_leaves", "bvh_max_depth", "bvh_max_leaf"):
            assert ia[k] == ib[k], k
    finally:
        ctx.release(a)
        ctx.release(b)
