"""GPU BVH build: records, boxes, normals and materials that the GPU makes from staged
primitives are the host's bytes, across pieces (32,768 primitives), with and without
vertex normals in a piece, and with primitives that have no usable box."""
import json

import numpy as np
import pytest

import rtg

pytestmark = pytest.mark.gpu

PARTS = ["nodes", "nodes4", "prims", "slot_material", "slot_normals", "slot_prim"]


def _spheres(n, rng):
    return [{"type": "sphere", "center": c.tolist(), "radius": float(r), "material": "ab"[i % 2]}
            for i, (c, r) in enumerate(zip(rng.uniform(-9, 9, (n, 3)) + 1e3, rng.uniform(0.01, 0.1, n)))]


def _triangles(n, rng):
    v = rng.uniform(-9, 9, (n, 3, 3))
    v[::3, :, 1] = v[::3, :1, 1]  # every third one flat
    return [{"type": "triangle", "v0": a.tolist(), "v1": b.tolist(), "v2": c.tolist(), "material": "b"} for a, b, c in v]


def _smooth(n):
    return [{"type": "mesh", "name": "ball", "source": "icosphere", "subdivisions": n, "smooth": True, "material": "a"}]


NO_BOX = {"type": "sphere", "center": [1.7e308, 0, 0], "radius": 1.7e308, "material": "a"}


@pytest.mark.parametrize("name", ["small", "smooth", "one_piece", "pieces", "no_box"])
def test_converted_primitives_match_the_host(ctx, name):
    rng = np.random.default_rng(11)
    objects = {"small": lambda: _spheres(3, rng) + _triangles(5, rng),
               "smooth": lambda: _triangles(7, rng) + _smooth(3) + _spheres(2, rng),
               "one_piece": lambda: _spheres(32768 - 8, rng) + _triangles(8, rng),
               "pieces": lambda: _triangles(33000, rng) + _smooth(5) + _spheres(20000, rng),
               "no_box": lambda: [NO_BOX] + _triangles(2100, rng) + [NO_BOX] + _spheres(40, rng) + [NO_BOX]}[name]()
    host = rtg.parse_scene(json.dumps({
        "camera": {"look_from": [0, 2, 12], "look_at": [0, 0, 0], "vfov": 40},
        "render": {"width": 16, "height": 16, "spp": 1, "max_depth": 2, "seed": 5},
        "materials": {"a": {"type": "lambertian", "albedo": [0.6, 0.5, 0.4]},
                      "b": {"type": "lambertian", "albedo": [0.2, 0.5, 0.4]}}, "objects": objects,
        "lights": [{"type": "point", "position": [0, 6, 4], "intensity": [20, 20, 20]}]}))
    a, b = ctx.upload(host), ctx.upload_gpu_bvh(host)
    try:
        for part in PARTS:
            x, y = ctx.scene_layout(a, part), ctx.scene_layout(b, part)
            assert x.shape == y.shape and x.tobytes() == y.tobytes(), part
    finally:
        ctx.release(a)
        ctx.release(b)
