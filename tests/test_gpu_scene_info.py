"""rtg_scene_get_info of a scene whose tree the GPU built: the host tree's SAH cost, to the bit,
and no host build to find it."""
import json
import time

import numpy as np
import pytest

import rtg
import workloads

pytestmark = pytest.mark.gpu


def _spheres(n):
    rng = np.random.default_rng(n)
    return json.dumps({"materials": {"m": {"type": "lambertian"}},
                       "objects": [{"type": "sphere", "center": rng.uniform(-9, 9, 3).tolist(),
                                    "radius": float(rng.uniform(0.01, 0.2)), "material": "m"} for _ in range(n)]})


def _mesh():
    scene = workloads.mesh_stress()
    for o in scene["objects"]:
        if o.get("source") == "icosphere":
            o["subdivisions"] = 4
        elif o.get("source") == "torus":
            o["segments"], o["segments_v"] = 61, 47
    return json.dumps(scene)


@pytest.mark.parametrize("make", [lambda: _spheres(1024), lambda: _spheres(2049), lambda: _spheres(32767), _mesh,
                                  lambda: json.dumps({"materials": {"m": {"type": "lambertian"}}, "objects": [
                                      {"type": "sphere", "center": [1, 2, 3], "radius": 1, "material": "m"}] * 1500})],
                         ids=["1024", "2049", "32767", "mesh", "coincident"])
def test_sah_cost_is_the_host_trees(ctx, make):
    text = make()
    a, b = ctx.upload(rtg.parse_scene(text)), ctx.upload(rtg.parse_scene(text, defer_bvh="auto"))
    try:
        assert ctx.scene_layout(b, "roots")[0][3] == 1  # built on the GPU
        ia, ib = ctx.scene_info(a), ctx.scene_info(b)
        assert ia.pop("bvh_build_ms") > 0 and ib.pop("bvh_build_ms") > 0
        assert ia == ib and ia["bvh_sah_cost"] > 0
    finally:
        ctx.release(a)
        ctx.release(b)


def test_information_is_only_read(ctx):
    text = _spheres(20000)
    t = [time.perf_counter()]
    rtg.parse_scene(text)
    t.append(time.perf_counter())
    sid = ctx.upload(rtg.parse_scene(text, defer_bvh=True))
    t.append(time.perf_counter())
    compiled = rtg.parse_scene(text, defer_bvh=True)
    t.append(time.perf_counter())
    ctx.scene_info(sid)
    t.append(time.perf_counter())
    ctx.release(sid)
    del compiled
    build = (t[1] - t[0]) - (t[3] - t[2])  # the host build is some 25 ms
    assert t[4] - t[3] < 0.1 * build
