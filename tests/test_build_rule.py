"""Which scenes the automatic modes build on the GPU, and that nothing else about them
changes with it: the host view, the host layout and the scene's info are those of a
host-built scene up to 32,767 primitives (larger ones have no host tree)."""
import json

import numpy as np
import pytest

import rtg


def field(n):
    rng = np.random.default_rng(n)
    objs = [{"type": "sphere", "center": [float(x) for x in rng.uniform(-20, 20, 3)], "radius": 0.1, "material": "m"}
            for _ in range(n)]
    return json.dumps({"name": "field", "camera": {"look_from": [0, 0, 60], "look_at": [0, 0, 0], "vfov": 40},
                       "render": {"width": 16, "height": 16, "spp": 2, "max_depth": 3},
                       "materials": {"m": {"type": "lambertian", "albedo": 0.5}}, "objects": objs})


SIZES = [1023, 1024, 5000]


@pytest.mark.parametrize("n", SIZES)
def test_host_view_of_an_automatic_scene_has_its_tree(n):
    a, b = rtg.parse_scene(field(n), defer_bvh="auto"), rtg.parse_scene(field(n))
    va, vb = a.view(), b.view()
    for k in vb:
        assert np.array_equal(va[k], vb[k]) if isinstance(vb[k], np.ndarray) else va[k] == vb[k], k
    for part in ("nodes", "nodes4", "prims", "slot_prim", "roots", "nodes8"):
        assert np.array_equal(a.device_layout(part).view(np.uint32), b.device_layout(part).view(np.uint32)), part
    assert len(rtg.parse_scene(field(n), defer_bvh=True).view()["nodes"]) == 0


def test_large_automatic_scene_has_no_host_tree():
    assert len(rtg.parse_scene(field(32768), defer_bvh="auto").view()["nodes"]) == 0
    assert len(rtg.parse_scene(field(32767), defer_bvh="auto").view()["nodes"]) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["auto", True])
@pytest.mark.parametrize("n", SIZES)
def test_rule_and_info(ctx, n, mode):
    a = ctx.upload(rtg.parse_scene(field(n)))
    b = ctx.upload(rtg.parse_scene(field(n), defer_bvh=mode))
    try:
        assert ctx.scene_layout(b, "roots")[0][3] == int(n >= 1024)
        ia, ib = ctx.scene_info(a), ctx.scene_info(b)
        assert {k: v for k, v in ia.items() if k != "bvh_build_ms"} == {k: v for k, v in ib.items() if k != "bvh_build_ms"}
        for part in ("nodes", "nodes4", "prims", "slot_material", "slot_normals", "slot_prim"):
            assert ctx.scene_layout(a, part).tobytes() == ctx.scene_layout(b, part).tobytes(), part
    finally:
        ctx.release(a)
        ctx.release(b)
