"""A sample whose refracted ray leaves within rounding of the surface's plane: the side it
leaves on depends on the order in which the dot product fuses. The values are those the
renderer has always given (they are also what pins the order, in every instance)."""
import json

import numpy as np
import pytest

import rtg

pytestmark = pytest.mark.gpu

PIXEL, MEAN = (934, 459), ("0x1.6adbdec000000p-1", "0x1.9dfb638000000p-1", "0x1.eaaaaaaaaaaaap-1")


@pytest.mark.parametrize("count", [0, 1])
def test_grazing_refraction_leaves_on_the_same_side(ctx, count):
    rng = np.random.default_rng(0)
    materials = {f"g{k}": {"type": "dielectric", "ior": float(rng.uniform(1.05, 2.6)), "albedo": [1, 1, 1]}
                 for k in range(12)}
    materials["w"] = {"type": "lambertian", "albedo": [.8, .7, .6]}
    objects = [{"type": "sphere", "center": rng.uniform(-3, 3, 3).tolist(), "radius": float(rng.uniform(.5, 1.1)),
                "material": f"g{k % 12}"} for k in range(40)]
    sid = ctx.upload(rtg.parse_scene(json.dumps({
        "camera": {"look_from": [0, 0, 9], "look_at": [0, 0, 0], "vfov": 45},
        "render": {"width": 1024, "height": 1024, "spp": 48, "max_depth": 24, "seed": 0},
        "materials": materials, "objects": objects,
        "lights": [{"type": "point", "position": [0, 6, 4], "intensity": [20, 20, 20]}]})))
    ctx.set_tuning(count_traversal=count)
    try:
        s = ctx.scene_settings(sid)
        s.rr_min_depth = 24
        ctx.render(sid, s, rtg.RenderOptions(progressive=False))
        mean = ctx.framebuffer_mean(-1, 1024, 1024)[PIXEL]
        assert [float(v).hex() for v in mean] == list(MEAN)
    finally:
        ctx.set_tuning(count_traversal=0)
        ctx.release(sid)
