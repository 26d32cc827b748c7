"""The shadow ray of a diffuse hit starts on the light's side of the surface, whichever side
the scattered ray of the same hit leaves on.

The side is the sign of a dot product, which one rounding may call positive and another
not where a scattered direction lies in the surface's plane. The scene makes such
directions as frequent as can be (some three in 10^9 samples): one triangle fills the
view, its shading normals lie almost in its plane, a far red point light stands over it,
and the background is green. A sample is black (scattered below the surface), or it has
the light's red and, unless its scattered ray meets the triangle again, the background's
green. None has the green alone: that is a shadow ray that started below the triangle."""
import json

import numpy as np
import pytest

import rtg

pytestmark = pytest.mark.gpu

SIZE, SPP, DISTANCE = 2048, 1024, 1e6


def test_shadow_rays_start_on_the_lights_side(ctx, tmp_path):
    gn = np.ones(3) / np.sqrt(3)
    a = np.array([1, -1, 0]) / np.sqrt(2)
    b = np.cross(gn, a)
    corners = [20 * a, 20 * (-0.5 * a + 0.8 * b), 20 * (-0.5 * a - 0.8 * b)]
    shading = np.cos(1.5) * gn + np.sin(1.5) * a
    lines = ["v " + " ".join(repr(float(x)) for x in c) for c in corners]
    lines += ["vn " + " ".join(repr(float(x)) for x in shading)] * 3
    (tmp_path / "tilted.obj").write_text("\n".join(lines + ["f 1//1 2//2 3//3", ""]))
    to_light = (gn + a) / np.sqrt(2)
    sid = ctx.load_json(json.dumps({
        "camera": {"look_from": (3 * gn).tolist(), "look_at": [0, 0, 0], "vfov": 20},
        "render": {"width": SIZE, "height": SIZE, "spp": SPP, "max_depth": 2, "rr_min_depth": 2, "seed": 3},
        "background": {"type": "solid", "color": [0, 1, 0]},
        "materials": {"m": {"type": "lambertian", "albedo": [0.5, 0.5, 0.5]}},
        "objects": [{"type": "mesh", "source": "obj", "path": "tilted.obj", "smooth": True, "material": "m"}],
        "lights": [{"type": "point", "position": (DISTANCE * to_light).tolist(),
                    "intensity": [4 * DISTANCE ** 2, 0, 0]}]}), str(tmp_path))
    try:
        s = ctx.scene_settings(sid)
        s.rr_min_depth = 9
        ctx.render(sid, s, rtg.RenderOptions(progressive=False))
        total, _, n = ctx.framebuffer_moments(-1, SIZE, SIZE)
    finally:
        ctx.release(sid)
    red, green = total[..., 0], total[..., 1] / 0.5  # green: the number of samples that have it
    assert (n == SPP).all() and 0.4 < green.sum() / (SIZE * SIZE * SPP) < 0.7
    # Reds differ by the light's distance and rounding only, some 1e-6 each: 1,024 of them by 1e-3 of one.
    lit = red / float(np.median(red / green))
    assert int((lit < green - 0.5).sum()) == 0
