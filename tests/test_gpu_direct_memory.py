"""What the direct integrator allocates. A served request has the footprint that admission
counted and nothing more, however many samples its passes have and however deep its
branches may go; a render takes memory for its pending branches and gives it back."""
import json

import pytest

import rtg

pytestmark = pytest.mark.gpu


def _pool():
    """A glass plane between two diffuse balls: a tree has three vertices at most, whatever the depth."""
    balls = [{"type": "sphere", "center": [x, y, 0], "radius": 0.9, "material": "matt"} for x, y in ((0, 1), (0.5, -1.2))]
    return json.dumps({"camera": {"look_from": [0, 1.5, 6], "look_at": [0, 0, 0], "vfov": 40},
                       "background": {"type": "gradient", "top": [0.4, 0.6, 1.0], "bottom": [1, 1, 1]},
                       "materials": {"glass": {"type": "dielectric", "ior": 1.3},
                                     "matt": {"type": "lambertian", "albedo": 0.6}},
                       "objects": balls + [{"type": "plane", "point": [0, 0, 0], "normal": [0, 1, 0],
                                            "material": "glass"}],
                       "lights": [{"type": "point", "position": [-3, 5, 2], "intensity": 20}]})


@pytest.mark.parametrize("depth", [3, 60])
def test_a_request_allocates_nothing_while_it_renders(ctx, depth):
    sid = ctx.load_json(_pool())
    try:
        s = ctx.scene_settings(sid)
        s.width = s.height = 512
        s.spp, s.max_depth, s.rr_min_depth, s.integrator = 4, depth, 3, "direct"  # a pass of 2^20 samples
        opts = rtg.RenderOptions(progressive=False)
        rid = ctx.submit(sid, s, opts)
        before = rtg.allocation_count()
        while not ctx.request_progress(rid).finished:
            ctx.pump(50.0)
        assert rtg.allocation_count() == before
        served = ctx.request_mean(rid, 512, 512).tobytes()
        ctx.release_request(rid)
        for _ in range(2):
            ctx.render(sid, s, opts)
            assert ctx.framebuffer_mean(-1, 512, 512).tobytes() == served
    finally:
        ctx.release(sid)


def test_branch_memory_is_given_back():
    """The branches of a deep render (458 MB) lie in the pool afterwards, where a framebuffer of that size fits: the
    device has as much memory free as before it."""
    import torch

    with rtg.Context(0) as ctx:
        sid = ctx.load_json(_pool())
        s = ctx.scene_settings(sid)
        s.width = s.height = 512
        s.spp, s.max_depth, s.rr_min_depth, s.integrator = 4, 60, 3, "direct"
        ctx.render(sid, s, rtg.RenderOptions(progressive=False))
        free = torch.cuda.mem_get_info()[0]
        s.width, s.height, s.spp, s.max_depth, s.integrator = 2560, 2048, 1, 2, "normals"  # 68 bytes a pixel: 357 MB
        ctx.render(sid, s, rtg.RenderOptions(progressive=False))
        assert torch.cuda.mem_get_info()[0] > free - (64 << 20)
