"""The path kernel and the direct integrator's kernel at the edges of their scheduling.

A sample's radiance does not depend on which warp holds it, what else the warp
holds, or whether it is left to a later iteration, so a render under any tuning has
to give the default's framebuffer to the bit. The sizes are around a warp's batch (1,
31, 33, 1023 samples) and around what an iteration of the smallest pool takes; with a
pool of 1024 paths and one block, paths are left over at the end of every iteration.
A one-pixel, one-sample render is compared with the same sample of a larger one, and
the direct integrator's deepest trees with the oracle."""
import json

import numpy as np
import pytest

import rtg
import rtoracle
import workloads

pytestmark = pytest.mark.gpu

TUNINGS = [dict(pool_paths=1024, extend_blocks=1), dict(pool_paths=1024, extend_blocks=1 << 20), dict(block=64),
           dict(block=256, chained=0), dict(count_traversal=1)]


def glass(nested=6):
    """Glass shells around a rough metal ball over a diffuse floor: deep trees of reflections and refractions."""
    objs = [{"type": "sphere", "center": [0, 1, 0], "radius": 1.0 - 0.1 * k, "material": "glass"} for k in range(nested)]
    objs += [{"type": "sphere", "center": [0, 1, 0], "radius": 0.3, "material": "rough"},
             {"type": "sphere", "center": [1, 4, 1], "radius": 0.6, "material": "lamp"},
             {"type": "plane", "point": [0, 0, 0], "normal": [0, 1, 0], "material": "floor"}]
    return {"name": "shells", "camera": {"look_from": [0, 1.5, 4], "look_at": [0, 1, 0], "vfov": 35},
            "render": {"width": 16, "height": 16, "spp": 1, "max_depth": 10, "rr_min_depth": 3, "seed": 5},
            "background": {"type": "gradient", "top": [0.4, 0.6, 1.0], "bottom": [1, 1, 1]},
            "materials": {"glass": {"type": "dielectric", "ior": 1.3}, "floor": {"type": "lambertian", "albedo": 0.6},
                          "rough": {"type": "metal", "albedo": [0.9, 0.7, 0.5], "roughness": 0.3},
                          "lamp": {"type": "emissive", "color": 1, "intensity": 9}},
            "objects": objs, "lights": [{"type": "point", "position": [-3, 5, 2], "intensity": 20}]}


SCENES = {"cornell": workloads.cornell, "spheres": workloads.sphere_field, "mirrors": lambda: workloads.mix_scene(5),
          "glass": glass}


@pytest.mark.parametrize("integrator,mis", [("path", False), ("path", True), ("normals", False), ("direct", False)])
@pytest.mark.parametrize("scene", list(SCENES))
def test_any_tuning_gives_the_same_framebuffer(ctx, scene, integrator, mis):
    sid = ctx.load_json(json.dumps(SCENES[scene]()))
    before = ctx.tuning()
    try:
        for w, h, spp, progressive in ((1, 1, 1, False), (31, 1, 1, False), (11, 3, 31, True), (40, 31, 7, False)):
            s = ctx.scene_settings(sid)
            s.width, s.height, s.spp, s.integrator, s.mis = w, h, spp, integrator, mis
            opts = rtg.RenderOptions(progressive=progressive)

            def run():
                assert ctx.render(sid, s, opts).finished
                st = ctx.stats()
                a = ctx.framebuffer_moments(-1, w, h)
                assert (a[2] == spp).all()
                return [x.tobytes() for x in a] + [st["rays"], st["shadow_rays"], st["rr_terminated"]]

            want = run()
            for t in TUNINGS:
                ctx.set_tuning(**t)
                assert run() == want, (w, h, spp, t)
                ctx.set_tuning(**{k: before[k] for k in t})
    finally:
        ctx.set_tuning(**{k: before[k] for k in ("pool_paths", "extend_blocks", "block", "chained", "count_traversal")})
        ctx.release(sid)


def test_leftover_paths_of_mixed_jobs(ctx):
    """Paths of several jobs (MIS, brute force, depth 40 and normals among them) left over together, many times."""
    scenes = [workloads.cornell(48, 40, 9), workloads.mix_scene(5), workloads.sphere_field(32, 24, 6), glass()]
    scenes[1]["render"].update(width=24, height=24, spp=5)
    scenes[2]["render"]["use_bvh"] = False
    sids = [ctx.load_json(json.dumps(s)) for s in scenes]
    settings = [ctx.scene_settings(i) for i in sids]
    settings[0].mis = True
    settings[3].integrator = "normals"
    alone = []
    for i, s in zip(sids, settings):
        ctx.render(i, s)
        alone.append(ctx.framebuffer_moments(-1, s.width, s.height)[0].tobytes())
    before = ctx.tuning()
    try:
        ctx.set_tuning(pool_paths=1024, extend_blocks=2)
        ctx.render_batch(sids, settings)
        assert [ctx.framebuffer_moments(j, s.width, s.height)[0].tobytes() for j, s in enumerate(settings)] == alone
    finally:
        ctx.set_tuning(pool_paths=before["pool_paths"], extend_blocks=before["extend_blocks"])
        for i in sids:
            ctx.release(i)


@pytest.mark.parametrize("depth", [0, 1, 2, 10])
def test_direct_trees_match_the_oracle(ctx, depth):
    """Samples of the direct integrator at 1 spp, against the oracle's recursion with the same RNG streams. As in
    the render tests, a sample may part where float32 and float64 round a hit or a Fresnel case apart: 97% within
    1e-3 for trees of hundreds of vertices (each has its own chance to part)."""
    if depth == 0:
        scene = workloads.cornell(width=16, height=16, spp=1)
        scene["render"]["max_depth"] = 1
        scene["objects"] = [o for o in scene["objects"] if o.get("name") != "ceiling light"]  # no light at all
    else:
        scene = glass()
        scene["render"]["max_depth"] = depth
    scene["render"]["integrator"] = "direct"
    scene["render"]["rr_min_depth"] = 1
    sid = ctx.load_json(json.dumps(scene))
    s = ctx.scene_settings(sid)
    ctx.render(sid, s, rtg.RenderOptions(progressive=False))
    got = ctx.framebuffer_moments(-1, s.width, s.height)[0]
    ctx.release(sid)
    want, _, _ = rtoracle.OracleScene(rtg.parse_scene(json.dumps(scene)).view()).render()
    err = np.abs(got - want).max(-1) / np.maximum(1.0, np.abs(want).max(-1))
    print(depth, "largest error", err.max(), "agree", (err <= 1e-3).mean())
    assert (err <= 1e-3).mean() >= 0.97


@pytest.mark.parametrize("scene", ["mesh", "glass", "cornell"])
def test_direct_kernels_agree(ctx, scene):
    """A direct pass of 2^20 samples takes the per-warp kernel, smaller launches a thread a sample: the same render as
    one pass of 512x512x4 and with its passes in callbacks' sight has to give the same bits. The callbacks see every
    pass, in order, each with just its samples; a cancel in one drops the passes traced with it."""
    make = SCENES.get(scene, workloads.mesh_stress)()
    sid = ctx.load_json(json.dumps(make))
    try:
        s = ctx.scene_settings(sid)
        s.width = s.height = 512
        s.spp, s.max_depth, s.integrator, s.rr_min_depth = 4, 4, "direct", 3
        ctx.render(sid, s, rtg.RenderOptions(progressive=False))
        one = [x.tobytes() for x in ctx.framebuffer_moments(-1, 512, 512)]
        s.width, s.height = 500, 520  # 260,000 pixels: passes of 1, 1 and 2 samples together are just under 2^20
        seen = []

        def on_pass(p):
            n = ctx.framebuffer_moments(-1, 500, 520)[2]
            assert (n == p.spp_done).all()
            seen.append((p.pass_, p.spp_done))

        ctx.render(sid, s, rtg.RenderOptions(progressive=True), on_pass)
        assert seen == [(1, 1), (2, 2), (3, 4)]
        small = [x.tobytes() for x in ctx.framebuffer_moments(-1, 500, 520)]
        s.spp = 5  # with a fourth pass, over 2^20 samples
        ctx.render(sid, s, rtg.RenderOptions(progressive=True))
        assert (ctx.framebuffer_moments(-1, 500, 520)[2] == 5).all()
        s.spp = 4
        ctx.render(sid, s, rtg.RenderOptions(progressive=True))
        assert [x.tobytes() for x in ctx.framebuffer_moments(-1, 500, 520)] == small
        # 512x512 in passes of one sample: 2^18 samples each, four in a launch of 2^20 or alone.
        s.width = s.height = 512
        ctx.render(sid, s, rtg.RenderOptions(progressive=True, max_pass_spp=1))
        assert [x.tobytes() for x in ctx.framebuffer_moments(-1, 512, 512)] == one
        before = ctx.tuning()
        ctx.set_tuning(max_pass_samples=512 * 512)  # room for one such pass
        try:
            ctx.render(sid, s, rtg.RenderOptions(progressive=True, max_pass_spp=1))
        finally:
            ctx.set_tuning(max_pass_samples=before["max_pass_samples"])
        assert [x.tobytes() for x in ctx.framebuffer_moments(-1, 512, 512)] == one
        import ctypes
        cancel = ctypes.c_int32(0)

        def stop(p):
            cancel.value = 1

        prog = ctx.render(sid, s, rtg.RenderOptions(progressive=True, max_pass_spp=1), stop, cancel)
        assert prog.cancelled and prog.spp_done == 1
        assert (ctx.framebuffer_moments(-1, 512, 512)[2] == 1).all()
    finally:
        ctx.release(sid)
