"""A batch that nobody can look into before its end (no cancel word) renders its jobs one
after the other; with a cancel word, pass by pass. The framebuffers, sums of squares,
counts and ray totals are the same bits either way, and the same as rendering alone."""
import ctypes as C
import json

import pytest

import rtg
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jobs", [1, 3, 7])
@pytest.mark.parametrize("pool", [4096, 1 << 20])
def test_batch_order_changes_no_bit(ctx, jobs, pool):
    ids = [ctx.upload(rtg.parse_scene(json.dumps(make()))) for make in (workloads.cornell, workloads.sphere_field)]
    before = ctx.tuning()["pool_paths"]
    ctx.set_tuning(pool_paths=pool)
    try:
        scenes, settings = [], []
        for k in range(jobs):
            s = ctx.scene_settings(ids[k % 2])
            s.width, s.height, s.spp, s.max_depth, s.seed = 40 + 9 * k, 33 - 2 * k, (13, 1, 40)[k % 3], 3 + k, k
            s.integrator = "direct" if k == 2 else "path"
            scenes.append(ids[k % 2])
            settings.append(s)
        opts = rtg.RenderOptions(progressive=True, max_pass_spp=4)

        def run(cancel):
            progress = ctx.render_batch(scenes, settings, opts, cancel)
            assert all(p.finished for p in progress)
            st = ctx.stats()
            return ([[x.tobytes() for x in ctx.framebuffer_moments(j, s.width, s.height)] for j, s in enumerate(settings)],
                    [st[n] for n in ("rays", "shadow_rays", "camera_samples", "passes")])
        by_job, by_pass = run(None), run(C.c_int32(0))
        assert by_job == by_pass
        for j, s in enumerate(settings):
            ctx.render(scenes[j], s, opts)
            assert [x.tobytes() for x in ctx.framebuffer_moments(-1, s.width, s.height)] == by_job[0][j]
    finally:
        ctx.set_tuning(pool_paths=before)
        for i in ids:
            ctx.release(i)
