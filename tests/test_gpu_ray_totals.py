"""Ray totals of batches that mix path jobs and direct ones are the sums of their jobs'.

The two kinds run beside one another, and the host learns of their counters in different
ways (snapshots of earlier iterations, and reads after a direct launch), so which news is
the latest depends on how the job sizes interleave. The sizes here are many, at pools
where the host cannot tell early that the path jobs are done."""
import json

import pytest

import rtg
import workloads

pytestmark = pytest.mark.gpu

COUNTERS = ("rays", "shadow_rays", "rr_terminated")


def _totals(ctx):
    st = ctx.stats()
    return [st[k] for k in COUNTERS]


@pytest.mark.parametrize("pool", [4096, 1 << 17])
def test_totals_are_the_sums_of_the_jobs(ctx, pool):
    sid = ctx.load_json(json.dumps(workloads.cornell()))
    before = ctx.tuning()["pool_paths"]
    ctx.set_tuning(pool_paths=pool)
    opts = rtg.RenderOptions(progressive=True, max_pass_spp=4)

    def settings(integrator, size, spp):
        s = ctx.scene_settings(sid)
        s.width, s.height, s.spp, s.max_depth, s.integrator = size, size, spp, 5, integrator
        return s

    def alone(s):
        p = ctx.render(sid, s, opts)
        assert p.rays == sum(_totals(ctx)[:2])
        return _totals(ctx)
    try:
        paths = [settings("path", size, spp) for size in (8, 24, 64, 128) for spp in (1, 7, 33, 64)]
        direct = [settings("direct", 16, spp) for spp in (1, 20, 60, 150)]
        path_totals, direct_totals = [alone(s) for s in paths], [alone(s) for s in direct]
        wrong = []
        for p, pt in zip(paths, path_totals):
            for d, dt in zip(direct, direct_totals):
                for jobs in ([p, d], [d, p]):
                    progress = ctx.render_batch([sid, sid], jobs, opts)
                    got, again = _totals(ctx), None
                    if [x.rays for x in progress] == [sum(got[:2])] * 2 and got == [x + y for x, y in zip(pt, dt)]:
                        ctx.render(sid, paths[0], opts)  # a base that is too low would show in the next render
                        again = _totals(ctx)
                    if again != path_totals[0]:
                        wrong.append((p.width, p.spp, d.spp, jobs[0].integrator))
        assert not wrong
    finally:
        ctx.set_tuning(pool_paths=before)
        ctx.release(sid)
