"""A direct render that someone watches goes pass by pass: what a callback, a cancel or another
request can see of it is that of the passes traced so far, and no more is traced."""
import ctypes as C
import json

import pytest

import rtg
import workloads

pytestmark = pytest.mark.gpu

OPTIONS = rtg.RenderOptions(progressive=True, max_pass_spp=2)
PASSES = [1, 2, 4, 6, 7]  # samples done after each


@pytest.fixture
def scene(ctx):
    sid = ctx.load_json(json.dumps(workloads.mix_scene(5)))
    s = ctx.scene_settings(sid)
    s.width, s.height, s.max_depth, s.rr_min_depth, s.integrator = 96, 70, 5, 5, "direct"
    yield sid, s
    ctx.release(sid)


def test_progress_counts_the_rays_so_far(ctx, scene):
    sid, s = scene
    want = []
    for s.spp in PASSES:
        ctx.render(sid, s, OPTIONS)
        want.append(ctx.stats()["rays"] + ctx.stats()["shadow_rays"])
    seen = []
    ctx.render(sid, s, OPTIONS, lambda p: seen.append((p.spp_done, p.rays)))
    assert seen == list(zip(PASSES, want))


@pytest.mark.parametrize("callback", [True, False])
def test_a_cancelled_render_traced_what_it_counts(ctx, scene, callback):
    sid, s = scene
    s.spp = 2
    ctx.render(sid, s, OPTIONS)
    alone = ctx.stats()
    s.spp = PASSES[-1]
    cancel = C.c_int32(0 if callback else 1)

    def stop(p):
        if p.spp_done == 2:
            cancel.value = 1

    p = ctx.render(sid, s, OPTIONS, stop if callback else None, cancel)
    assert p.cancelled and p.spp_done == (2 if callback else 0)
    st = ctx.stats()
    assert [st[k] for k in ("camera_samples", "rays", "shadow_rays")] == \
        ([alone[k] for k in ("camera_samples", "rays", "shadow_rays")] if callback else [0, 0, 0])


def test_a_request_traces_a_pass_at_a_time(ctx, scene):
    sid, s = scene
    s.spp = PASSES[-1]
    rid = ctx.submit(sid, s, OPTIONS)
    try:
        done = []
        while not done or done[-1] < s.spp:
            ctx.pump(0.0)  # one turn of the scheduler
            done.append(ctx.request_progress(rid).spp_done)
            assert len(done) < 100
        assert done == PASSES
    finally:
        while not ctx.request_progress(rid).finished:
            ctx.pump(50.0)
        ctx.release_request(rid)
