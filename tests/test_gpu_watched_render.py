"""A render with a callback or a cancel word goes in iterations of at most 2^20 paths (half of a
larger pool), with at most two of them under way when a cancel is seen, so that neither
waits for long."""
import ctypes as C
import json

import pytest

import rtg
import workloads

pytestmark = pytest.mark.gpu

POOL, SIZE, SPP = 1 << 20, 1024, 16
PASS = SIZE * SIZE  # samples of the first pass: an iteration's


@pytest.fixture
def render(ctx):
    sid = ctx.load_json(json.dumps(workloads.sphere_field(SIZE, SIZE, SPP)))
    s = ctx.scene_settings(sid)
    s.spp = SPP
    before = ctx.tuning()["pool_paths"]
    ctx.set_tuning(pool_paths=POOL)
    yield lambda on_pass=None, cancel=None: ctx.render(sid, s, rtg.RenderOptions(progressive=True, max_pass_spp=4),
                                                       on_pass, cancel)
    ctx.set_tuning(pool_paths=before)
    ctx.release(sid)


@pytest.mark.parametrize("how", ["callback", "cancel word", "both"])
def test_iterations_are_short(ctx, render, how):
    render()
    plain = [x.tobytes() for x in ctx.framebuffer_moments(-1, SIZE, SIZE)]
    seen = []
    assert render((lambda p: seen.append(p.spp_done)) if how != "cancel word" else None,
                  C.c_int32(0) if how != "callback" else None).finished
    assert ctx.stats()["iterations"] >= PASS * SPP // POOL
    assert seen == ([] if how == "cancel word" else [1, 2, 4, 8, 12, 16])
    assert [x.tobytes() for x in ctx.framebuffer_moments(-1, SIZE, SIZE)] == plain


def test_a_cancel_leaves_little_behind(ctx, render):
    """The callback's progress has the rays of the iterations before the one under way. That one ends, and at most
    one queued behind it; together they trace the rays of 2 x 2^20 samples, or a few more where paths are left over."""
    render()
    st = ctx.stats()
    rays_a_sample = (st["rays"] + st["shadow_rays"]) / (PASS * SPP)
    cancel, seen = C.c_int32(0), []

    def stop(p):
        cancel.value = 1
        seen.append(p.rays)

    p = render(stop, cancel)
    assert p.cancelled and 1 <= p.spp_done < SPP
    st = ctx.stats()
    assert 0 <= st["rays"] + st["shadow_rays"] - seen[0] <= 2.2 * POOL * rays_a_sample
