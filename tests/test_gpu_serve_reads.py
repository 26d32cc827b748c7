"""Reads of requests allocate nothing: what they go through is there once serving is prepared, so
that no read waits for the driver while requests render."""
import json

import pytest

import rtg
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prepare", [True, False])
@pytest.mark.parametrize("width,height", [(16, 9), (1500, 1100)])  # one piece, more pieces than slots
def test_reads_of_requests_do_not_allocate(prepare, width, height):
    with rtg.Context(0) as ctx:
        if prepare:
            ctx.serve_prepare()
        sid = ctx.load_json(json.dumps(workloads.cornell()))
        s = ctx.scene_settings(sid)
        s.width, s.height, s.spp, s.max_depth = width, height, 1, 2
        rid = ctx.submit(sid, s)
        before = rtg.allocation_count()
        while not ctx.request_progress(rid).finished:
            ctx.pump(50.0)
        assert ctx.request_image(rid, width, height).any() and ctx.request_mean(rid, width, height).any()
        ctx.release_request(rid)
        assert rtg.allocation_count() == before
