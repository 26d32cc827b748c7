"""Reads of frames in pieces: an image crosses in pieces of 2^18 pixels, several small images or
parts share one, means and moments have pieces of their own, and buffers of 16 MiB and
more are touched first. Every byte against the framebuffer's sums, resolved in NumPy; the
sizes are just below, at and above a piece, odd ones of more than five pieces and single
pixels, alone and in one read."""
import json

import numpy as np
import pytest

import rtg
import workloads

pytestmark = pytest.mark.gpu

SIZES = [(511, 513), (1, 1), (512, 512), (4033, 65), (3, 5), (1537, 1025), (2049, 2051), (7, 1), (640, 360)]


def _check(image, mean, tone_map, exposure):
    v = mean * exposure
    v = np.clip(v, 0, 1) if tone_map == "clamp" else v / (1 + v)
    s = np.where(v <= 0.0031308, 12.92 * v, 1.055 * np.clip(v, 0, 1) ** (1 / 2.4) - 0.055) * 255
    want = np.floor(s + 0.5)
    # Where the last bits of pow decide the rounding, either side is right.
    off = image != want
    assert (np.abs(s[off] - np.floor(s[off]) - 0.5) < 1e-9).all()


def test_reads_across_pieces(ctx):
    sid = ctx.load_json(json.dumps(workloads.cornell()))
    settings = []
    for k, (w, h) in enumerate(SIZES):
        s = ctx.scene_settings(sid)
        s.width, s.height, s.spp, s.max_depth, s.seed = w, h, 3, 2, k
        settings.append(s)
    try:
        ctx.render_batch([sid] * len(SIZES), settings)
        means = []
        for j, (w, h) in enumerate(SIZES):
            total, _, n = ctx.framebuffer_moments(j, w, h)
            assert (n == 3).all()
            means.append(total * (1.0 / 3))
            assert np.array_equal(ctx.framebuffer_mean(j, w, h), means[j])
        assert all(m.max() > 0 for m in means if m.size > 100)
        order = [6, 1, 0, 5, 4, 2, 3, 8, 7, 5, 1]
        for tone_map, exposure in (("clamp", 1.0), ("reinhard", 2.5)):
            images = ctx.images(order, [SIZES[j] for j in order], tone_map, exposure)
            for j, image in zip(order, images):
                _check(image, means[j], tone_map, exposure)
                assert np.array_equal(ctx.image(j, *SIZES[j], tone_map, exposure), image)
    finally:
        ctx.release(sid)
