"""Batch uploads of scenes with a host tree and scenes whose tree the GPU builds: every scene is
the one that a single upload makes, ids are in the batch's order, and the scenes with a host
tree are still flattened together."""
import json
import time

import numpy as np
import pytest

import rtg

pytestmark = pytest.mark.gpu

PARTS = ("nodes", "nodes4", "prims", "slot_material", "slot_normals", "materials", "slot_prim", "roots")


def _scene(n):
    rng = np.random.default_rng(n)
    text = json.dumps({"materials": {"m": {"type": "lambertian"}},
                       "objects": [{"type": "sphere", "center": rng.uniform(-9, 9, 3).tolist(),
                                    "radius": float(rng.uniform(0.01, 0.2)), "material": "m"} for _ in range(n)]})
    return rtg.parse_scene(text, defer_bvh="auto")


@pytest.mark.parametrize("sizes", [[1024], [5, 1024], [1500, 7], [3, 2000, 900, 1100, 1023, 1]])
def test_each_scene_is_that_of_a_single_upload(ctx, sizes):
    scenes = [_scene(n) for n in sizes]
    ids = ctx.upload_many(scenes)
    try:
        assert ids == list(range(ids[0], ids[0] + len(ids)))
        for sid, host, n in zip(ids, scenes, sizes):
            alone = ctx.upload(host)
            assert alone > ids[-1]
            assert ctx.scene_info(sid)["primitives"] == n
            for part in PARTS:
                assert ctx.scene_layout(sid, part).tobytes() == ctx.scene_layout(alone, part).tobytes(), (n, part)
            ctx.release(alone)
    finally:
        for sid in ids:
            ctx.release(sid)


def test_one_gpu_built_scene_leaves_the_others_together(ctx):
    small, large = [_scene(960 + k) for k in range(63)], _scene(1024)

    def upload(scenes):
        t = time.perf_counter()
        ids = ctx.upload_many(scenes)
        t = time.perf_counter() - t
        for sid in ids:
            ctx.release(sid)
        return t
    both, apart = [], []
    for _ in range(25):
        apart.append(upload(small) + upload([large]))
        both.append(upload(small + [large]))
    # One by one, the small ones take some three times as long as together.
    assert min(both) < 1.3 * min(apart)
