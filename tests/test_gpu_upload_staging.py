"""Pinned staging of uploads: scenes of about one size, and one scene in the two forms that cross
the bus (records for the GPU build, flattened), go through what is there."""
import json

import numpy as np
import pytest

import rtg

pytestmark = pytest.mark.gpu


def _text(n):
    rng = np.random.default_rng(n)
    return json.dumps({"materials": {"m": {"type": "lambertian"}},
                       "objects": [{"type": "sphere", "center": rng.uniform(-9, 9, 3).tolist(),
                                    "radius": float(rng.uniform(0.01, 0.2)), "material": "m"} for _ in range(n)]})


def _allocations(ctx, scene):
    before = rtg.allocation_count()
    ctx.release(ctx.upload(scene))
    return rtg.allocation_count() - before


@pytest.mark.parametrize("n", [1500, 9000])
def test_staging_is_kept(n):
    with rtg.Context(0) as ctx:
        gpu_built = [rtg.parse_scene(_text(n + n * k // 100), defer_bvh="auto") for k in range(11)]  # up to a tenth more
        for _ in range(2):  # there are two buffers, in turn
            ctx.release(ctx.upload(gpu_built[0]))
        host_built = [rtg.parse_scene(_text(n))] * 4
        for scenes in (gpu_built, host_built):
            counts = [_allocations(ctx, s) for s in scenes]
            # What every upload takes from the device pool, and nothing else.
            assert counts == [_allocations(ctx, scenes[0])] * len(counts)
