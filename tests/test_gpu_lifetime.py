"""Scenes and caches that are destroyed after their context, as a garbage
collector may order it."""
import numpy as np
import pytest

from vision_b200 import scenes

pytestmark = pytest.mark.gpu


def test_scene_and_cache_outlive_their_context(vb, gpu_ctx):
    keep = vb.Scene(gpu_ctx, scenes.box_room(width=32, height=32, max_depth=2)).build_accel()
    keep.render(0, 2)
    want = keep.film()
    for _ in range(8):
        ctx = vb.Context(0)
        s = vb.Scene(ctx, scenes.box_room(width=64, height=64, max_depth=2)).build_accel()
        cache = vb.RadianceCache(ctx)
        s.render(0, 1)
        vb.lib.vs_synchronize(s.handle)
        ctx.close()
        other = [vb.Context(-1) for _ in range(4)]  # a context's memory, used again
        s.close()
        cache.close()
        del other
        keep.render(0, 2)
        assert np.array_equal(keep.film(), want)
