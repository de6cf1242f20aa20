"""The autotuner's choice among candidates that launch the same kernels."""

import numpy as np
import pytest

import gsplat_ffi as ffi
import gsplat_scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blend", [ffi.BLEND_FP32, ffi.BLEND_UNORM8])
def test_equal_candidates_are_one(blend):
    """1,200 tiles of 16x16 and 4,800 of 8x8, more than the few-tile kernels
    take: chunk 256 launches what chunk 128 does in the FP32 mode, and the
    UNORM8 mode has one kernel a tile size. The first of each is chosen; every
    candidate is compared."""
    scene, cam, _, _ = gsplat_scenes.config1(seed=5)
    with ffi.Batch() as b:
        b.set_blend_mode(blend)
        b.add_scene(scene)
        views = [(0, cam, 640, 480)]
        b.render(views)
        before = b.readback_rgba8(0).copy()
        r = b.autotune(views, None, reps=1)
        assert r.candidates == 15 and 0 < r.best_ms <= r.default_ms
        if blend == ffi.BLEND_UNORM8:
            assert (r.tile_size, r.chunk, r.blocks_per_sm) in ((16, 256, 0), (8, 64, 0))
        else:
            assert r.chunk != 128
        b.render(views)
        assert np.array_equal(b.readback_rgba8(0), before)


def test_candidates_are_timed_on_the_graph_they_run():
    """The default shape's time is that of its repeated render, one graph
    launch: the renders that plan without predictions and that capture the
    graph (host milliseconds between the launches of well under one) are not
    timed. The margin is for a busy host and the clocks."""
    scene, cam, _, _ = gsplat_scenes.config1(seed=6)
    views = [(0, cam, 400 + 16 * k, 300) for k in range(12)]
    with ffi.Batch() as b:
        b.add_scene(scene)
        r = b.autotune(views, None, reps=1)
        b.set_tile_size(16)
        b.set_raster_config(256, 0)
        steady = sorted(b.render(views).device_ms for _ in range(9))[4]
        assert r.default_ms < 2.0 * steady, (r.default_ms, steady)
