"""The depth keys and the vertex stage beside them: splat counts around the
blocks of both (1,024 keys, 256 splats), some behind the camera, against the
oracle; view sets of two scenes in one launch; a reused order."""

import numpy as np
import pytest

import gsplat_ffi as ffi
import gsplat_scenes
from conftest import assert_fp32_image
from test_gpu_parity import _compare_stages, _render

pytestmark = pytest.mark.gpu


def _scene(n):
    rng = np.random.default_rng(n)
    means = rng.normal(0.0, 1.5, (n, 3)).astype(np.float32)
    means[0] = 0.0
    return gsplat_scenes.make_scene(rng, means, -2.5, 0.5, 0.5, 1.0, 1)


CAM = gsplat_scenes.camera((0.0, 0.0, -1.5), (0, 0, 0), 60.0)


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1023, 1024, 1025, 2049, 5000])
def test_keys_against_oracle(oracle, n):
    scene = _scene(n)
    sv = oracle.SceneView(scene)
    fr = oracle.Frame(sv, CAM, 97, 65, tile=16)
    ctx = _render(scene, CAM, 97, 65, tile=16)
    _compare_stages(ctx, fr, sv)
    image = ctx.readback_rgba8()
    assert_fp32_image(image, fr.raster_tiles_fp32())
    ctx.set_sort_interval(1000)
    for _ in range(3):  # the reused order: the keys are only counted
        ctx.render_frame()
        assert np.array_equal(ctx.readback_rgba8(), image)
        assert ctx.frame_counts().visible == len(fr.order)


@pytest.mark.parametrize("a,b", [(1024, 1025), (1, 2049), (257, 700)])
def test_key_sets_of_a_batch(a, b):
    """Sets of up to 16 views: every view's image is its plain frame's."""
    scenes = [_scene(a), _scene(b)]
    rng = np.random.default_rng(7)
    views = [(k // 17 % 2, gsplat_scenes.orbit_camera(rng, (1.0, 3.0)), 64, 48) for k in range(51)]
    with ffi.Batch() as batch:
        ids = [batch.add_scene(s) for s in scenes]
        batch.render([(ids[s], c, w, h) for s, c, w, h in views])
        for k in (0, 15, 16, 17, 33, 34, 50):
            s, cam, w, h = views[k]
            ctx = _render(scenes[s], cam, w, h, debug=False)
            assert np.array_equal(batch.readback_rgba8(k), ctx.readback_rgba8()), k
            assert batch.view_stats(k).visible_count == ctx.frame_counts().visible
