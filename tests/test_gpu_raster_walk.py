"""The raster's two walks of a bin's list: a frame of few tiles walks ahead
(four or seven blocks a SM), a batch of the same view with many tiles does
not; both make the same bytes, in every blend mode and tile size."""

import numpy as np
import pytest

import gsplat_ffi as ffi
import gsplat_scenes
from test_gpu_parity import _render

pytestmark = pytest.mark.gpu


def _scene(n, clump):
    """n tiny splats, all but every `clump`-th around one point of the image,
    so that the lists of the other tiles are thin in their bin's."""
    rng = np.random.default_rng(n + clump)
    means = rng.uniform(-1.2, 1.2, (n, 3)).astype(np.float32)
    if clump > 1:
        near = np.arange(n) % clump != 0
        means[near, :2] = rng.normal(-0.7, 0.05, (int(near.sum()), 2))
    scene = gsplat_scenes.make_scene(rng, means, -5.0, 0.4, -2.5, 0.5, 0)
    return scene, gsplat_scenes.camera((0.0, 0.0, -4.0), (0, 0, 0), 45.0)


@pytest.mark.parametrize("w,h,tile,n,clump,views", [
    (64, 64, 16, 60_000, 40, 160),   # chunks that span up to 15 windows of the list
    (64, 64, 16, 60_000, 4, 160),    # one or two windows a chunk
    (64, 64, 16, 5_000, 1, 160),     # a list of little more than one window
    (16, 16, 16, 20_000, 1, 2600),   # every entry of the list, groups of up to 1,024 views
    (32, 32, 8, 30_000, 30, 160),    # 8x8 tiles, thin lists
    (40, 24, 8, 12_000, 2, 160),     # 8x8 tiles, bins at the image's edge
    (480, 360, 16, 50_000, 8, 3)])   # seven blocks a SM
def test_walks_agree(w, h, tile, n, clump, views):
    scene, cam = _scene(n, clump)
    for blend in (ffi.BLEND_FP32, ffi.BLEND_UNORM8):
        frame = _render(scene, cam, w, h, blend=blend, tile=tile, debug=False).readback_rgba8()
        with ffi.Batch() as b:
            sid = b.add_scene(scene)
            b.set_tile_size(tile)
            b.set_blend_mode(blend)
            b.render([(sid, cam, w, h)] * views)
            assert frame.any()
            for k in (0, views - 1):
                assert np.array_equal(b.readback_rgba8(k), frame), (blend, k)
