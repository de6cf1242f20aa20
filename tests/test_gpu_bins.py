"""The bin pairs (4x4 tiles) and the raster's walk of a bin's list, on the GPU
against the oracle: image sizes around the edges of a tile and a bin, splats
from one tile to the whole image (a warp of the emission then has more bin
rows than it keeps), lists below and above one chunk and one 1,024-entry step."""

import numpy as np
import pytest

import gsplat_ffi as ffi
import gsplat_scenes
from conftest import assert_fp32_image
from test_gpu_parity import _compare_stages, _render

pytestmark = pytest.mark.gpu


def _scene(n, huge):
    """n small splats and `huge` that cover most of the image, interleaved."""
    rng = np.random.default_rng(n + huge)
    means = rng.normal(0.0, 0.8, (n + huge, 3)).astype(np.float32)
    scene = gsplat_scenes.make_scene(rng, means, -3.0, 0.8, -1.0, 1.0, 1)
    scene["scale_xyz"][rng.permutation(n + huge)[:huge]] += np.float32(3.0)
    return scene, gsplat_scenes.camera((0.2, 0.1, -4.0), (0, 0, 0), 55.0)


@pytest.mark.parametrize("w,h,tile,n,huge", [
    (16, 16, 16, 300, 4), (17, 1, 16, 300, 4), (64, 64, 16, 4000, 40), (65, 63, 16, 2000, 1200),
    (128, 129, 16, 700, 90), (321, 240, 16, 3000, 300), (1040, 48, 16, 300, 700),
    (31, 33, 8, 300, 20), (32, 32, 8, 3000, 40), (257, 65, 8, 900, 300), (1, 400, 8, 500, 10)])
def test_bins_against_oracle(oracle, w, h, tile, n, huge):
    scene, cam = _scene(n, huge)
    sv = oracle.SceneView(scene)
    fr = oracle.Frame(sv, cam, w, h, tile=tile)
    ctx = _render(scene, cam, w, h, tile=tile)
    _compare_stages(ctx, fr, sv)
    assert_fp32_image(ctx.readback_rgba8(), fr.raster_tiles_fp32())
    unorm = _render(scene, cam, w, h, blend=ffi.BLEND_UNORM8, tile=tile, debug=False)
    assert np.array_equal(unorm.readback_rgba8(), fr.raster_unorm8())


def test_views_past_the_bins_of_one_run():
    """600 views of 512 bins each (2^18 bins are the most of one run): two
    launch groups, every image the plain frame's."""
    scene, cam = _scene(150, 3)
    with ffi.Batch() as b:
        sid = b.add_scene(scene)
        b.set_tile_size(8)
        rng = np.random.default_rng(1)
        cams = [gsplat_scenes.orbit_camera(rng, (3.0, 5.0)) for _ in range(600)]
        t = b.render([(sid, c, 16384, 8) for c in cams])
        assert t.groups == 2
        assert [b.view_stats(k).group for k in (0, 511, 512, 599)] == [0, 0, 1, 1]
        for k in (0, 511, 512, 599):
            ctx = _render(scene, cams[k], 16384, 8, tile=8, debug=False)
            assert np.array_equal(b.readback_rgba8(k), ctx.readback_rgba8()), k
            assert b.view_stats(k).tile_pairs == ctx.frame_counts().tile_keys


@pytest.mark.parametrize("w,h,tile", [
    (1100, 1000, 16),  # 288 bins: one pass of 512 digits
    (2048, 128, 8),    # 256 bins: the last of one 8-bit pass
    (700, 900, 8),     # 638 bins: one pass of 1,024 digits
    (1024, 1024, 8),   # 1,024 bins: the last of it
    (1100, 1000, 8)])  # 1,120 bins: two 8-bit passes
def test_bin_sort_digits(oracle, w, h, tile):
    """The tile lists over every kind of bin sort, with several sort tiles."""
    scene, cam = _scene(30_000, 40)
    sv = oracle.SceneView(scene)
    fr = oracle.Frame(sv, cam, w, h, tile=tile)
    ctx = _render(scene, cam, w, h, tile=tile)
    _compare_stages(ctx, fr, sv)
