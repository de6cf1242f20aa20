"""Routes that a plain frame does not reach: the one wide pass of the bin sort
over many views with partial bins, and the list walked ahead in a persistent
grid whose blocks take several tiles each. Both against plain frames, bit for
bit."""

import numpy as np
import pytest

import gsplat_ffi as ffi
import gsplat_scenes

pytestmark = pytest.mark.gpu

SIZES = [(130, 70), (65, 65), (16, 200), (255, 33)]  # 6, 4, 4 and 4 bins, partial ones among them


def _scene(n, seed):
    rng = np.random.default_rng(seed)
    return gsplat_scenes.make_scene(rng, rng.normal(0.0, 0.8, (n, 3)), -2.5, 0.8, 0.0, 1.0, 1)


def _frame(scene, cam, w, h, **shape):
    with ffi.Context(w, h) as ctx:
        ctx.load_scene(scene)
        ctx.set_camera(cam)
        if shape:
            ctx.set_raster_config(**shape)
        ctx.render_frame()
        return ctx.readback_rgba8()


@pytest.mark.parametrize("count,bins", [(57, 258), (114, 514), (227, 1022)])
def test_wide_pass_over_many_views(count, bins):
    """258 bins take the pass of 512 digits, 514 and 1,022 that of 1,024."""
    scenes = [_scene(700, 1), _scene(90, 2)]
    rng = np.random.default_rng(count)
    views = [(k % 2, gsplat_scenes.orbit_camera(rng, (3.0, 6.0)), *SIZES[k % 4])
             for k in range(count)]
    assert sum(-(-w // 64) * -(-h // 64) for *_, w, h in views) == bins
    with ffi.Batch() as b:
        for s in scenes:
            b.add_scene(s)
        assert b.render(views).groups == 1
        for k in list(range(0, count, 13)) + [count - 1]:
            sid, cam, w, h = views[k]
            assert np.array_equal(b.readback_rgba8(k), _frame(scenes[sid], cam, w, h)), k


@pytest.mark.parametrize("w,h", [(500, 480), (400, 320)])  # 960 and 500 tiles: 7 and 4 an SM
@pytest.mark.parametrize("blocks_per_sm", [1, 2])
def test_persistent_blocks_walk_ahead(w, h, blocks_per_sm):
    scene = _scene(20_000, 3)
    cam = gsplat_scenes.camera((0.2, 0.1, -4.0), (0, 0, 0), 55.0)
    one = _frame(scene, cam, w, h, chunk=64)
    assert np.array_equal(_frame(scene, cam, w, h, chunk=256, blocks_per_sm=blocks_per_sm), one)
