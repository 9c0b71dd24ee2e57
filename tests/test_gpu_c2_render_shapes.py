"""Megakernel variants by image and scene size (6 or 8 blocks per SM, samples split
over a block's warps or not) against the oracle bit for bit, on images whose sides are no multiples
of the 8 x 4 tiles."""
import numpy as np
import pytest

from crender_gb300 import api, scenes
from test_gpu_c_render import _assert_identical, _box_variant, _render_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,rr", [(1, 3), (0, 0)])
@pytest.mark.parametrize("size", [(403, 301), (1, 5), (7, 3), (9, 4), (33, 6)])
def test_small_scene(ctx, orc, size, mode, rr):
    st = api.make_settings(size[0], size[1], 2, max_bounces=5, rr_depth=rr, mode=mode, seed=71, aspect=size[0] / size[1])
    kw = dict(sun_enabled=True) if mode == 0 else {}
    _assert_identical(*_render_both(ctx, orc, _box_variant("materials"), st, passes=2, **kw))


@pytest.mark.parametrize("mode,rr", [(1, 3), (0, 0)])
@pytest.mark.parametrize("spp", [3, 4, 5, 7, 63, 64, 65, 131])
def test_split_samples(ctx, orc, spp, mode, rr):
    """Samples of a pixel over a block's four warps: counts around 4, the round of 64
    and its quarters, on an image that leaves part of its last tile empty."""
    st = api.make_settings(13, 7, spp, max_bounces=4, rr_depth=rr, mode=mode, seed=73, aspect=13 / 7)
    _assert_identical(*_render_both(ctx, orc, _box_variant("materials"), st, passes=2))


def test_whole_warps_of_many_pixels(ctx, orc):
    """Enough pixels of a small scene that its samples are not split."""
    st = api.make_settings(801, 603, 4, max_bounces=2, rr_depth=0, mode=1, seed=74, aspect=801 / 603)
    _assert_identical(*_render_both(ctx, orc, _box_variant("materials"), st))


@pytest.mark.parametrize("mode,rr", [(1, 3), (0, 0)])
@pytest.mark.parametrize("size", [(401, 303), (61, 47)])
def test_larger_scene(ctx, orc, size, mode, rr):
    sc = scenes.displaced_scene(freq=8)
    st = api.make_settings(size[0], size[1], 1, max_bounces=8, rr_depth=rr, mode=mode, seed=72, aspect=size[0] / size[1])
    _assert_identical(*_render_both(ctx, orc, sc, st, skybox=np.ones((1, 1, 4), np.float32)))
