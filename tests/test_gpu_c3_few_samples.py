"""Megakernel at one to three samples a pixel: images whose samples are split over a
block's warps and images just too large for that, against the oracle bit for bit."""
import numpy as np
import pytest

from crender_gb300 import api, scenes
from test_gpu_c_render import _assert_identical, _box_variant, _render_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,rr", [(1, 3), (0, 0)])
@pytest.mark.parametrize("spp", [1, 2, 3])
@pytest.mark.parametrize("size", [(13, 7), (171, 171), (97, 301)])
def test_small_scene(ctx, orc, size, spp, mode, rr):
    st = api.make_settings(size[0], size[1], spp, max_bounces=4, rr_depth=rr, mode=mode, seed=91, aspect=size[0] / size[1])
    kw = dict(sun_enabled=True) if mode == 0 else {}
    _assert_identical(*_render_both(ctx, orc, _box_variant("materials"), st, passes=2, **kw))


@pytest.mark.parametrize("mode,rr", [(1, 3), (0, 0)])
@pytest.mark.parametrize("spp", [1, 2, 3, 4])
@pytest.mark.parametrize("size", [(13, 7), (152, 96), (153, 96), (304, 96), (197, 197), (198, 197), (512, 304), (513, 304)])
def test_larger_scene(ctx, orc, size, spp, mode, rr):
    sc = scenes.displaced_scene(freq=8)
    st = api.make_settings(size[0], size[1], spp, max_bounces=5, rr_depth=rr, mode=mode, seed=92, aspect=size[0] / size[1])
    _assert_identical(*_render_both(ctx, orc, sc, st, skybox=np.ones((1, 1, 4), np.float32)))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("spp", [2, 3])
@pytest.mark.parametrize("size", [(13, 7), (152, 128), (153, 128)])
def test_placements(ctx, orc, size, spp, mode):
    sc = scenes.multi_model_box()
    s = api.Scene.from_models(ctx, sc).build(8, 1)
    st = api.make_settings(size[0], size[1], spp, 5, 3 if mode else 0, mode, 93, size[0] / size[1])
    f = api.Film(ctx, st.width, st.height, f64=True, aov=True)
    try:
        api.render(s, sc["camera"], st, f)
        g = f.download(f64=True, aov=True)
    finally:
        f.close()
        s.close()
    o = orc.render(sc, sc["camera"], st)
    for k in ("sum", "sum64", "sumsq64", "albedo", "normal", "depth"):
        assert np.array_equal(g[k].view(np.uint8), o[k].view(np.uint8)), k
