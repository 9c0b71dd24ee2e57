"""Wavefront form, its split stages asked for by name: small batches take the
fused kernel by default, so what is tested here at small sizes gives `fuse`."""
import numpy as np
import pytest

from crender_gb300 import api, scenes
from test_gpu_c_render import _box_variant
from test_gpu_d_wavefront import OFF, _mega, _same
from test_gpu_h_textures import gpu_scene as textured_scene

pytestmark = pytest.mark.gpu

TIMEOUT = 4  # CRG_ERR_TIMEOUT


@pytest.mark.parametrize("cap", [1, 3, 7])
@pytest.mark.parametrize("opts", [dict(fuse=1), dict(fuse=1, path_pool=96), dict(fuse=1, path_pool=96, refill=OFF),
                                  dict(fuse=2, path_pool=96), dict(fuse=3, path_pool=96)])
@pytest.mark.parametrize("host_loop", [1, 2])
def test_iteration_cap_in_the_host_driven_loop(ctx, opts, cap, host_loop):
    """The host polls every eighth iteration only, so iterations follow the one that
    reached the cap: they take up nothing, and the same context then renders."""
    sc = _box_variant("materials")
    s = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    st = api.make_settings(32, 32, 3, max_bounces=8, rr_depth=0, mode=1, seed=6)
    view = [(0, sc["camera"], st)]
    f, g = api.Film(ctx, 32, 32, f64=True), api.Film(ctx, 32, 32, f64=True)
    try:
        stats = []
        for loop in (0, host_loop):  # the graph stops at the cap itself
            assert api.render_batch([s], view, [f], dict(opts, max_iterations=cap, host_loop=loop)) == TIMEOUT
            stats.append(api.batch_stats(ctx))
            f.reset()
        assert stats[0] == stats[1] and stats[0]["iterations"] == cap
        ctx.check(api.render_batch([s], view, [g], dict(opts, host_loop=host_loop)))
        _same(g.download(f64=True), _mega(ctx, s, sc["camera"], st))
    finally:
        f.close()
        g.close()
        s.close()


@pytest.mark.parametrize("opts", [dict(fuse=1), dict(fuse=1, path_pool=1000, refill=8), dict(fuse=1, refill=OFF), dict(fuse=2)])
def test_textures(ctx, opts):
    """Texture colours through the hit records that extend hands to shade."""
    sc = scenes.textured_box()
    s = textured_scene(ctx, sc)
    views = [(0, sc["camera"], api.make_settings(96, 64, 8, 8, 3, 1, 4, 1.5)),
             (0, sc["camera"], api.make_settings(40, 40, 16, 8, 3, 0, 5))]
    films = [api.Film(ctx, st.width, st.height, f64=True) for _, _, st in views]
    try:
        ctx.check(api.render_batch([s], views, films, opts))
        for (_, cam, st), f in zip(views, films):
            _same(f.download(f64=True), _mega(ctx, s, cam, st))
    finally:
        for f in films:
            f.close()
        s.close()


@pytest.mark.parametrize("opts", [dict(fuse=1), dict(fuse=1, path_pool=200)])
def test_displaced_mesh(ctx, opts):
    sc = scenes.displaced_scene(freq=40)
    s = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    s.set_skybox(sc["skybox"])
    st = api.make_settings(24, 14, 2, 16, 3, 1, 7, 24 / 14)
    f = api.Film(ctx, 24, 14, f64=True)
    try:
        ctx.check(api.render_batch([s], [(0, sc["camera"], st)], [f], opts))
        _same(f.download(f64=True), _mega(ctx, s, sc["camera"], st))
    finally:
        f.close()
        s.close()


def test_accumulates_after_megakernel_passes(ctx):
    sc = _box_variant("plain")
    s = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    st = api.make_settings(24, 24, 3, 8, 3, 1, 5)
    f = api.Film(ctx, 24, 24, f64=True)
    try:
        api.render(s, sc["camera"], st, f)
        ctx.check(api.render_batch([s], [(0, sc["camera"], st)], [f], dict(fuse=1)))
        assert f.spp == 6
        _same(f.download(f64=True), _mega(ctx, s, sc["camera"], st, passes=2))
    finally:
        f.close()
        s.close()


@pytest.mark.parametrize("size,spp", [((1, 1), 1), ((31, 1), 1), ((33, 1), 3), ((37, 29), 5)])
@pytest.mark.parametrize("opts", [dict(fuse=1), dict(fuse=1, path_pool=33), dict(fuse=1, path_pool=100, refill=8),
                                  dict(fuse=1, path_pool=33, refill=1, block_size=64)])
def test_queue_edges_with_refill(ctx, size, spp, opts):
    """Queues of a few entries and pools that are no multiple of a warp, lanes refilled."""
    sc = _box_variant("materials")
    s = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    st = api.make_settings(size[0], size[1], spp, max_bounces=8, rr_depth=3, mode=1, seed=31, aspect=size[0] / size[1])
    f = api.Film(ctx, size[0], size[1], f64=True)
    try:
        ctx.check(api.render_batch([s], [(0, sc["camera"], st)], [f], opts))
        _same(f.download(f64=True), _mega(ctx, s, sc["camera"], st))
    finally:
        f.close()
        s.close()


@pytest.mark.parametrize("host_loop", [0, 1])
def test_async_cap_arrives_with_the_wait(ctx, host_loop):
    sc = _box_variant("plain")
    s = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    st = api.make_settings(32, 32, 8, 8, 3, 1, 6)
    view = [(0, sc["camera"], st)]
    f, g = api.Film(ctx, 32, 32, f64=True), api.Film(ctx, 32, 32, f64=True)
    try:
        opts = dict(fuse=1, host_loop=host_loop)
        assert api.render_batch([s], view, [f], dict(opts, max_iterations=2), wait=False) == 0
        assert api.render_batch([s], view, [g], opts, wait=False) == 0
        assert api.batch_wait(ctx) == TIMEOUT
        assert api.batch_wait(ctx) == 0
        _same(g.download(f64=True), _mega(ctx, s, sc["camera"], st))
    finally:
        f.close()
        g.close()
        s.close()
