"""crg_post_process (the post-processor's bloom / gray-scale / tone-mapping passes as
CUDA kernels) against the CPU oracle, through the C ABI.  Bit-exact except for the
gamma step's powf, which CUDA documents to within 4 ulp of the exact result (the
oracle's glibc powf is within 1): that tolerance is written below."""
import numpy as np
import pytest

from crender_gb300 import _abi, api, scenes
from test_post_cpu import CASES, hdr_image, settings, ulp_diff, uses_pow

pytestmark = pytest.mark.gpu

POW_ULP = 5  # CUDA powf (<= 4 ulp) vs glibc powf (< 1 ulp)


def run_gpu(ctx, img, s):
    h, w = img.shape[:2]
    src = api.DeviceBuffer.from_array(ctx, np.ascontiguousarray(img, np.float32))
    dst = api.DeviceBuffer(ctx, img.nbytes)
    api.post_process(ctx, src, dst, w, h, s)
    out = dst.download(np.zeros_like(img, np.float32))
    src.free()
    dst.free()
    return out


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("shape", [(512, 512), (250, 130), (37, 300), (1920, 1080)])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_post_matches_oracle(ctx, orc, mode, shape, case):
    w, h = shape
    img = hdr_image(w, h, 11 + case)
    s = settings(mode=mode, **CASES[case])
    got = run_gpu(ctx, img, s)
    want = orc.post_process(img, s)
    assert ulp_diff(got, want) <= (POW_ULP if uses_pow(s) else 0)


def test_no_effect_copies(ctx):
    img = hdr_image(64, 33, 2)
    assert np.array_equal(run_gpu(ctx, img, api.post_settings()), img)


def test_defaults_match_the_reference():
    s = api.post_settings()
    assert (s.bloom, s.gray_scale, s.tonemapping, s.tonemap_type, s.mode) == (0, 0, 0, 0, 0)
    assert np.float32(s.bloom_threshold) == np.float32(0.7) and s.bloom_strength == 1.0
    assert s.exposure == 1.0 and np.float32(s.gamma) == np.float32(2.2)


def test_render_display_post_chain(ctx, orc):
    """Box render -> crg_film_display -> crg_post_process (the export path of the
    reference UI, src/ui/ui.h:604-628), checked against the oracle on the same
    display image."""
    sc = scenes.box_scene()
    W = H = 128
    st = api.make_settings(W, H, 16, 8, 3, 1, 5)
    scene = api.Scene(ctx, sc["verts"], sc["mat_idx"], sc["mats"]).build()
    film = api.Film(ctx, W, H)
    api.render(scene, sc["camera"], st, film)
    disp = api.DeviceBuffer(ctx, W * H * 16)
    api.film_display(film, disp)
    out = api.DeviceBuffer(ctx, W * H * 16)
    s = api.post_settings(bloom=1, bloom_threshold=0.6, tonemapping=1, tonemap_type=_abi.TONEMAP_UNCHARTED)
    api.post_process(ctx, disp, out, W, H, s)
    img = disp.download(np.zeros((H, W, 4), np.float32))
    got = out.download(np.zeros((H, W, 4), np.float32))
    assert ulp_diff(got, orc.post_process(img, s)) <= POW_ULP
    assert np.isfinite(got).all() and got[..., :3].max() > 0
    for b in (disp, out):
        b.free()
    film.close()
    scene.close()


def test_bad_arguments(ctx):
    b = api.DeviceBuffer(ctx, 64 * 64 * 16)
    s = api.post_settings(bloom=1)
    lib = ctx.lib
    assert lib.crg_post_process(ctx.h, b.ptr, b.ptr, 64, 64, s, None) == 1  # aliasing
    c = api.DeviceBuffer(ctx, 64 * 64 * 16)
    assert lib.crg_post_process(ctx.h, b.ptr, c.ptr, 0, 64, s, None) == 1
    s.mode = 9
    assert lib.crg_post_process(ctx.h, b.ptr, c.ptr, 64, 64, s, None) == 1
    b.free()
    c.free()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("shape", [(1, 1), (7, 27), (8, 28), (15, 29), (31, 113), (33, 8), (40, 64), (1931, 1093)])
def test_blur_tile_edges_bit_exact(ctx, orc, mode, shape):
    """Bloom alone (no powf) at the edges of the blur's tiles: widths around 8 and 32,
    heights around 28 rows and, for the last size, 112."""
    w, h = shape
    img = hdr_image(w, h, 91)
    s = settings(mode=mode, bloom=1, bloom_threshold=0.4, bloom_strength=0.8)
    assert ulp_diff(run_gpu(ctx, img, s), orc.post_process(img, s)) == 0
