"""The kernels' order of work (csrc/work_order.h), compiled by the host compiler."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crender_gb300", "csrc")

SOURCE = """
#include "work_order.h"
extern "C" void tile_pixels(const uint32_t *place, uint32_t n, uint32_t w, uint32_t h, uint32_t *out) {
    for (uint32_t i = 0; i < n; ++i) out[i] = crg::tile_pixel(place[i], w, h);
}
extern "C" void sample_share(uint32_t spp, uint32_t parts, uint32_t part, uint32_t *out) {
    crg::sample_share(spp, parts, part, out[0], out[1]);
}
extern "C" uint32_t render_form(uint64_t npix, uint32_t spp, uint32_t ntri, uint32_t placed, uint32_t sms) {
    const crg::RenderForm f = crg::render_form(npix, spp, ntri, placed != 0, sms);
    return f.pixels << 8 | f.blocks * 2u | (f.split ? 1u : 0u);
}
extern "C" uint32_t default_fusion(uint64_t pool, uint64_t largest_chunk, uint32_t host_loop) {
    return crg::default_fusion(pool, largest_chunk, host_loop);
}
extern "C" uint32_t few_rays_per_warp(uint64_t n, uint32_t width, uint32_t ntri, uint32_t lanes) {
    return crg::few_rays_per_warp(n, width, ntri, lanes != 0);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("work_order")
    (d / "w.cpp").write_text(SOURCE)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "w.cpp"), "-o",
                    str(d / "w.so")], check=True)
    return C.CDLL(str(d / "w.so"))


def tile_pixels(lib, places, w, h):
    places = np.ascontiguousarray(places, np.uint32)
    out = np.empty_like(places)
    lib.tile_pixels(places.ctypes.data_as(C.c_void_p), C.c_uint32(len(places)), C.c_uint32(w), C.c_uint32(h),
                    out.ctypes.data_as(C.c_void_p))
    return out


@pytest.mark.parametrize("size", [(1, 1), (1, 9), (7, 3), (7, 4), (8, 4), (9, 5), (33, 6), (40, 12), (403, 301)])
def test_tiles_cover_every_pixel_once(lib, size):
    w, h = size
    assert np.array_equal(np.sort(tile_pixels(lib, np.arange(w * h), w, h)), np.arange(w * h))


@pytest.mark.parametrize("size", [(1 << 29, 4), ((1 << 29) - 3, 4), (1 << 30, 2), ((1 << 30) + 1, 1), (1 << 30, 1), (1 << 31, 1),
                                  (3, 715827882)])
def test_tiles_of_the_largest_films_stay_inside(lib, size):
    """Up to 2^31 pixels, where four rows of the widest images no longer fit 32 bits."""
    w, h = size
    n = w * h
    places = np.r_[0:64, n // 2:n // 2 + 64, n - 64:n]
    out = tile_pixels(lib, places, w, h)
    assert (out < n).all() and len(np.unique(out)) == len(places)


@pytest.mark.parametrize("parts", [1, 4])
@pytest.mark.parametrize("spp", [1, 3, 4, 5, 8, 9, 131, (1 << 31) + 1, (1 << 32) - 5, (1 << 32) - 3, (1 << 32) - 1])
def test_sample_shares_follow_one_another(lib, spp, parts):
    at = 0
    for part in range(parts):
        out = (C.c_uint32 * 2)()
        lib.sample_share(C.c_uint32(spp), C.c_uint32(parts), C.c_uint32(part), out)
        assert out[0] == at and out[0] <= out[1] <= spp and out[1] - out[0] <= -(-spp // parts)
        at = out[1]
    assert at == spp


@pytest.mark.parametrize("width", [2, 4, 8])
def test_few_rays_share_a_warp_unless_lanes_are_asked_for(lib, width):
    few = lambda n, ntri=10, lanes=0: lib.few_rays_per_warp(C.c_uint64(n), width, ntri, lanes)
    assert [few(n) for n in (1, 31, 32, 4096)] == ([0, 0, 1, 1] if width == 2 else [1, 1, 1, 1])
    assert [few(n) for n in (4097, 8192, 8193, 16384)] == ([2, 2, 4, 4] if width == 8 else [0] * 4)
    assert few(16385) == few(1 << 33) == 0
    assert few(1, ntri=0) == 0
    assert not any(few(n, lanes=1) for n in (1, 4096, 8192, 16384))


def test_default_fusion_goes_by_the_pool_and_its_refills(lib):
    fuse = lambda pool, chunk, loop=0: lib.default_fusion(C.c_uint64(pool), C.c_uint64(chunk), loop)
    assert [fuse(p, p) for p in (1, 1 << 19, (1 << 19) + 1, 1 << 27)] == [3, 3, 1, 1]
    assert [fuse(p, 1 << 24) for p in (1, 1 << 17, (1 << 17) + 1, 1 << 19)] == [3, 3, 1, 1]
    assert [fuse(1000, 1000, loop) for loop in (0, 1, 2)] == [3, 3, 1]


def test_render_form_by_samples_pixels_and_scene(lib):
    def form(npix, spp, ntri=5000, placed=0, sms=152):
        v = lib.render_form(C.c_uint64(npix), spp, ntri, placed, sms)
        return (v & 0xFF) // 2, bool(v & 1)

    def pixels(npix, spp, ntri=5000, placed=0, sms=152):
        return lib.render_form(C.c_uint64(npix), spp, ntri, placed, sms) >> 8

    lane = 6 * 152 * 128  # pixels of one wave at a lane each
    # one sample is never split; a large scene takes six blocks up to two waves, eight above
    assert [form(n, 1) for n in (1, 2 * lane, 2 * lane + 1)] == [(6, False), (6, False), (8, False)]
    assert [form(n, 1, ntri=36) for n in (1, 10 * lane)] == [(6, False)] * 2
    # two and three only where all blocks run at once, four times as many of a large scene
    assert [form(n, spp) for spp in (2, 3) for n in (4 * 32 * 8 * 152, 4 * 32 * 8 * 152 + 1)] == [(8, True), (6, False)] * 2
    assert form(2 * lane + 1, 3) == (8, False)
    assert [form(n, 2, ntri=36) for n in (32 * 6 * 152, 32 * 6 * 152 + 1)] == [(6, True), (6, False)]
    assert [form(n, 2, placed=1) for n in (32 * 4 * 152, 32 * 4 * 152 + 1)] == [(4, True), (4, False)]
    # four and more: split, but not views of four waves of a small scene without placements
    assert [form(n, 4) for n in (1, lane // 4, lane // 4 + 1, 1 << 31)] == [(6, True), (6, True), (8, True), (8, True)]
    assert [form(n, 4, ntri=36) for n in (4 * lane - 1, 4 * lane)] == [(6, True), (6, False)]
    assert form(4 * lane, 4, ntri=36, placed=1) == (4, True)
    # pixels of a warp: as few as keep all warps running at once, for a large scene unsplit
    warps = lane // 32
    assert [pixels(warps * k + d, 1) for k in (4, 8, 16) for d in (0, 1)] == [4, 8, 8, 16, 16, 32]
    assert [pixels(1, *a) for a in ((1, 36), (1, 5000, 1), (2, 5000), (4, 5000))] == [32] * 4
