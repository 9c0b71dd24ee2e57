// work_order.h — in which order and shares the kernels take their work: plain
// functions, also compiled by the host compiler for their tests.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define CRG_HD __host__ __device__ __forceinline__
#else
#define CRG_HD inline
#endif

namespace crg {

// Pixel at `place` of an image's order of work: 8 x 4 tiles, so that the 32 lanes
// of a warp start on a compact patch, whose rays share nodes for longer than a
// row's.  Tiles run along bands of four rows, then come the columns right of the
// last full tile; a last band of fewer than four rows goes row by row, as does an
// image of fewer (four rows of its width may not fit 32 bits).
CRG_HD uint32_t tile_pixel(uint32_t place, uint32_t w, uint32_t h) {
    if (h < 4u) return place;
    const uint32_t band = place / (4u * w), r = place - band * 4u * w;
    if (4u * band + 4u > h) return place;
    const uint32_t tiles = w / 8u, t = r / 32u, k = r % 32u;
    if (t < tiles) return (4u * band + k / 8u) * w + t * 8u + k % 8u;
    const uint32_t rest = w - tiles * 8u, q = r - tiles * 32u;
    return (4u * band + q / rest) * w + tiles * 8u + q % rest;
}

// Samples [begin, end) of `spp` that part `part` of `parts` takes, as even as whole
// samples allow, the later parts less.
CRG_HD void sample_share(uint32_t spp, uint32_t parts, uint32_t part, uint32_t &begin, uint32_t &end) {
    const uint32_t share = spp / parts + (spp % parts ? 1u : 0u);
    begin = part * share < spp ? part * share : spp;
    end = begin + (spp - begin < share ? spp - begin : share);
}

// Rays that a warp takes with W lanes to each, or 0: one ray per lane (`lanes`
// asks for that, and a scene without triangles has nothing to share).
//
// Few rays leave the GPU idle whatever runs them, and a call lasts as long as its
// longest ray's chain of steps.  W lanes to a ray make each step short (a child
// box per lane), and a warp to a ray keeps the rays of a warp from waiting for
// each other's branches: soup, 4,000 closest hits 107 -> 64 us, 127 on a mesh of
// 11,520 triangles 30 -> 21, at width 2 1,000 on the soup 670 -> 461.  More rays
// than warps that are resident together share them: 8,000 on the mesh take 39 us
// at one to a warp, 34 at two and 39 a lane each, 16,000 take 37 at four and 40.
// Two lanes to a ray gain little on a step: below 32 rays they lose more than the
// company costs (10K triangles at width 2: one ray 49 against 35 us, 32 rays 74 against 86).
constexpr uint64_t kFewRays = 4096;
CRG_HD uint32_t few_rays_per_warp(uint64_t n, uint32_t width, uint32_t ntri, bool lanes) {
    if (lanes || ntri == 0u || (width == 2u && n < 32u) || n > (width == 8u ? 4u * kFewRays : kFewRays)) return 0u;
    return n <= kFewRays ? 1u : n <= 2u * kFewRays ? 2u : 4u;
}

// Stage fusion (crg_wavefront_opts::fuse, 1 to 3) of a batch that asks for none, with
// `pool` paths in flight and chunks of at most `largest_chunk` samples.
//
// A small pool takes one kernel a bounce: its stages last as long as their longest
// ray's chain of steps, which fused they start only once.  Split / fused, a pool that
// holds its chunk: 4,096 paths 320 / 245 us, 20K 767 / 616, 140K 1,032 / 822, 930K
// 1,634 / 1,571, 4M 3,280 / 3,865.  A pool refilled many times keeps its kernels
// full, so the split stages win earlier: 16.8M samples of the 72K-triangle mesh at
// 2^17 paths 51.5 / 51.3 ms, at 2^19 24.3 / 35.0 (the box 33.6 / 26.5 and 23.0 / 18.9).
// Stage times are those of the split stages (host_loop 2).
CRG_HD uint32_t default_fusion(uint64_t pool, uint64_t largest_chunk, uint32_t host_loop) {
    return host_loop != 2u && pool <= (pool < largest_chunk ? 1u << 17 : 1u << 19) ? 3u : 1u;
}

} // namespace crg
