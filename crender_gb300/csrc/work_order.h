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

// Form of the megakernel for an image: a pixel's samples split over a block's four
// warps or not, blocks of 128 threads per SM (4 with placements), and pixels of a
// warp where it has them to itself.
//
// Blocks: a few triangles lie in L1 and the kernel is bound by issue: six (80
// registers; 12.7 ms on the box's 36 triangles, 13.9 at eight); more wait on loads:
// eight (64 registers; 4.63 against 4.67 ms at 1,602 triangles, 7.06 against 7.41 at
// 33K, 12.65 against 13.59 at 4.2M), but six where an image fills those once (split)
// or twice, which gains little from more and loses what spills cost (72K triangles
// 64x64x1 226 against 220 us, 100x75x1 269 / 261, 256x256x1 317 / 307; 44K triangles
// 477x315x1 411 / 396 with the faithful estimator, 560x380x1 711 / 697 with the other).
//
// Split: a quarter of the pixels then fills the GPU, the end of the launch is evened
// out and a tile's rays stay in one SM's L1: mesh 1920x1080x4 12.4 -> 11.6 ms,
// 174x136x229 98 -> 35, box 65x70x256 14.7 -> 4.6, 517x333x64 6.3 -> 5.9.  A view of a
// small scene that fills the GPU four times only pays for the rounds (box 800x600x16
// 4.45 -> 4.59, 1920x1080x16 13.1 -> 14.7); from twice on it goes either way by the
// view (512x512x64 11.8 -> 12.4, 700x500x64 13.3 -> 12.6).  Two or three samples leave
// warps of a block idle, so they are split only where all blocks run at once, or up to
// four times as many where rays wait on memory: 72K triangles 64x64x2 366 -> 216 us
// (327 on a traversal per thread), 64x64x3 532 -> 218 (505), 400x300x2 489 -> 334,
// 640x480x2 637 -> 626, 1283x721x2 1,164 -> 1,340; six placements 160x120x2 254 -> 143,
// 256x256x2 353 -> 406; the box 160x120x2 138 -> 86, 256x256x2 162 -> 186.
//
// Pixels of a warp: an image of one sample that leaves warps idle lasts as long as its
// slowest warp, and a warp of fewer pixels is faster: its lanes without a ray test
// triangles only.  A large scene takes 16, 8 or 4 where the warps then still run at
// once, against 32 (and a traversal per thread): 11K triangles 80x75x1 with 16 bounces
// 456 -> 243 us at 4 (346), 480K triangles 254x96x1 529 -> 365 at 8 (495), 200x200x1
// 642 -> 486 at 16 (546); 380x300x1, too large for 16, 674 against 658.
struct RenderForm {
    bool split;
    uint32_t blocks, pixels;
};
CRG_HD RenderForm render_form(uint64_t npix, uint32_t spp, uint32_t ntri, bool placed, uint32_t sms) {
    const bool small = ntri < 1024u;
    const uint64_t wave = 6ull * sms * 128ull; // pixels that six blocks per SM hold, a lane each
    RenderForm f{};
    f.blocks = placed ? 4u : small ? 6u : 8u;
    if (spp >= 4u) f.split = !(small && !placed && npix >= 4u * wave);
    else f.split = spp >= 2u && npix <= (f.blocks == 8u ? 4u : 1u) * 32ull * f.blocks * sms;
    f.pixels = 32u;
    if (f.blocks == 8u && !f.split)
        while (f.pixels > 4u && npix * 64u <= wave * f.pixels) f.pixels /= 2u;
    if (f.blocks == 8u && npix * (f.split ? 4u : 1u) <= (f.split ? wave : 2u * wave)) f.blocks = 6u;
    return f;
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
