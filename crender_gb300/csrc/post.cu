// post.cu — image post-processing (bloom, gray scale, tone mapping).
//
// Restates cr::post_processor::process (CRender
// src/render/post/post_processor.cpp:110-307) and its two compute shaders
// (assets/app/shaders/blur.comp, post_process.comp) as CUDA kernels on RGBA32F
// device images.  The passes and their order are the reference's:
//
//   bloom:  threshold (_brightness) -> 10 separable blur passes, horizontal
//           on even passes, ping-ponging between two images (_blur)
//   final:  source (+ bloom * strength) -> gray scale -> tone mapping
//
// Every float operation is written in the shader's order and compiled
// without contraction (-fmad=false), so results equal the oracle's CPU
// restatement bit for bit except where powf is involved (tone-mapping gamma).
//
// The blur's ten passes run as five kernels (k_bloom), each a horizontal and the
// following vertical pass on a tile whose horizontal result stays in shared
// memory.  Between them the image lies in three float planes: the passes write
// alpha 1 (0 outside the covered region) and nothing reads it.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "crg_internal.h"

namespace crg {
namespace {

// blur.comp:11-19 (the GLSL float array)
constexpr float kBlurW[8] = {0.19744746769063704f, 0.1746973469158936f, 0.12099884565428047f,
                                0.06560233156931679f, 0.027839605612666265f, 0.009246250740395456f,
                                0.002403157286908872f, 0.00048872837522002f};

struct PostDims {
    uint32_t w, h;   // image size
    uint32_t rw, rh; // region the reference's dispatches cover (8 * floor(n / 8) in FAITHFUL mode)
    uint32_t faithful;
    float threshold;
};

// _brightness (post_processor.cpp:296-307) visits pixel (i % w, i / h) for
// i < w*h.  Pixel (x, y) is visited iff some i = x + k*w lies in [y*h, y*h + h)
// and below w*h; visits are idempotent, so one visit decides.
__device__ __forceinline__ bool bright_visited(uint32_t x, uint32_t y, const PostDims &p) {
    if (!p.faithful) return true;
    const unsigned long long lo = (unsigned long long)y * p.h;
    const unsigned long long i0 = lo + ((unsigned long long)x + p.w - lo % p.w) % p.w;
    return i0 < lo + p.h && i0 < (unsigned long long)p.w * p.h;
}

__device__ __forceinline__ float4 bright(float4 c, uint32_t x, uint32_t y, const PostDims &p) {
    if (!bright_visited(x, y, p)) return c;
    // glm::dot(vec3, vec3(0.2126, 0.7152, 0.0722)): (x*bx + y*by) + z*bz
    const float l = (c.x * 0.2126f + c.y * 0.7152f) + c.z * 0.0722f;
    if (l < p.threshold) return make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    return c;
}

// blur.comp:21-44 for N neighbouring pixels of a line: centre * w0, then +i and
// -i for i = 1..7.  v holds their values with seven more on either side.  Two
// pixels N / 2 apart go through each instruction: the packed operations round
// each half as the scalar ones do.  The compiler contracts a packed product and
// sum into an FMA even where scalar ones may not be, so the product is an FMA
// itself, with the -0 (which leaves it exact) handed in at run time.
template <int N>
__device__ __forceinline__ void blur_taps(const float *v, float *out, float neg_zero) {
    constexpr int H = N / 2;
    const float2 zero = make_float2(neg_zero, neg_zero);
    auto times = [&](int k, int i) {
        constexpr float w[8] = {kBlurW[0], kBlurW[1], kBlurW[2], kBlurW[3], kBlurW[4], kBlurW[5], kBlurW[6], kBlurW[7]};
        return __ffma2_rn(make_float2(v[k], v[k + H]), make_float2(w[i], w[i]), zero);
    };
#pragma unroll
    for (int j = 0; j < H; ++j) {
        float2 r = times(j + 7, 0);
#pragma unroll
        for (int i = 1; i < 8; ++i) {
            r = __fadd2_rn(r, times(j + 7 + i, i));
            r = __fadd2_rn(r, times(j + 7 - i, i));
        }
        out[j] = r.x;
        out[j + H] = r.y;
    }
}

// post_process.comp:48-51 / 74-108 tone curves
__device__ __forceinline__ float uncharted_map(float x) {
    const float A = 0.15f, B = 0.50f, C = 0.10f, D = 0.20f, E = 0.02f, F = 0.30f;
    return ((x * (A * x + C * B) + D * E) / (x * (A * x + B) + D * F)) - E / F;
}

__device__ __forceinline__ float gamma_of(float c, float inv_gamma) { return powf(c, inv_gamma); }

// What the curves need that does not depend on the pixel.
struct ToneConst {
    float inv_gamma, white; // 1 / gamma; 1 / Hable's curve at the white point
};
__device__ __forceinline__ ToneConst tone_const(const crg_post_settings &s) {
    return ToneConst{1.0f / s.gamma, 1.0f / uncharted_map(11.2f)};
}

__device__ __forceinline__ float3 tonemap(float3 c, const crg_post_settings &s, const ToneConst &t) {
    const float e = s.exposure;
    const float ig = t.inv_gamma;
    switch (s.tonemap_type) {
    case CRG_TONEMAP_LINEAR:
        c = make_float3(c.x * e, c.y * e, c.z * e);
        return make_float3(gamma_of(c.x, ig), gamma_of(c.y, ig), gamma_of(c.z, ig));
    case CRG_TONEMAP_REINHARD:
        c = make_float3(c.x * e, c.y * e, c.z * e);
        c = make_float3(c.x / (c.x + 1.0f), c.y / (c.y + 1.0f), c.z / (c.z + 1.0f));
        return make_float3(gamma_of(c.x, ig), gamma_of(c.y, ig), gamma_of(c.z, ig));
    case CRG_TONEMAP_JIM_RICHARD: {
        c = make_float3(c.x * e, c.y * e, c.z * e);
        const float x = fmaxf(0.0f, c.x - 0.004f), y = fmaxf(0.0f, c.y - 0.004f), z = fmaxf(0.0f, c.z - 0.004f);
        return make_float3((x * (6.2f * x + 0.5f)) / (x * (6.2f * x + 1.7f) + 0.06f),
                           (y * (6.2f * y + 0.5f)) / (y * (6.2f * y + 1.7f) + 0.06f),
                           (z * (6.2f * z + 0.5f)) / (z * (6.2f * z + 1.7f) + 0.06f));
    }
    case CRG_TONEMAP_UNCHARTED: {
        c = make_float3(c.x * e, c.y * e, c.z * e);
        const float ws = t.white;
        c = make_float3(uncharted_map(2.0f * c.x) * ws, uncharted_map(2.0f * c.y) * ws, uncharted_map(2.0f * c.z) * ws);
        return make_float3(gamma_of(c.x, ig), gamma_of(c.y, ig), gamma_of(c.z, ig));
    }
    default:
        return c;
    }
}

// post_process.comp:116-136 for one pixel: the source colour, the blurred one.
__device__ __forceinline__ float4 compose(float4 v, float3 b, const crg_post_settings &s, const ToneConst &t) {
    float3 f = make_float3(v.x, v.y, v.z);
    if (s.bloom) {
        const float k = s.bloom_strength;
        f = make_float3(f.x + b.x * k, f.y + b.y * k, f.z + b.z * k);
    }
    if (s.gray_scale) {
        const float g = (0.2126f * f.x + 0.7162f * f.y) + 0.0722f * f.z;
        f = make_float3(g, g, g);
    }
    if (s.tonemapping) f = tonemap(f, s, t);
    return make_float4(f.x, f.y, f.z, 1.0f);
}

// The chain without bloom.
__global__ void __launch_bounds__(256) k_post_final(const float4 *__restrict__ src, float4 *__restrict__ dst, PostDims p,
                                                    crg_post_settings s) {
    const size_t n = (size_t)p.w * p.h;
    const ToneConst tone = tone_const(s);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t x = (uint32_t)(i % p.w), y = (uint32_t)(i / p.w);
        float4 out = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (x < p.rw && y < p.rh) out = compose(src[i], make_float3(0.0f, 0.0f, 0.0f), s, tone);
        dst[i] = out;
    }
}

// _brightness into three float planes.
__global__ void __launch_bounds__(256) k_bright(const float4 *__restrict__ src, float *__restrict__ out, PostDims p,
                                                uint32_t pitch) {
    const uint32_t x = blockIdx.x * 256u + threadIdx.x, y = blockIdx.y;
    if (x >= p.w) return;
    const size_t plane = (size_t)pitch * p.h, o = (size_t)y * pitch + x;
    const float4 c = bright(__ldg(&src[(size_t)y * p.w + x]), x, y, p);
    out[o] = c.x;
    out[plane + o] = c.y;
    out[2 * plane + o] = c.z;
}

// A horizontal and the following vertical blur pass on tiles of 32 columns x 7 N
// rows, one float plane at a time.  Horizontally a thread forms eight
// neighbouring pixels from six 16-byte loads, vertically N pixels of a column
// from N + 14 shared values, so that at N = 16 a pixel costs 2.75 and 1.9 reads
// instead of 15; the rows above and below the tile (126 of 112) are blurred
// twice.  LAST: the blurred tile goes into the final composition, not to memory.
// Bound by the arithmetic, which may not be contracted (29 operations a pixel,
// pass and channel: 0.2 ms for 3840x2160 if nothing else were issued); 4 blocks
// of 224 per SM (2 / 3 / 4: 664 / 548 / 498 us for the whole chain, against 917 us
// for a kernel per pass with 15 shared reads of 16 bytes a pixel).
// Pixels outside the covered region come out as zero from each pass, as the
// reference clears its target before each dispatch.
// N: pixels of a column that a thread forms; the tile has seven strips of N rows.
constexpr int kTileW = 32, kHalo = 7, kStrips = 7, kBloomThreads = 32 * kStrips;

template <bool LAST, int N>
__global__ void __launch_bounds__(kBloomThreads, 4) k_bloom(const float *__restrict__ in, float *__restrict__ out,
                                                               const float4 *__restrict__ src, float4 *__restrict__ dst,
                                                               PostDims p, uint32_t pitch, crg_post_settings set, float neg_zero) {
    constexpr int kTileH = kStrips * N, kTileRows = kTileH + 2 * kHalo;
    __shared__ float s_row[3][kTileRows][kTileW]; // the horizontal pass's result
    const int x0 = (int)(blockIdx.x * kTileW), y0 = (int)(blockIdx.y * kTileH) - kHalo;
    const size_t plane = (size_t)pitch * p.h;
    constexpr int kGroups = kTileW / 8;
    for (int task = (int)threadIdx.x; task < kTileRows * kGroups * 3; task += kBloomThreads) {
        const int g = task % kGroups, line_of = task / kGroups;
        const int ch = line_of / kTileRows, row = line_of - ch * kTileRows;
        const int x = x0 + 8 * g, y = y0 + row;
        float r[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (y >= 0 && y < (int)p.rh && x < (int)p.rw) {
            const float *line = in + ch * plane + (size_t)y * pitch;
            float v[24]; // pixels x - 8 .. x + 15
            if (x >= 8 && x + 16 <= (int)p.w) {
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const float4 f = __ldg(reinterpret_cast<const float4 *>(line + x - 8) + q);
                    v[4 * q] = f.x;
                    v[4 * q + 1] = f.y;
                    v[4 * q + 2] = f.z;
                    v[4 * q + 3] = f.w;
                }
            } else {
#pragma unroll
                for (int k = 1; k < 23; ++k) {
                    const int xx = x + k - 8;
                    v[k] = xx >= 0 && xx < (int)p.w ? __ldg(line + xx) : 0.0f;
                }
            }
            blur_taps<8>(v + 1, r, neg_zero);
            if (x + 8 > (int)p.rw)
#pragma unroll
                for (int j = 0; j < 8; ++j) r[j] = x + j < (int)p.rw ? r[j] : 0.0f;
        }
        float4 *d = reinterpret_cast<float4 *>(&s_row[ch][row][8 * g]);
        d[0] = make_float4(r[0], r[1], r[2], r[3]);
        d[1] = make_float4(r[4], r[5], r[6], r[7]);
    }
    __syncthreads();
    const int lane = (int)(threadIdx.x & 31u), strip = (int)(threadIdx.x >> 5) * N;
    const int x = x0 + lane, yt = y0 + kHalo + strip;
    float r[LAST ? 3 : 1][N];
#pragma unroll(LAST ? 3 : 1)
    for (int c = 0; c < 3; ++c) {
        float v[N + 14];
#pragma unroll
        for (int k = 0; k < N + 14; ++k) v[k] = s_row[c][strip + k][lane];
        blur_taps<N>(v, r[LAST ? c : 0], neg_zero);
        if (!LAST && x < (int)p.w) {
            float *o = out + c * plane + (size_t)yt * pitch + x;
            if (x < (int)p.rw && yt + N <= (int)p.rh) {
#pragma unroll
                for (int j = 0; j < N; ++j) o[(size_t)j * pitch] = r[0][j];
            } else {
#pragma unroll
                for (int j = 0; j < N; ++j)
                    if (yt + j < (int)p.h) o[(size_t)j * pitch] = x < (int)p.rw && yt + j < (int)p.rh ? r[0][j] : 0.0f;
            }
        }
    }
    if (LAST) {
        __syncthreads();
        // the strip's own values through shared memory: a loop over them must not be unrolled (the tone
        // curves are some 300 instructions a pixel)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int j = 0; j < N; ++j) s_row[c][strip + j][lane] = r[LAST ? c : 0][j];
        if (x >= (int)p.w) return;
        const ToneConst tone = tone_const(set);
#pragma unroll 1
        for (int j = 0; j < N && yt + j < (int)p.h; ++j) {
            const int y = yt + j;
            const size_t i = (size_t)y * p.w + x;
            float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (x < (int)p.rw && y < (int)p.rh)
                o = compose(__ldg(&src[i]), make_float3(s_row[0][strip + j][lane], s_row[1][strip + j][lane],
                                                        s_row[2][strip + j][lane]), set, tone);
            dst[i] = o;
        }
    }
}

} // namespace
} // namespace crg

using namespace crg;

extern "C" crg_status crg_post_settings_default(crg_post_settings *s) {
    if (!s) return CRG_ERR_INVALID_ARG;
    *s = crg_post_settings{};
    s->bloom = 0;
    s->bloom_threshold = 0.7f;
    s->bloom_strength = 1.0f;
    s->gray_scale = 0;
    s->tonemapping = 0;
    s->tonemap_type = CRG_TONEMAP_LINEAR;
    s->exposure = 1.0f;
    s->gamma = 2.2f;
    s->mode = CRG_POST_FAITHFUL;
    return CRG_OK;
}

extern "C" crg_status crg_post_process(crg_context *ctx, const float *d_src, float *d_dst, uint32_t width,
                                       uint32_t height, const crg_post_settings *settings, crg_stream stream) {
    if (!ctx || !d_src || !d_dst || !settings) return set_error(ctx, CRG_ERR_INVALID_ARG, "null argument");
    if (width == 0 || height == 0) return set_error(ctx, CRG_ERR_INVALID_ARG, "empty image");
    if (width > 65536u * 256u || height > 65535u) return set_error(ctx, CRG_ERR_INVALID_ARG, "image too large");
    if (d_src == d_dst) return set_error(ctx, CRG_ERR_INVALID_ARG, "source and destination alias");
    const crg_post_settings &s = *settings;
    if (s.mode > CRG_POST_FULL) return set_error(ctx, CRG_ERR_INVALID_ARG, "bad post-process mode");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t npix = (size_t)width * height;
    if (!s.bloom && !s.gray_scale && !s.tonemapping) {
        // post_processor.cpp:112-114: nothing enabled returns the input
        CRG_CUDA(ctx, cudaMemcpyAsync(d_dst, d_src, npix * 16, cudaMemcpyDeviceToDevice, st));
        return CRG_OK;
    }
    PostDims p;
    p.w = width;
    p.h = height;
    p.faithful = s.mode == CRG_POST_FAITHFUL;
    p.rw = p.faithful ? width / 8 * 8 : width;
    p.rh = p.faithful ? height / 8 * 8 : height;
    p.threshold = s.bloom_threshold;
    const float4 *src = (const float4 *)d_src;
    if (s.bloom) {
        // _blur (post_processor.cpp:246-294): ten passes, even ones horizontal, two to a kernel
        const uint32_t pitch = (width + 3) / 4 * 4;
        const size_t image = sizeof(float) * 3 * (size_t)pitch * height;
        crg_status rc = dev_alloc(ctx, ctx->post_ws, 2 * image);
        if (rc != CRG_OK) return rc;
        float *b[2] = {(float *)ctx->post_ws.ptr, (float *)((char *)ctx->post_ws.ptr + image)};
        k_bright<<<dim3((width + 255) / 256, height), 256, 0, st>>>(src, b[0], p, pitch);
        auto passes = [&](auto strip) {
            constexpr int N = decltype(strip)::value;
            const dim3 grid((width + kTileW - 1) / kTileW, (height + kStrips * N - 1) / (kStrips * N));
            for (int i = 0; i < 4; ++i)
                k_bloom<false, N><<<grid, kBloomThreads, 0, st>>>(b[i % 2], b[(i + 1) % 2], nullptr, nullptr, p, pitch, s, -0.0f);
            k_bloom<true, N><<<grid, kBloomThreads, 0, st>>>(b[0], nullptr, src, (float4 *)d_dst, p, pitch, s, -0.0f);
        };
        // tall strips read and blur least twice, short ones fill the GPU: with 16 / 4 rows 3840x2160 takes
        // 499 / 591 us, 1920x1080 (600 tall tiles) 159 / 169, 1280x720 (280) 105 / 96, 333x200 80 / 47
        const uint64_t tiles = (uint64_t)((width + kTileW - 1) / kTileW) * ((height + kStrips * 16 - 1) / (kStrips * 16));
        if (tiles >= 3ull * (uint64_t)std::max(ctx->sm_count, 1)) passes(std::integral_constant<int, 16>{});
        else passes(std::integral_constant<int, 4>{});
        CRG_CUDA(ctx, cudaGetLastError());
        return CRG_OK;
    }
    const unsigned blocks = (unsigned)std::min<size_t>((npix + 255) / 256, (size_t)std::max(ctx->sm_count, 1) * 8);
    k_post_final<<<blocks, 256, 0, st>>>(src, (float4 *)d_dst, p, s);
    CRG_CUDA(ctx, cudaGetLastError());
    return CRG_OK;
}
