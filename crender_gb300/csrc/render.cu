// render.cu — path-tracing megakernel (sm_103a).
//
// The drop-in for cr::renderer's sample passes (CRender
// src/render/renderer.cpp:116-144, 240-384): a lane (or one lane of each of a
// block's four warps) owns a pixel and draws its settings.spp samples, which are
// added to the pixel's FP32 sum (and optional FP64 sum / sum of squares) in
// sample order, so the film is bit-identical to a sequential CPU accumulation of
// the same samples.
//
// FAITHFUL follows process_hit / _sample_pixel (renderer.cpp:21-102,
// 258-384): Lambert = normalize(Ng + uniform sphere point), mirror metal,
// Fresnel-less glass, emission folded into the throughput, optional sun NEE
// with the reference's colour-squared weight.  EXTENDED adds emissive-
// triangle NEE with power-heuristic MIS, GGX (VNDF sampling), Fresnel
// dielectric and Russian roulette; Lambert still scatters into the geometric
// normal's hemisphere as the reference does.
//
// Random dimension groups: 0 = pixel jitter, 1 + 2i = BSDF at segment i,
// 2 + 2i = light sample at segment i (pcg4d keyed by pixel/sample/group/seed).
#include <cmath>

#include "render_common.cuh"

namespace crg {

CamDev camera_params(const crg_camera &c) {
    CamDev p;
    for (int a = 0; a < 3; ++a) p.pos[a] = c.position[a];
    const double k = 3.14159265358979323846 / 180.0;
    const double ax = c.rotation[0] * k, ay = c.rotation[1] * k, az = c.rotation[2] * k;
    const double Ry[3][3] = {{std::cos(ax), 0, std::sin(ax)}, {0, 1, 0}, {-std::sin(ax), 0, std::cos(ax)}};
    const double Rx[3][3] = {{1, 0, 0}, {0, std::cos(ay), -std::sin(ay)}, {0, std::sin(ay), std::cos(ay)}};
    const double Rz[3][3] = {{std::cos(az), -std::sin(az), 0}, {std::sin(az), std::cos(az), 0}, {0, 0, 1}};
    double T[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            T[i][j] = 0;
            for (int m = 0; m < 3; ++m) T[i][j] += Ry[i][m] * Rx[m][j];
        }
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            double r = 0;
            for (int m = 0; m < 3; ++m) r += T[i][m] * Rz[m][j];
            p.R[3 * i + j] = (float)r;
        }
    p.w = (float)(1.0 / std::tan(0.5 * (double)c.fov * k));
    p.mode = c.mode;
    p.scale = c.scale;
    return p;
}

using namespace rc;

namespace {

// MINB: blocks of 128 threads per SM, see render_form.
// PL: how the scene's placements are traced (warp_trace).
//
// A warp traces its lanes' segments together and then their shadow tests, sharing
// the triangle tests (warp_traverse).  Both go through one place in the code, the
// phase loop: the kernel is bound by instruction issue and fetch as much as by
// divergence, and two copies of the traversal do not fit the instruction cache.
// Lanes cover 8 x 4 pixel tiles (tile_pixel).  Against a traversal per thread on
// rows of pixels: box 512x512x64 15.6 -> 12.7 ms (19.6 instead of 11.3 lanes
// active), 4.2M-triangle mesh 1920x1080x4 15.5 -> 12.7, six placements with the
// reference estimator 1283x721 1.99 -> 1.23.
//
// SPLIT: a block's four warps render the same 32 pixels, a quarter of the samples
// each, in rounds of kRound samples whose radiances meet in shared memory and
// are added to the film in sample order; else a warp has its pixels to itself.
constexpr uint32_t kRound = 64;

// A warp with its pixels to itself is a block, whose place is free again as soon as
// the warp ends: box 1920x1080x8 7.36 -> 6.88 ms against blocks of four, mesh
// 1920x1080x1 3.23 -> 3.16.  Not with placements, where neighbouring warps do better
// close together (six placements 1283x721x1 1.24, 1.30 so).
template <int PL, bool SPLIT> constexpr uint32_t kRenderThreads = SPLIT || PL ? 128 : 32;

template <int W, int MODE, bool CNT, int MINB, int PL, bool SPLIT>
__global__ void __launch_bounds__((kRenderThreads<PL, SPLIT>), MINB * 128 / kRenderThreads<PL, SPLIT>)
k_render(SceneDev S, CamDev cam, crg_settings set, FilmDev F, uint64_t spp0, uint32_t pixels) {
    constexpr uint32_t T = kRenderThreads<PL, SPLIT>;
    constexpr bool kOwnBlock = T == 32u; // a warp with its pixels to itself, `pixels` of them
    __shared__ WarpRays s_rays[T / 32];
    // SPLIT: the round's radiances [sample][channel][pixel]; else, for films with FP64
    // planes, 6 sums per thread
    extern __shared__ double s_sums[];
    float *s_round = reinterpret_cast<float *>(s_sums);
    WarpRays &sh = s_rays[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, part = threadIdx.x >> 5;
    const uint32_t place = SPLIT ? blockIdx.x * 32u + lane : kOwnBlock ? blockIdx.x * pixels + lane : blockIdx.x * T + threadIdx.x;
    const uint32_t Wd = set.width, Hd = set.height;
    const bool inside = place < Wd * Hd && (!kOwnBlock || lane < pixels);
    const uint32_t pix = inside ? tile_pixel(place, Wd, Hd) : 0u;
    PathCtx C{pix, 0, set.seed, 0, 0, 0, 0ull, 0ull};
    const uint32_t px = pix % Wd, py = pix / Wd;
    const size_t fidx = (size_t)(Wd - 1 - px) + (size_t)(Hd - 1 - py) * Wd;
    float acc[3] = {0.0f, 0.0f, 0.0f};
    if (!SPLIT && inside) {
        for (int k = 0; k < 3; ++k) acc[k] = F.sum[fidx * 3 + k];
        if (F.sum64)
            for (int k = 0; k < 3; ++k) {
                s_sums[k * T + threadIdx.x] = F.sum64[fidx * 3 + k];
                s_sums[(3 + k) * T + threadIdx.x] = F.sumsq64[fidx * 3 + k];
            }
    }
    PathState ps;
    path_start(ps, mk(0, 0, 0), mk(0, 0, 1));
    for (uint32_t base = 0, count = 0; base < set.spp; base += count) {
        count = SPLIT ? min(kRound, set.spp - base) : set.spp;
        const uint32_t quarter = (count + 3u) / 4u;
        // Path regeneration (Novak, Havran and Dachsbacher 2010): one loop over
        // segments, in which a lane whose path has ended starts its pixel's next
        // sample, so a warp runs for the largest total segment count of its lanes
        // instead of the longest path of every sample.  A pixel's samples still
        // accumulate in order, so the film is unchanged.
        uint32_t s = base + (SPLIT ? min(count, part * quarter) : 0u), i = 0;
        const uint32_t end = inside ? (SPLIT ? base + min(count, (part + 1u) * quarter) : set.spp) : s;
        while (__any_sync(0xFFFFFFFFu, s < end)) {
            const bool alive = s < end;
            if (alive && i == 0) {
                C.sample = (uint32_t)(spp0 + s);
                const f4 g0 = rand4(pix, C.sample, 0, set.seed);
                const float x = ((float)px + g0.x) / (float)Wd;
                const float y = ((float)py + g0.y) / (float)Hd;
                v3 o, d;
                camera_ray(cam, x, y, set.aspect, o, d);
                path_start(ps, o, d);
            }
            const bool seg = alive && i < set.max_bounces;
            bool cont = false;
            Aov aov{mk(0, 0, 0), mk(0, 0, 0), 0.0f};
            NeeReq nr;
            nr.kind = 0;
#pragma unroll 1
            for (bool shadow = false;; shadow = true) {
                const bool on = shadow ? nr.kind != 0 : seg;
                if (shadow && !__any_sync(0xFFFFFFFFu, on)) break;
                Hit h;
                const v3 o = shadow ? nr.o : ps.o, d = shadow ? nr.d : ps.d;
                warp_trace<W, CNT, PL>(S, sh, on, shadow && MODE == CRG_MODE_EXTENDED, o, d, shadow ? nr.tmax : INFINITY, h, C);
                const bool found = h.prim != 0xFFFFFFFFu;
                if (!on) continue;
                if (!shadow) {
                    C.segments++;
                    cont = MODE == CRG_MODE_EXTENDED ? shade_extended(S, set, C, i, ps, found, h, aov, nr)
                                                     : shade_faithful(S, set, C, i, ps, found, h, aov, nr);
                    continue;
                }
                C.shadow++;
                nr.kind = 0;
                if (!found) {
                    ps.L = add(ps.L, nr.c);
                } else if (MODE == CRG_MODE_FAITHFUL) {
                    // the sun test steps 0.1 past alpha-zero surfaces (renderer.cpp:330-345)
                    const HitGeom hg = hit_geom<false>(S, h, o, d);
                    if (hit_colour(S, S.mats[hg.mat], h.prim, h.slot, hg.ro, hg.rd).w == 0.0f) {
                        nr.o = add(hg.p, mul(nr.d, 0.1f));
                        nr.kind = 2;
                    }
                }
            }
            if (!alive) continue;
            if (i == 0 && s + 1 == set.spp && F.aov_albedo) { // the last sample's first hit stays
                reinterpret_cast<float4 *>(F.aov_albedo)[fidx] = make_float4(aov.albedo.x, aov.albedo.y, aov.albedo.z, 1.0f);
                reinterpret_cast<float4 *>(F.aov_normal)[fidx] =
                    make_float4(aov.normal.x * 0.5f + 0.5f, aov.normal.y * 0.5f + 0.5f, aov.normal.z * 0.5f + 0.5f, 1.0f);
                const float dv = mn(aov.depth, 200.0f) / 200.0f;
                reinterpret_cast<float4 *>(F.aov_depth)[fidx] = make_float4(dv, dv, dv, 1.0f);
            }
            if (seg && cont && ++i < set.max_bounces) continue;
            const v3 L = ps.L;
            if (SPLIT) {
                float *q = s_round + (s - base) * 96u + lane;
                q[0] = L.x;
                q[32] = L.y;
                q[64] = L.z;
            }
            ++s;
            i = 0;
            if (SPLIT) continue;
            acc[0] += L.x;
            acc[1] += L.y;
            acc[2] += L.z;
            if (F.sum64) {
                double *q = s_sums + threadIdx.x;
                q[0] += (double)L.x; q[T] += (double)L.y; q[2 * T] += (double)L.z;
                q[3 * T] += (double)L.x * (double)L.x;
                q[4 * T] += (double)L.y * (double)L.y;
                q[5 * T] += (double)L.z * (double)L.z;
            }
        }
        if (SPLIT) {
            __syncthreads();
            if (inside && part < 3u) { // warp c adds channel c
                const size_t k = fidx * 3 + part;
                const float *q = s_round + part * 32u + lane;
                float sum = F.sum[k];
                for (uint32_t j = 0; j < count; ++j) sum += q[j * 96u];
                F.sum[k] = sum;
                if (F.sum64) {
                    double a64 = F.sum64[k], q64 = F.sumsq64[k];
                    for (uint32_t j = 0; j < count; ++j) {
                        const double v = (double)q[j * 96u];
                        a64 += v;
                        q64 += v * v;
                    }
                    F.sum64[k] = a64;
                    F.sumsq64[k] = q64;
                }
            }
            __syncthreads();
        }
    }
    if (!SPLIT && inside) {
        for (int k = 0; k < 3; ++k) F.sum[fidx * 3 + k] = acc[k];
        if (F.sum64)
            for (int k = 0; k < 3; ++k) {
                F.sum64[fidx * 3 + k] = s_sums[k * T + threadIdx.x];
                F.sumsq64[fidx * 3 + k] = s_sums[(3 + k) * T + threadIdx.x];
            }
    }
    if (C.err) atomicOr(S.err, C.err);
    if (CNT) {
        unsigned long long seg = C.segments, shr = C.shadow, nd = C.nodes, tr = C.tris;
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            seg += __shfl_xor_sync(0xFFFFFFFFu, seg, off);
            shr += __shfl_xor_sync(0xFFFFFFFFu, shr, off);
            nd += __shfl_xor_sync(0xFFFFFFFFu, nd, off);
            tr += __shfl_xor_sync(0xFFFFFFFFu, tr, off);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&S.counters[1], seg);
            atomicAdd(&S.counters[2], shr);
            atomicAdd(&S.counters[3], nd);
            atomicAdd(&S.counters[4], tr);
        }
    }
}

template <int W, int MINB, int PL, bool SPLIT, bool CNT = false>
void launch_m(const SceneDev &S, const CamDev &cam, const crg_settings &set, const FilmDev &F, uint64_t spp0, cudaStream_t st,
              uint32_t pixels = 32) {
    constexpr uint32_t T = kRenderThreads<PL, SPLIT>;
    const uint32_t per_block = SPLIT ? 32 : T == 32 ? pixels : T;
    const uint32_t blocks = (uint32_t)(((uint64_t)set.width * set.height + per_block - 1) / per_block);
    const size_t shared = SPLIT ? sizeof(float) * 96 * (set.spp < kRound ? set.spp : kRound) : F.sum64 ? sizeof(double) * 6 * T : 0;
    if (set.mode == CRG_MODE_EXTENDED)
        k_render<W, CRG_MODE_EXTENDED, CNT, MINB, PL, SPLIT><<<blocks, T, shared, st>>>(S, cam, set, F, spp0, pixels);
    else
        k_render<W, CRG_MODE_FAITHFUL, CNT, MINB, PL, SPLIT><<<blocks, T, shared, st>>>(S, cam, set, F, spp0, pixels);
}

template <int W>
void launch_w(const SceneDev &S, const CamDev &cam, const crg_settings &set, const FilmDev &F, uint64_t spp0, int sm_count,
              cudaStream_t st) {
    const uint64_t npix = (uint64_t)set.width * set.height;
    const RenderForm form = render_form(npix, set.spp, S.ntri, S.ninst != 0, (uint32_t)(sm_count > 0 ? sm_count : 1));
    const bool split = form.split;
    if (S.counters) { // the instrumented variants: one form per kind of scene
        if (S.ninst > kLoopPlacements) launch_m<W, 4, 2, false, true>(S, cam, set, F, spp0, st);
        else if (S.ninst) launch_m<W, 4, 1, false, true>(S, cam, set, F, spp0, st);
        else launch_m<W, 4, 0, false, true>(S, cam, set, F, spp0, st);
    } else if (S.ninst > kLoopPlacements) { // the top-level tree
        if (split) launch_m<W, 4, 2, true>(S, cam, set, F, spp0, st);
        else launch_m<W, 4, 2, false>(S, cam, set, F, spp0, st);
    } else if (S.ninst) {
        if (split) launch_m<W, 4, 1, true>(S, cam, set, F, spp0, st);
        else launch_m<W, 4, 1, false>(S, cam, set, F, spp0, st);
    } else if (form.blocks == 6u) {
        if (split) launch_m<W, 6, 0, true>(S, cam, set, F, spp0, st);
        else launch_m<W, 6, 0, false>(S, cam, set, F, spp0, st, form.pixels);
    } else {
        if (split) launch_m<W, 8, 0, true>(S, cam, set, F, spp0, st);
        else launch_m<W, 8, 0, false>(S, cam, set, F, spp0, st, form.pixels);
    }
}

} // namespace

namespace {
// Emitter records (see SceneDev::light_rec), built once per emitter table with
// the same device arithmetic the NEE sample would otherwise repeat per path.
__global__ void k_light_records(SceneDev S, float4 *__restrict__ rec) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= S.nlights) return;
    const uint32_t prim = S.light_prim[j];
    v3 a, b, c;
    prim_verts(S, prim, a, b, c);
    if (S.ninst) {
        const float4 *F = S.inst + 6 * (size_t)S.light_inst[j] + 3;
        a = xf_point(F, a);
        b = xf_point(F, b);
        c = xf_point(F, c);
    }
    const uint32_t mi = S.mat_idx[prim];
    const crg_material &m = S.mats[mi];
    float4 *r = rec + kLightVec * (size_t)j;
    r[0] = make_float4(a.x, a.y, a.z, S.light_pdf[j]);
    r[1] = make_float4(b.x, b.y, b.z, __uint_as_float(prim));
    r[2] = make_float4(c.x, c.y, c.z, __uint_as_float(mi));
    r[3] = make_float4(m.colour[0] * m.emission, m.colour[1] * m.emission, m.colour[2] * m.emission,
                       __uint_as_float(textured(S, m) ? 1u : 0u));
    const v3 n = normalize(cross(sub(b, a), sub(c, a)));
    r[4] = make_float4(n.x, n.y, n.z, 0.0f);
}

} // namespace

// Builds the emitter records of a scene's current emitter table (call after the
// table, the materials, the textures or the instances change).
crg_status build_light_records(crg_scene *s) {
    if (s->nlights == 0) return CRG_OK;
    crg_status rc = dev_alloc(s->ctx, s->light_rec, sizeof(float4) * kLightVec * (size_t)s->nlights);
    if (rc != CRG_OK) return rc;
    const SceneDev S = scene_dev(s);
    k_light_records<<<(s->nlights + 127) / 128, 128>>>(S, (float4 *)s->light_rec.ptr);
    CRG_CUDA(s->ctx, cudaGetLastError());
    CRG_CUDA(s->ctx, cudaDeviceSynchronize());
    return CRG_OK;
}

namespace rc {
SceneDev scene_dev(const crg_scene *s) {
    SceneDev S{};
    S.nodes = (const uint4 *)s->wide.ptr;
    S.tris = (const float4 *)s->tris.ptr;
    S.slot_nm = (const float4 *)s->slot_nm.ptr;
    S.mat_idx = (const uint32_t *)s->mat_idx.ptr;
    S.mats = (const crg_material *)s->mats.ptr;
    S.light_prim = (const uint32_t *)s->light_prim.ptr;
    S.light_alias = (const float2 *)s->light_alias.ptr;
    S.light_pdf = (const float *)s->light_pdf.ptr;
    S.mat_light_pdf = (const float *)s->mat_light_pdf.ptr;
    S.verts = (const float *)s->verts.ptr;
    S.uvs = (const float *)s->uvs.ptr;
    S.texels = (const float4 *)s->texels.ptr;
    S.tex_info = (const uint4 *)s->tex_info.ptr;
    S.ntex = s->texels.ptr ? s->ntex : 0;
    S.inst = (const float4 *)s->inst.ptr;
    S.inst_root = (const uint32_t *)s->inst_root.ptr;
    S.tlas = (const float4 *)s->tlas.ptr;
    S.tlas_root = s->tlas_root;
    S.light_inst = (const uint32_t *)s->light_inst.ptr;
    S.light_rec = (const float4 *)s->light_rec.ptr;
    S.ninst = s->inst.ptr ? s->ninst : 0;
    S.nlights = s->nlights;
    S.ntri = s->ntri;
    S.sky = (const float4 *)s->sky.ptr;
    S.sky_w = s->sky.ptr ? s->sky_w : 0;
    S.sky_h = s->sky_h;
    S.sky_rot_u = s->sky_rot_u;
    S.sky_rot_v = s->sky_rot_v;
    S.sun_on = s->sun_enabled;
    for (int k = 0; k < 9; ++k) S.sun_frame[k] = s->sun_frame[k];
    S.sun_cos = s->sun_cos;
    S.sun_pdf = s->sun_pdf;
    for (int k = 0; k < 3; ++k) {
        S.sun_neg_dir[k] = -s->sun.direction[k];
        S.sun_rad[k] = s->sun.colour[k] * s->sun.intensity;
    }
    S.err = (uint32_t *)s->err.ptr;
    S.counters = s->counting ? (unsigned long long *)s->counters.ptr : nullptr;
    return S;
}
} // namespace rc

crg_status launch_render(crg_scene *s, const CamDev &cam, const crg_settings &set, crg_film *film, cudaStream_t st) {
    const SceneDev S = scene_dev(s);
    FilmDev F{(float *)film->sum.ptr,
              (double *)film->sum64.ptr,
              (double *)film->sumsq64.ptr,
              (float *)film->aov_albedo.ptr,
              (float *)film->aov_normal.ptr,
              (float *)film->aov_depth.ptr,
              film->width,
              film->height};
    if (s->ntri == 0) return set_error(s->ctx, CRG_ERR_INVALID_ARG, "crg_render: scene has no triangles");
    switch (s->width) {
    case 2: launch_w<2>(S, cam, set, F, film->spp, s->ctx->sm_count, st); break;
    case 4: launch_w<4>(S, cam, set, F, film->spp, s->ctx->sm_count, st); break;
    default: launch_w<8>(S, cam, set, F, film->spp, s->ctx->sm_count, st); break;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(s->ctx, e, "k_render launch");
    return CRG_OK;
}

} // namespace crg
