// traverse.cu — batched closest-hit / any-hit queries (the rtcIntersect1 /
// rtcOccluded1 replacements, CRender src/objects/model.cpp:5-49).
//
// One ray per lane; rays are two 16-byte loads, hits one 16-byte store.  The
// wide nodes are read with 16-byte vector loads through the read-only path;
// per-lane group stack of 64 entries (overflow raises the scene's error word
// instead of trapping).
#include <algorithm>

#include "render_common.cuh"

namespace crg {
namespace {

// Queries on an instanced scene: model::intersect's loop over the instances
// (model.cpp:99-126) through the shared closest / any-hit functions.  The
// ray's tmin applies in each instance's object space (the reference's tnear);
// t is the world distance of the hit point.
template <int W, bool ANY>
__global__ void __launch_bounds__(128) k_intersect_inst(rc::SceneDev S, const float4 *__restrict__ rays,
                                                       float4 *__restrict__ hits, uint32_t *__restrict__ occluded,
                                                       uint64_t n) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 r0 = __ldg(&rays[2 * i]);
    const float4 r1 = __ldg(&rays[2 * i + 1]);
    const v3 o = mk(r0.x, r0.y, r0.z), d = mk(r1.x, r1.y, r1.z);
    rc::PathCtx C{0, 0, 0, 0, 0, 0, 0ull, 0ull};
    if (ANY) {
        occluded[i] = rc::occluded_t<W, false, true>(S, o, d, r0.w, r1.w, C) ? 1u : 0u;
    } else {
        rc::Hit h;
        if (rc::closest_t<W, false, true>(S, o, d, r0.w, r1.w, h, C)) {
            v3 oo, od;
            float len;
            rc::inst_ray(S, h.inst, o, d, oo, od, len);
            const float t = rc::vdist(rc::inst_point(S, h.inst, oo, od, h.t), o);
            hits[i] = make_float4(t, __uint_as_float(h.prim), h.u, h.v);
        } else {
            hits[i] = make_float4(INFINITY, __uint_as_float(0xFFFFFFFFu), 0.0f, 0.0f);
        }
    }
    if (C.err) atomicOr(S.err, C.err);
}

// Lanes without pending triangles below which a warp turns to the triangle
// tests: 16 / 20 / 24 measured 12.15 / 11.91 / 12.22 ms on the soup's 16.8M
// closest hits, 1.76 / 1.76 / 1.79 ms on 5.0M any hits.
constexpr uint32_t kVisitors = 20;

// One ray per lane, triangle tests shared by the warp, lanes refilled from the
// block's run of `chunk` rays (dyn_traverse).  The run's counter lies in the
// block's shared memory, so calls on several streams share nothing.  Bound by
// instruction issue (71% of cycles, the ALU pipe 70%) on incoherent rays; 8 blocks of 128 per SM
// (64 registers).  1M-triangle soup, width 8: 16.8M closest hits 20.97 -> 11.91
// ms against one thread per ray with its own triangle tests (9.1 lanes active),
// 5.0M any hits 2.73 -> 1.76 ms against per-lane refill without shared tests.
// 9 and 10 blocks per SM (spills) were 2-3% slower.
template <int W, bool ANY, bool COUNT>
__global__ void __launch_bounds__(128, 8) k_intersect(const uint4 *__restrict__ nodes, const float4 *__restrict__ tris,
                                                   const float4 *__restrict__ rays, float4 *__restrict__ hits,
                                                   uint32_t *__restrict__ occluded, uint32_t *__restrict__ ncount,
                                                   uint32_t *__restrict__ tcount, uint64_t n, uint32_t chunk,
                                                   uint32_t refill, uint32_t ntri, uint32_t *__restrict__ err) {
    __shared__ WarpRays s_rays[4];
    __shared__ unsigned int s_head;
    if (threadIdx.x == 0) s_head = 0u;
    __syncthreads();
    WarpRays &sh = s_rays[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t first = (uint64_t)blockIdx.x * chunk;
    const uint32_t count = (uint32_t)(n - first < chunk ? n - first : chunk);
    TravStats st{0, 0};
    uint32_t e = 0;
    auto put = [&](uint32_t i, float t, uint32_t prim, float u, float v) {
        hits[first + i] = make_float4(t, __uint_as_float(prim), u, v);
    };
    auto put_counts = [&](uint32_t i) {
        if (ncount) ncount[first + i] = st.nodes;
        if (tcount) tcount[first + i] = st.tris;
    };
    dyn_traverse<W, ANY, COUNT, kVisitors>(
        sh, [&](uint32_t cnt) { return atomicAdd(&s_head, cnt); }, count, refill,
        [&](unsigned int i, uint32_t &payload, RayPre &r, float &tmax, uint32_t &, const uint4 *&nd, const float4 *&tr) {
            if (COUNT) st = TravStats{0, 0};
            if (ntri == 0) {
                if (ANY) occluded[first + i] = 0u;
                else put(i, INFINITY, 0xFFFFFFFFu, 0.0f, 0.0f);
                if (COUNT) put_counts(i);
                return false;
            }
            payload = i;
            const float4 r0 = __ldg(&rays[2 * (first + i)]);
            const float4 r1 = __ldg(&rays[2 * (first + i) + 1]);
            r = ray_prep(r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r0.w);
            tmax = r1.w;
            nd = nodes;
            tr = tris;
            return true;
        },
        [](uint32_t, const LaneTrav &, RayPre &, float &, uint32_t &) { return false; },
        [&](uint32_t i, const LaneTrav &T) {
            if (ANY) {
                occluded[first + i] = T.occluded ? 1u : 0u;
            } else if (T.best_prim == 0xFFFFFFFFu) {
                put(i, INFINITY, 0xFFFFFFFFu, 0.0f, 0.0f);
            } else {
                float u, v;
                stored_uv(sh, lane, T.best_slot, tris, u, v);
                put(i, T.best_t, T.best_prim, u, v);
            }
            if (COUNT) put_counts(i);
        },
        st, e);
    if (e) atomicOr(err, e);
}

// Warp-cooperative traversal: G = W lanes per ray, 32 / W rays per warp.  A
// ray's node is read with 16-byte vector loads by its lanes into shared
// memory, each lane tests one child box against the ray, and the hit bits are
// OR-reduced over the lanes; its pending triangles are tested G at a time (one
// per lane, 16-byte loads) and the lexicographic minimum (t, primitive) of
// the lanes' hits is reduced by shuffles, so the closest hit equals the
// per-thread traversal's (accept_hit's order, conservative culling).  Each
// ray keeps its group stack in the warp's shared memory; an idle group takes
// the next ray index with one atomic per warp for all idle groups (head), or
// each group has one ray (no head).
template <int W>
struct WarpShared {
    static constexpr int R = 32 / W;
    uint4 node[4][R][NodeLayout<W>::VEC];
    uint2 stack[4][R][kStack];
};

// One iteration for the group in `gmask` (c = lane in group): the pending
// triangles, then one node.  Returns true when the ray is finished.
template <int W, bool ANY>
__device__ __forceinline__ bool warp_step(Trav &T, uint2 *stack, uint4 *nbuf, const uint4 *__restrict__ nodes,
                                          const float4 *__restrict__ tris, const RayPre &r, uint32_t gmask, uint32_t c,
                                          uint32_t &err) {
    using L = NodeLayout<W>;
    constexpr int G = W;
    while (T.tg.y != 0u) {
        const uint32_t pend = T.tg.y;
        uint32_t rest = pend, mine = 0u; // this lane's triangle: the (c+1)-th pending bit; the first G are taken now
#pragma unroll
        for (uint32_t k = 0; k < (uint32_t)G; ++k) {
            if (k == c) mine = rest;
            rest &= rest - 1u;
        }
        T.tg.y = rest;
        bool hit = false;
        float ct = INFINITY;
        uint32_t cp = 0xFFFFFFFFu, slot = 0u;
        TriHit h{0.0f, 0.0f, 0.0f, 1.0f};
        if (mine) {
            slot = T.tg.x + (uint32_t)(__ffs(mine) - 1);
            const float4 a = __ldg(&tris[slot * 3 + 0]);
            const float4 b = __ldg(&tris[slot * 3 + 1]);
            const float4 cc = __ldg(&tris[slot * 3 + 2]);
            hit = watertight(r, a, b, cc, h);
            if (ANY) {
                hit = hit && h.t > r.tmin && h.t < T.tmax;
            } else if (hit && h.t > r.tmin) {
                ct = h.t;
                cp = __float_as_uint(a.w);
            }
        }
        if (ANY) {
            if (__ballot_sync(gmask, hit) != 0u) {
                T.occluded = true;
                return true;
            }
            continue;
        }
        float mt = ct;
        uint32_t mp = cp;
#pragma unroll
        for (int off = G / 2; off >= 1; off >>= 1) {
            const float ot = __shfl_xor_sync(gmask, mt, off, G);
            const uint32_t op = __shfl_xor_sync(gmask, mp, off, G);
            if (ot < mt || (ot == mt && op < mp)) {
                mt = ot;
                mp = op;
            }
        }
        if (mp != 0xFFFFFFFFu && accept_hit(mt, mp, r.tmin, T.best_t, T.best_prim)) {
            const uint32_t win = (uint32_t)__ffs(__ballot_sync(gmask, cp == mp && ct == mt)) - 1u;
            T.best_t = mt;
            T.best_prim = mp;
            T.best_slot = __shfl_sync(gmask, slot, win);
            T.best_V = __shfl_sync(gmask, h.V, win);
            T.best_W = __shfl_sync(gmask, h.W, win);
            T.best_det = __shfl_sync(gmask, h.det, win);
        }
    }
    if ((T.ng.y >> 24) == 0u) {
        if (T.sp == 0) return true;
        T.ng = stack[--T.sp];
    }
    const uint32_t hb = T.ng.y >> 24;
    const uint32_t pos = 31u - __clz(hb);
    const uint32_t code = pos ^ T.oct;
    T.ng.y &= ~(1u << (24 + pos));
    const uint32_t child = T.ng.x + __popc(T.ng.y & ((1u << code) - 1u) & 0xFFu);
    if ((T.ng.y >> 24) != 0u) {
        if (T.sp < kStack) {
            if (c == 0u) stack[T.sp] = T.ng;
            T.sp++;
        } else {
            err = 1u;
        }
    }
    const uint4 *np = nodes + (size_t)child * L::VEC;
    for (int k = (int)c; k < L::VEC; k += G) nbuf[k] = __ldg(np + k);
    __syncwarp(gmask);
    const uint4 h0 = nbuf[0];
    const uint2 h1 = *reinterpret_cast<const uint2 *>(&nbuf[1]);
    const uint8_t *nb = reinterpret_cast<const uint8_t *>(nbuf);
    const uint32_t meta = nb[24 + c];
    const float qlx = (float)nb[24 + W + c], qly = (float)nb[24 + 2 * W + c], qlz = (float)nb[24 + 3 * W + c];
    const float qhx = (float)nb[24 + 4 * W + c], qhy = (float)nb[24 + 5 * W + c], qhz = (float)nb[24 + 6 * W + c];
    const uint32_t eb = h0.w;
    const float sx = __uint_as_float((eb & 0xFFu) << 23) * r.ix;
    const float sy = __uint_as_float(((eb >> 8) & 0xFFu) << 23) * r.iy;
    const float sz = __uint_as_float(((eb >> 16) & 0xFFu) << 23) * r.iz;
    const float ox = (__uint_as_float(h0.x) - r.ox) * r.ix;
    const float oy = (__uint_as_float(h0.y) - r.oy) * r.iy;
    const float oz = (__uint_as_float(h0.z) - r.oz) * r.iz;
    const float tx0 = __fmaf_rn(r.ix >= 0.0f ? qlx : qhx, sx, ox);
    const float tx1 = __fmaf_rn(r.ix >= 0.0f ? qhx : qlx, sx, ox);
    const float ty0 = __fmaf_rn(r.iy >= 0.0f ? qly : qhy, sy, oy);
    const float ty1 = __fmaf_rn(r.iy >= 0.0f ? qhy : qly, sy, oy);
    const float tz0 = __fmaf_rn(r.iz >= 0.0f ? qlz : qhz, sz, oz);
    const float tz1 = __fmaf_rn(r.iz >= 0.0f ? qhz : qlz, sz, oz);
    const float tn = fmaxf(fmaxf(tx0, ty0), fmaxf(tz0, r.tmin));
    const float tf = fminf(fminf(tx1, ty1), fminf(tz1, T.best_t * kHitSlack));
    const uint32_t mine = tn <= tf * 1.00000095f ? (meta >> 5) << (meta & 31u) : 0u;
    const uint32_t bits = __reduce_or_sync(gmask, mine);
    uint32_t m = bits >> 24;
    if (T.oct & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (T.oct & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (T.oct & 4u) m = ((m & 0x0Fu) << 4) | ((m >> 4) & 0x0Fu);
    T.ng = make_uint2(h1.x, (m << 24) | (eb >> 24));
    T.tg = make_uint2(h1.y, bits & 0x00FFFFFFu);
    __syncwarp(gmask); // every lane has read the node before the group's next one overwrites it
    return false;
}

template <int W, bool ANY>
__global__ void __launch_bounds__(128) k_intersect_warp(const uint4 *__restrict__ nodes, const float4 *__restrict__ tris,
                                                      const float4 *__restrict__ rays, float4 *__restrict__ hits,
                                                      uint32_t *__restrict__ occluded, unsigned int *head, uint32_t n,
                                                      uint32_t per_warp, uint32_t *__restrict__ err) {
    constexpr int G = W;
    __shared__ WarpShared<W> sh;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint32_t g = lane / G, c = lane % G;
    const uint32_t gmask = ((1u << G) - 1u) << (g * G);
    uint4 *nbuf = sh.node[wib][g];
    uint2 *stack = sh.stack[wib][g];
    bool has = false, exhausted = false;
    uint32_t ray = 0, e = 0;
    RayPre r;
    Trav T;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, c == 0u && !has); // one bit per idle group
        if (!exhausted && idle != 0u) {
            const uint32_t cnt = (uint32_t)__popc(idle);
            unsigned int base = 0;
            if (head) {
                if (lane == 0) base = atomicAdd(head, cnt);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                if (base + cnt >= n) exhausted = true;
            } else { // the warp's own rays, one for each of its first `per_warp` groups
                base = g < per_warp ? (blockIdx.x * 4u + wib) * per_warp : n;
                exhausted = true;
            }
            if (!has) {
                const unsigned int my = base + (unsigned int)__popc(idle & ((1u << (g * G)) - 1u));
                if (my < n) {
                    const float4 r0 = __ldg(&rays[2 * (size_t)my]);
                    const float4 r1 = __ldg(&rays[2 * (size_t)my + 1]);
                    r = ray_prep(r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r0.w);
                    trav_init(T, r, r1.w);
                    ray = my;
                    has = true;
                }
            }
        }
        if (!__any_sync(0xFFFFFFFFu, has)) {
            if (exhausted) break;
            continue;
        }
        if (has) {
            bool done = false;
            for (int it = 0; it < 4 && !done; ++it) done = warp_step<W, ANY>(T, stack, nbuf, nodes, tris, r, gmask, c, e);
            if (done) {
                if (c == 0u) {
                    if (ANY) occluded[ray] = T.occluded ? 1u : 0u;
                    else if (T.best_prim == 0xFFFFFFFFu)
                        hits[ray] = make_float4(INFINITY, __uint_as_float(0xFFFFFFFFu), 0.0f, 0.0f);
                    else
                        hits[ray] = make_float4(T.best_t, __uint_as_float(T.best_prim), T.best_V / T.best_det,
                                                T.best_W / T.best_det);
                }
                has = false;
            }
        }
    }
    if (e) atomicOr(err, e);
}

// Idle lanes that make a warp refill: 4 / 8 / 12 measured 15.13 / 15.04 / 15.43
// ms on the soup's 16.8M closest hits, 2.12 / 2.10 / 2.15 ms on 5.0M any hits.
constexpr uint32_t kRefill = 8;
// Rays of a block at most: 1024 / 2048 / 8192 measured 14.97 / 15.04 / 15.91 ms
// (closest) and 2.28 / 2.10 / 2.12 ms (any).
constexpr uint32_t kChunkMax = 2048;

template <int W>
void launch_warp(const crg_scene *s, const crg_ray *rays, crg_hit *hits, uint32_t *occluded, uint64_t n, bool any,
                 cudaStream_t st) {
    int per_sm = 0;
    if (any) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_intersect_warp<W, true>, 128, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_intersect_warp<W, false>, 128, 0);
    const uint32_t grid = (uint32_t)(std::max(s->ctx->sm_count, 1) * std::max(per_sm, 1));
    unsigned int *head = (unsigned int *)s->qhead.ptr;
    cudaMemsetAsync(head, 0, sizeof(unsigned int), st);
    const uint4 *nd = (const uint4 *)s->wide.ptr;
    const float4 *tr = (const float4 *)s->tris.ptr;
    if (any)
        k_intersect_warp<W, true><<<grid, 128, 0, st>>>(nd, tr, (const float4 *)rays, nullptr, occluded, head, (uint32_t)n,
                                                       0u, (uint32_t *)s->err.ptr);
    else
        k_intersect_warp<W, false><<<grid, 128, 0, st>>>(nd, tr, (const float4 *)rays, (float4 *)hits, nullptr, head,
                                                        (uint32_t)n, 0u, (uint32_t *)s->err.ptr);
}

// One call of few rays (few_rays_per_warp): every warp has its own.
template <int W>
void launch_few(const crg_scene *s, const crg_ray *rays, crg_hit *hits, uint32_t *occluded, uint64_t n, uint32_t per_warp, bool any,
                cudaStream_t st) {
    const uint32_t grid = (uint32_t)((n + 4 * per_warp - 1) / (4 * per_warp));
    const uint4 *nd = (const uint4 *)s->wide.ptr;
    const float4 *tr = (const float4 *)s->tris.ptr;
    uint32_t *err = (uint32_t *)s->err.ptr;
    if (any)
        k_intersect_warp<W, true><<<grid, 128, 0, st>>>(nd, tr, (const float4 *)rays, nullptr, occluded, nullptr, (uint32_t)n,
                                                       per_warp, err);
    else
        k_intersect_warp<W, false><<<grid, 128, 0, st>>>(nd, tr, (const float4 *)rays, (float4 *)hits, nullptr, nullptr,
                                                        (uint32_t)n, per_warp, err);
}

template <int W>
void launch_w(const crg_scene *s, const crg_ray *rays, crg_hit *hits, uint32_t *occluded, uint32_t *nodes, uint32_t *tris,
              uint64_t n, bool any, bool lanes, cudaStream_t st) {
    if (s->ninst && s->ntri > 0) {
        const rc::SceneDev S = rc::scene_dev(s);
        const uint64_t blocks = (n + 127) / 128;
        if (any) k_intersect_inst<W, true><<<blocks, 128, 0, st>>>(S, (const float4 *)rays, nullptr, occluded, n);
        else k_intersect_inst<W, false><<<blocks, 128, 0, st>>>(S, (const float4 *)rays, (float4 *)hits, nullptr, n);
        if (nodes) cudaMemsetAsync(nodes, 0, 4 * n, st);
        if (tris) cudaMemsetAsync(tris, 0, 4 * n, st);
        return;
    }
    if (const uint32_t per_warp = few_rays_per_warp(n, W, s->ntri, lanes || nodes || tris)) {
        launch_few<W>(s, rays, hits, occluded, n, per_warp, any, st);
        return;
    }
    // a block's run of rays: long enough that its warps mostly run full, short
    // enough that every SM gets several blocks one after the other
    const uint64_t resident = (uint64_t)std::max(s->ctx->sm_count, 1) * 8;
    const uint64_t share = (n / (resident * 6) + 127) / 128 * 128;
    const uint32_t chunk = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(share, 128), kChunkMax);
    const uint64_t blocks = (n + chunk - 1) / chunk;
    const uint4 *nd = (const uint4 *)s->wide.ptr;
    const float4 *tr = (const float4 *)s->tris.ptr;
    uint32_t *err = (uint32_t *)s->err.ptr;
    if (any)
        k_intersect<W, true, false><<<blocks, 128, 0, st>>>(nd, tr, (const float4 *)rays, nullptr, occluded, nullptr, nullptr,
                                                           n, chunk, kRefill, s->ntri, err);
    else if (nodes || tris)
        k_intersect<W, false, true><<<blocks, 128, 0, st>>>(nd, tr, (const float4 *)rays, (float4 *)hits, nullptr, nodes, tris,
                                                           n, chunk, kRefill, s->ntri, err);
    else
        k_intersect<W, false, false><<<blocks, 128, 0, st>>>(nd, tr, (const float4 *)rays, (float4 *)hits, nullptr, nullptr,
                                                            nullptr, n, chunk, kRefill, s->ntri, err);
}

} // namespace

crg_status launch_intersect(const crg_scene *s, const crg_ray *rays, crg_hit *hits, uint32_t *occluded, uint32_t *nodes,
                            uint32_t *tris, uint64_t n, bool any, cudaStream_t st, int traversal) {
    if (n == 0) return CRG_OK;
    if (traversal == CRG_TRAVERSAL_WARP && s->ninst == 0 && s->ntri > 0 && !nodes && !tris) {
        if (n >= 0xFFFF0000ull) return set_error(s->ctx, CRG_ERR_INVALID_ARG, "warp traversal: at most 2^32 - 2^16 rays per call");
        switch (s->width) {
        case 2: launch_warp<2>(s, rays, hits, occluded, n, any, st); break;
        case 4: launch_warp<4>(s, rays, hits, occluded, n, any, st); break;
        default: launch_warp<8>(s, rays, hits, occluded, n, any, st); break;
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_error(s->ctx, e, "k_intersect_warp launch");
        return CRG_OK;
    }
    const bool lanes = traversal == CRG_TRAVERSAL_THREAD;
    switch (s->width) {
    case 2: launch_w<2>(s, rays, hits, occluded, nodes, tris, n, any, lanes, st); break;
    case 4: launch_w<4>(s, rays, hits, occluded, nodes, tris, n, any, lanes, st); break;
    default: launch_w<8>(s, rays, hits, occluded, nodes, tris, n, any, lanes, st); break;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(s->ctx, e, "k_intersect launch");
    return CRG_OK;
}

} // namespace crg
