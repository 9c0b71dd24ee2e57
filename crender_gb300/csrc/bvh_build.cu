// bvh_build.cu — GPU LBVH builder and wide-BVH collapse (sm_103a).
//
// Replaces rtcCommitScene (CRender src/objects/model.cpp:52-97).  Pipeline:
//   k_bounds        triangle boxes + centroid bounds (order-preserving int atomics)
//   k_morton        30-bit Morton codes of AABB centres
//   radix sort      stable LSD, 8-bit digits, 4 passes: hist / scan_rows / scatter
//                   (warp match_any ranking keeps equal digits in input order,
//                   so the result is the unique (code, index) order)
//   k_gather        the sorted order and the triangle boxes in it
//   k_karras        Karras 2012 hierarchy, one thread per internal node
//   k_bottom_up     boxes, primitive counts and SAH costs (Ci = 1.2, Ct = 1), second arrival computes
//   k_treelet       optional Karras & Aila 2013 treelet restructuring
//   k_level_*       level-by-level greedy collapse to a W-wide BVH
//   k_emit          its quantized nodes and triangle slots
// Every float decision is evaluated in the same order as the CPU form, so the
// binary tree, the wide nodes and the triangle array are bit-identical to a
// CPU run of the same algorithm.
#include <cfloat>
#include <cmath>
#include <mutex>

#include "crg_dev.cuh"
#include "crg_internal.h"

namespace crg {
namespace {

constexpr uint32_t LEAF = 0x80000000u;
constexpr uint32_t NONE = 0xFFFFFFFFu;

__device__ __forceinline__ float fmn(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float fmx(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ uint32_t f2key(float f) {
    const uint32_t i = __float_as_uint(f);
    return (i & 0x80000000u) ? ~i : (i | 0x80000000u);
}
__device__ __forceinline__ float key2f(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
__device__ __forceinline__ float area3(float dx, float dy, float dz) { return 2.0f * ((dx * dy + dy * dz) + dz * dx); }

struct Box {
    float lo[3], hi[3];
};
__device__ __forceinline__ Box merge(const Box &a, const Box &b) {
    Box r;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r.lo[k] = fmn(a.lo[k], b.lo[k]);
        r.hi[k] = fmx(a.hi[k], b.hi[k]);
    }
    return r;
}
__device__ __forceinline__ float area(const Box &b) {
    return area3(b.hi[0] - b.lo[0], b.hi[1] - b.lo[1], b.hi[2] - b.lo[2]);
}

// ----------------------------------------------------------------- bounds
__global__ void k_bounds(const float *__restrict__ v, uint32_t n, float4 *__restrict__ tbox, uint32_t *__restrict__ cb) {
    float mn3[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx3[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float *p = v + (size_t)i * 9;
        float lo[3], hi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float x0 = p[a], x1 = p[3 + a], x2 = p[6 + a];
            lo[a] = fmn(fmn(x0, x1), x2);
            hi[a] = fmx(fmx(x0, x1), x2);
            const float c = (lo[a] + hi[a]) * 0.5f;
            mn3[a] = fminf(mn3[a], c);
            mx3[a] = fmaxf(mx3[a], c);
        }
        tbox[2 * (size_t)i] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        tbox[2 * (size_t)i + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            mn3[a] = fminf(mn3[a], __shfl_xor_sync(0xFFFFFFFFu, mn3[a], off));
            mx3[a] = fmaxf(mx3[a], __shfl_xor_sync(0xFFFFFFFFu, mx3[a], off));
        }
    // a block's six bounds by one atomic each: atomics on one address run one after another
    // (4.2M triangles: 190 us with six a warp, 46 so)
    __shared__ uint32_t s_key[6][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    if (lane == 0u) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            s_key[a][warp] = f2key(mn3[a]);
            s_key[3 + a][warp] = f2key(mx3[a]);
        }
    }
    __syncthreads();
    if (threadIdx.x < 6u) {
        uint32_t key = s_key[threadIdx.x][0];
        for (uint32_t w = 1; w < warps; ++w) key = threadIdx.x < 3u ? min(key, s_key[threadIdx.x][w]) : max(key, s_key[threadIdx.x][w]);
        if (threadIdx.x < 3u) atomicMin(&cb[threadIdx.x], key);
        else atomicMax(&cb[threadIdx.x], key);
    }
}

// Standard 10-bit interleave (Karras, "Thinking Parallel III", 2012).
__device__ __forceinline__ uint32_t expand10(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__global__ void k_morton(const float4 *__restrict__ tbox, uint32_t n, const uint32_t *__restrict__ cb,
                         uint32_t *__restrict__ keys, uint32_t *__restrict__ vals) {
    float clo[3], scale[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        clo[a] = key2f(cb[a]);
        const float ext = key2f(cb[3 + a]) - clo[a];
        scale[a] = ext > 0.0f ? 1024.0f / ext : 0.0f;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 lo = tbox[2 * (size_t)i], hi = tbox[2 * (size_t)i + 1];
        const float c[3] = {(lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f};
        uint32_t q[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) q[a] = (uint32_t)fmn(fmx((c[a] - clo[a]) * scale[a], 0.0f), 1023.0f);
        keys[i] = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
        vals[i] = i;
    }
}

// ----------------------------------------------------------------- radix sort
// ROWS: keys of a thread; a block sorts 256 ROWS, its warps 32 ROWS consecutive ones
// each.  Sixteen keep the counts short; two spread a small array over the GPU
// (a pass over 10,007 keys is the time of one block: 14 us of scatter at 16).
constexpr int kSortThreads = 256;
constexpr uint32_t kSmallSort = 1u << 17; // keys up to which ROWS is 2
constexpr uint32_t sort_blocks(uint32_t n) { return n <= kSmallSort ? (n + 511u) / 512u : (n + 4095u) / 4096u; }

template <int ROWS>
__global__ void __launch_bounds__(kSortThreads) k_hist(const uint32_t *__restrict__ keys, uint32_t n, int shift,
                                                       uint32_t *__restrict__ hist) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * (kSortThreads * ROWS);
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        const uint32_t i = base + k * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// Exclusive prefix of x over the block's 256 threads; *total receives the sum.
__device__ __forceinline__ uint32_t block_prefix(uint32_t x, uint32_t *warp_sums, uint32_t *total) {
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    uint32_t incl = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if ((int)lane >= off) incl += o;
    }
    if (lane == 31u) warp_sums[wib] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t t = warp_sums[k];
        before += k < wib ? t : 0u;
        all += t;
    }
    __syncthreads();
    *total = all;
    return before + incl - x;
}

// Exclusive scan of each digit's row of per-block counts in place, a block per
// digit; the scatter adds the sums of the smaller digits.  (One block over all
// 256 rows took 140 us a pass at 4.2M keys.)
__global__ void __launch_bounds__(256) k_scan_rows(uint32_t *__restrict__ hist, uint32_t nblk, uint32_t *__restrict__ digit_sum) {
    __shared__ uint32_t sums[8];
    uint32_t *row = hist + (size_t)blockIdx.x * nblk;
    uint32_t run = 0;
    for (uint32_t base = 0; base < nblk; base += 1024u) {
        uint32_t v[4], own = 0;
        const uint32_t i = base + threadIdx.x * 4u;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            v[k] = i + k < nblk ? row[i + k] : 0u;
            own += v[k];
        }
        uint32_t total;
        uint32_t at = run + block_prefix(own, sums, &total);
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            if (i + k < nblk) row[i + k] = at;
            at += v[k];
        }
        run += total;
    }
    if (threadIdx.x == 0) digit_sum[blockIdx.x] = run;
}

template <int ROWS>
__global__ void __launch_bounds__(kSortThreads) k_scatter(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin,
                                                          uint32_t n, int shift, const uint32_t *__restrict__ hist,
                                                          const uint32_t *__restrict__ digit_sum,
                                                          uint32_t *__restrict__ kout, uint32_t *__restrict__ vout) {
    __shared__ uint32_t wcnt[8][256];
    __shared__ uint32_t goff[256];
    __shared__ uint32_t sums[8];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int k = 0; k < 8; ++k) wcnt[k][tid] = 0;
    {
        uint32_t total;
        const uint32_t before = block_prefix(digit_sum[tid], sums, &total);
        goff[tid] = before + hist[tid * gridDim.x + blockIdx.x];
    }
    __syncthreads();
    const uint32_t base = blockIdx.x * (kSortThreads * ROWS) + w * (32 * ROWS);
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t kk[ROWS], vv[ROWS], rk[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const uint32_t i = base + r * 32 + lane;
        const bool valid = i < n;
        const uint32_t key = valid ? kin[i] : 0u;
        const uint32_t val = valid ? vin[i] : 0u;
        const uint32_t d = (key >> shift) & 255u;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, valid ? d : 256u + lane);
        const uint32_t before = valid ? wcnt[w][d] : 0u;
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wcnt[w][d] += __popc(peers);
        __syncwarp();
        kk[r] = key;
        vv[r] = val;
        rk[r] = before + __popc(peers & lt);
    }
    __syncthreads();
    {
        uint32_t run = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t c = wcnt[k][tid];
            wcnt[k][tid] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const uint32_t i = base + r * 32 + lane;
        if (i < n) {
            const uint32_t d = (kk[r] >> shift) & 255u;
            const uint32_t pos = goff[d] + wcnt[w][d] + rk[r];
            kout[pos] = kk[r];
            vout[pos] = vv[r];
        }
    }
}

// ----------------------------------------------------------------- hierarchy
__device__ __forceinline__ int kdelta(const uint32_t *__restrict__ code, int n, int i, int j) {
    if (j < 0 || j > n - 1) return -1;
    const uint32_t a = code[i], b = code[j];
    if (a != b) return __clz(a ^ b);
    return 32 + __clz((uint32_t)i ^ (uint32_t)j);
}

__global__ void k_karras(const uint32_t *__restrict__ code, int n, float4 *__restrict__ nbox,
                         uint32_t *__restrict__ parent, uint32_t *__restrict__ leaf_parent) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += gridDim.x * blockDim.x) {
        const int d = (kdelta(code, n, i, i + 1) - kdelta(code, n, i, i - 1)) >= 0 ? 1 : -1;
        const int dmin = kdelta(code, n, i, i - d);
        int lmax = 2;
        while (kdelta(code, n, i, i + lmax * d) > dmin) lmax *= 2;
        int l = 0;
        for (int t = lmax / 2; t >= 1; t /= 2)
            if (kdelta(code, n, i, i + (l + t) * d) > dmin) l += t;
        const int j = i + l * d;
        const int dnode = kdelta(code, n, i, j);
        int s = 0, t = l;
        do {
            t = (t + 1) >> 1;
            if (kdelta(code, n, i, i + (s + t) * d) > dnode) s += t;
        } while (t > 1);
        const int g = i + s * d + min(d, 0);
        const uint32_t lc = (min(i, j) == g) ? (LEAF | (uint32_t)g) : (uint32_t)g;
        const uint32_t rc = (max(i, j) == g + 1) ? (LEAF | (uint32_t)(g + 1)) : (uint32_t)(g + 1);
        // in place of the box, until the bottom-up pass: the node's first and last leaf
        nbox[2 * (size_t)i] = make_float4(__int_as_float(min(i, j)), 0.0f, 0.0f, __uint_as_float(lc));
        nbox[2 * (size_t)i + 1] = make_float4(__int_as_float(max(i, j)), 0.0f, 0.0f, __uint_as_float(rc));
        if (lc & LEAF) leaf_parent[lc & ~LEAF] = (uint32_t)i; else parent[lc] = (uint32_t)i;
        if (rc & LEAF) leaf_parent[rc & ~LEAF] = (uint32_t)i; else parent[rc] = (uint32_t)i;
        if (i == 0) parent[0] = NONE;
    }
}

// The primitive order and the triangle boxes in that order, so that a leaf's
// box is one record at the leaf's own index.
__global__ void k_gather(const float4 *__restrict__ tbox, const uint32_t *__restrict__ vals, uint32_t n,
                         uint32_t *__restrict__ order, float4 *__restrict__ lbox) {
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const uint32_t prim = vals[j];
        order[j] = prim;
        lbox[2 * (size_t)j] = tbox[2 * (size_t)prim];
        lbox[2 * (size_t)j + 1] = tbox[2 * (size_t)prim + 1];
    }
}

struct Tree {
    const float4 *lbox; // leaf boxes in sorted order
    const uint32_t *order;
    float4 *nbox;
    uint32_t *parent;
    uint32_t *leaf_parent;
    uint32_t *count;
    float *cost;
};

// Coherent (L2) reads of data written by other threads of the same kernel.
__device__ __forceinline__ Box box_of_cg(const Tree &T, uint32_t r) {
    float4 lo, hi;
    if (r & LEAF) {
        const size_t j = r & ~LEAF;
        lo = T.lbox[2 * j];
        hi = T.lbox[2 * j + 1];
    } else {
        lo = __ldcg(&T.nbox[2 * (size_t)r]);
        hi = __ldcg(&T.nbox[2 * (size_t)r + 1]);
    }
    return Box{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}};
}
__device__ __forceinline__ uint32_t left_of(const Tree &T, uint32_t x) { return __float_as_uint(__ldcg(&T.nbox[2 * (size_t)x]).w); }
__device__ __forceinline__ uint32_t right_of(const Tree &T, uint32_t x) { return __float_as_uint(__ldcg(&T.nbox[2 * (size_t)x + 1]).w); }

constexpr float kCi = 1.2f, kCt = 1.0f;

__device__ __forceinline__ float cost_of_cg(const Tree &T, uint32_t r) {
    if (r & LEAF) {
        const Box b = box_of_cg(T, r);
        return kCt * area(b);
    }
    return __ldcg(&T.cost[r]);
}

// Arrival at a node: earlier arrivals.  Releases what the thread (and, after a
// __syncwarp, its warp) wrote below the node and acquires what the other arrival
// did: one operation in place of two full fences around a relaxed atomic.
__device__ __forceinline__ uint32_t arrive(uint32_t *p) {
    uint32_t old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
    return old;
}

// The same between the threads of a block, for a counter in shared memory.
__device__ __forceinline__ uint32_t arrive_block(uint32_t *p) {
    uint32_t old;
    asm volatile("atom.acq_rel.cta.shared.add.u32 %0, [%1], 1;"
                 : "=r"(old)
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
    return old;
}

// Boxes, primitive counts and SAH costs, the second arrival at a node computing
// it.  A climb is a chain of arrivals and of reads of what other threads wrote,
// so a block takes 128 neighbouring leaves and the nodes of the same indices: those
// over leaves of its own (all but one in forty or so; such a node's index is among
// its leaves') are counted and their boxes handed on in shared memory, and only the
// nodes above go through L2 with fences for the device.  Over 4.2M leaves 490 us
// with every node through L2, 341 so with 256 leaves; two builds of that mesh with
// the block-wise bounds 10.6 -> 9.9 ms (256 leaves 9.94, 64 9.88, 512 10.3).
constexpr uint32_t kClimbLeaves = 128;
__global__ void __launch_bounds__(kClimbLeaves, 16) k_bottom_up(Tree T, uint32_t n, uint32_t *__restrict__ visits) {
    __shared__ float4 s_lo[2 * kClimbLeaves], s_hi[2 * kClimbLeaves]; // {low corner, cost}, {high corner, -}: leaves, nodes
    __shared__ uint4 s_links[kClimbLeaves]; // of the nodes with the leaves' indices: children, first and last leaf
    __shared__ uint32_t s_up[kClimbLeaves], s_visits[kClimbLeaves];
    const uint32_t base = blockIdx.x * kClimbLeaves, i = threadIdx.x, j = base + i;
    s_visits[i] = 0u;
    if (j < n) {
        const float4 lo = T.lbox[2 * (size_t)j], hi = T.lbox[2 * (size_t)j + 1];
        s_lo[i] = make_float4(lo.x, lo.y, lo.z, kCt * area(Box{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}}));
        s_hi[i] = hi;
    }
    if (j + 1u < n) {
        const float4 l = T.nbox[2 * (size_t)j], r = T.nbox[2 * (size_t)j + 1];
        s_links[i] = make_uint4(__float_as_uint(l.w), __float_as_uint(r.w), __float_as_uint(l.x), __float_as_uint(r.x));
        s_up[i] = T.parent[j];
    }
    __syncthreads();
    uint32_t x = j < n ? T.leaf_parent[j] : NONE;
    while (x != NONE) {
        uint32_t up;
        uint4 links;
        if (x - base < kClimbLeaves) {
            links = s_links[x - base];
            up = s_up[x - base];
        } else { // there before the arrival, and unchanged until the second
            const float4 l = __ldcg(&T.nbox[2 * (size_t)x]), r = __ldcg(&T.nbox[2 * (size_t)x + 1]);
            links = make_uint4(__float_as_uint(l.w), __float_as_uint(r.w), __float_as_uint(l.x), __float_as_uint(r.x));
            up = T.parent[x];
        }
        const uint32_t lc = links.x, rc = links.y, first = links.z, last = links.w;
        const bool own = first >= base && last < base + kClimbLeaves;
        Box b;
        float cost;
        if (own) {
            if (arrive_block(&s_visits[x - base]) == 0u) break;
            const uint32_t l = (lc & LEAF) ? (lc & ~LEAF) - base : lc - base + kClimbLeaves;
            const uint32_t r = (rc & LEAF) ? (rc & ~LEAF) - base : rc - base + kClimbLeaves;
            const float4 l0 = s_lo[l], l1 = s_hi[l], r0 = s_lo[r], r1 = s_hi[r];
            b = merge(Box{{l0.x, l0.y, l0.z}, {l1.x, l1.y, l1.z}}, Box{{r0.x, r0.y, r0.z}, {r1.x, r1.y, r1.z}});
            cost = kCi * area(b) + (l0.w + r0.w);
            const uint32_t own_place = x - base + kClimbLeaves;
            s_lo[own_place] = make_float4(b.lo[0], b.lo[1], b.lo[2], cost);
            s_hi[own_place] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.0f);
        } else {
            if (arrive(&visits[x]) == 0u) break;
            b = merge(box_of_cg(T, lc), box_of_cg(T, rc));
            cost = kCi * area(b) + (cost_of_cg(T, lc) + cost_of_cg(T, rc));
        }
        T.count[x] = last - first + 1u;
        T.cost[x] = cost;
        T.nbox[2 * (size_t)x] = make_float4(b.lo[0], b.lo[1], b.lo[2], __uint_as_float(lc));
        T.nbox[2 * (size_t)x + 1] = make_float4(b.hi[0], b.hi[1], b.hi[2], __uint_as_float(rc));
        x = up;
    }
}

// ----------------------------------------------------------------- treelets
// A warp's working set for one treelet, in shared memory.
struct TreeletWork {
    float aS[128], cS[128]; // subset areas and costs
    uint8_t pS[128];        // best partition of each subset
    float4 lo[7], hi[7];    // the treelet leaves' boxes
    uint32_t leaves[7], count[7], internals[6];
    int st_s[8];            // rebuild stack: subset, node
    uint32_t st_n[8];
};

// The subsets of seven leaves by size (2..5), ascending within a size.
struct SubsetTable {
    uint8_t s[112];
};
constexpr SubsetTable make_subsets() {
    SubsetTable t{};
    int at = 0;
    for (int k = 2; k <= 5; ++k) {
        for (int s = 1; s < 128; ++s) {
            int c = 0;
            for (int b = 0; b < 7; ++b) c += (s >> b) & 1;
            if (c == k) t.s[at++] = (uint8_t)s;
        }
    }
    return t;
}
__device__ const SubsetTable kSubsets = make_subsets();
// First subset of size k in the table (21, 35, 35 and 21 of them).
template <int K> constexpr int kSubsetFirst = K == 2 ? 0 : K == 3 ? 21 : K == 4 ? 56 : K == 5 ? 91 : 112;

// Costs of the subsets of size K: one lane per subset, its 2^(K-1) - 1
// partitions (those with the lowest leaf) in the CPU form's order.  A
// partition's cells follow from an earlier one's by an addition each: part j
// without its highest leaf's cell is a part already formed, and the other half
// is what is left of the whole.
template <int K>
__device__ __forceinline__ void treelet_subsets(TreeletWork &w, const uint8_t *subsets, int nsub, uint32_t lane) {
    for (int i = kSubsetFirst<K> + (int)lane; i < kSubsetFirst<K + 1>; i += 32) {
        const int s = subsets[i];
        if (s >= nsub) continue;
        // part[j]: the lowest leaf and those of the others but the highest that j's bits choose
        constexpr int H = 1 << (K - 2);
        int part[H];
        int left = s & (s - 1);
        part[0] = s ^ left;
#pragma unroll
        for (int k = 0; k < K - 2; ++k) {
            const int bit = left & -left;
            left ^= bit;
#pragma unroll
            for (int j = 0; j < (1 << k); ++j) part[j + (1 << k)] = part[j] + bit;
        }
        // the parts with the highest leaf (`left` by now), the whole set apart, and then those without
        float best = FLT_MAX;
        int bp = part[0];
#pragma unroll
        for (int j = H - 2; j >= 0; --j) {
            const int P = part[j] + left;
            const float c = w.cS[P] + w.cS[s - P];
            if (c < best) { best = c; bp = P; }
        }
#pragma unroll
        for (int j = H - 1; j >= 0; --j) {
            const float c = w.cS[part[j]] + w.cS[s - part[j]];
            if (c < best) { best = c; bp = part[j]; }
        }
        w.cS[s] = kCi * w.aS[s] + best;
        w.pS[s] = (uint8_t)bp;
    }
    __syncwarp();
}

// One node or leaf as a treelet lane holds it.
struct TreeletLeaf {
    uint32_t ref, left, right, count;
    float4 lo, hi;
    float cost;
};
__device__ __forceinline__ TreeletLeaf treelet_leaf(const Tree &T, uint32_t ref) {
    // leaves and nodes by the same loads: the two lanes that read at a time do not wait for one another
    const bool leaf = (ref & LEAF) != 0u;
    const size_t j = ref & ~LEAF;
    const float4 *p = leaf ? T.lbox : T.nbox;
    TreeletLeaf l;
    l.ref = ref;
    l.lo = __ldcg(&p[2 * j]);
    l.hi = __ldcg(&p[2 * j + 1]);
    l.count = 1u;
    float cost = 0.0f;
    if (!leaf) {
        l.count = __ldcg(&T.count[j]);
        cost = __ldcg(&T.cost[j]);
    }
    l.left = __float_as_uint(l.lo.w);
    l.right = __float_as_uint(l.hi.w);
    l.cost = leaf ? kCt * area3(l.hi.x - l.lo.x, l.hi.y - l.lo.y, l.hi.z - l.lo.z) : cost;
    return l;
}

// The 7-leaf treelet rooted at r is restructured (Karras & Aila 2013) by the
// 32 lanes of a warp, with the same result as the CPU form: growth by largest
// area (first maximum), DP over subsets in increasing size with partitions
// containing the lowest set bit, first minimum kept (in the CPU's
// enumeration, q = rest, (q - 1) & rest, ...: the larger partition wins a
// tie), internal nodes reused in formation order, pre-order rebuild.
//
// One treelet is a chain of dependent steps, and a round has as many treelets
// one after another as the tree is deep, so both its instructions (a large
// mesh) and its latency (a small one) count.  Lane j holds treelet leaf j with
// its box, children, count and cost, so that a growth step is one node read; areas
// and costs are never negative, so their maxima and minima are one REDUX on the
// bits; subsets of 2 to 5 leaves come from a table (a lane per subset, no lane
// idle for another size's), those of 6 and 7 spread their partitions over the
// lanes; the rebuilt nodes are written by a lane each, with counts from the
// leaves' own.  Against areas reduced by shuffles, subsets filtered by
// population count, children read after the choice and one lane rebuilding: two
// builds of a 4.2M-triangle mesh, one with three rounds, 49.3 -> 21.6 ms; the
// 10,007-triangle build with three rounds 2.73 -> 1.12 ms.
// `left`, `right` and `root_area` are the root's children and box area.
__device__ void optimize_treelet(const Tree &T, uint32_t r, uint32_t left, uint32_t right, float root_area, TreeletWork &w,
                                 const uint8_t *subsets) {
    const uint32_t lane = threadIdx.x & 31u;
    TreeletLeaf l{};
    l.ref = LEAF;
    if (lane < 2u) l = treelet_leaf(T, lane ? right : left);
    const float cost_r = kCi * root_area + (__shfl_sync(0xFFFFFFFFu, l.cost, 0) + __shfl_sync(0xFFFFFFFFu, l.cost, 1));
    int nl = 2;
    while (nl < 7) {
        // the internal leaf of largest area (lowest index on ties); none: the treelet is complete.
        // A NaN area is never chosen.
        const float a = area3(l.hi.x - l.lo.x, l.hi.y - l.lo.y, l.hi.z - l.lo.z);
        const uint32_t key = !(l.ref & LEAF) && a >= 0.0f ? __float_as_uint(a) + 1u : 0u;
        const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, key);
        if (top == 0u) break;
        const int bj = __ffs(__ballot_sync(0xFFFFFFFFu, key == top)) - 1;
        const uint32_t x = __shfl_sync(0xFFFFFFFFu, l.ref, bj);
        const uint32_t xl = __shfl_sync(0xFFFFFFFFu, l.left, bj), xr = __shfl_sync(0xFFFFFFFFu, l.right, bj);
        if (lane == 0u) w.internals[nl - 2] = x;
        if ((int)lane == bj || (int)lane == nl) l = treelet_leaf(T, (int)lane == bj ? xl : xr);
        ++nl;
    }
    if (nl < 3) {
        if (lane == 0u) T.cost[r] = cost_r;
        return;
    }
    const int nsub = 1 << nl;
    if ((int)lane < nl) {
        w.lo[lane] = l.lo;
        w.hi[lane] = l.hi;
        w.leaves[lane] = l.ref;
        w.count[lane] = l.count;
        w.cS[1 << lane] = l.cost;
        w.pS[1 << lane] = 0;
    }
    __syncwarp();
    {
        // a lane's four subsets share its choice of the first five leaves; leaves are merged in their
        // order (it counts where a corner is a NaN)
        Box b{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
        auto with = [&](const Box &x, int j) {
            const float4 lo = w.lo[j], hi = w.hi[j];
            return merge(x, Box{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}});
        };
#pragma unroll
        for (int j = 0; j < 5; ++j)
            if (j < nl && (lane >> j) & 1u) b = with(b, j);
        w.aS[lane] = area(b);
        if (nl >= 6) {
            const Box b5 = with(b, 5);
            w.aS[lane + 32] = area(b5);
            if (nl >= 7) {
                w.aS[lane + 64] = area(with(b, 6));
                w.aS[lane + 96] = area(with(b5, 6));
            }
        }
    }
    __syncwarp();
    treelet_subsets<2>(w, subsets, nsub, lane);
    treelet_subsets<3>(w, subsets, nsub, lane);
    treelet_subsets<4>(w, subsets, nsub, lane);
    treelet_subsets<5>(w, subsets, nsub, lane);
    if (nl >= 6) {
        // the subsets of six leaves (all but leaf m): their 31 partitions over the lanes
#pragma unroll
        for (int m = 0; m < 7; ++m) {
            const int s = 127 ^ (1 << m);
            if (s >= nsub) continue;
            // lane's bits deposited into the subset without its lowest leaf
            const uint32_t q = m == 0 ? lane << 2
                                      : ((lane & ((1u << (m - 1)) - 1u)) << 1) | ((lane >> (m - 1)) << (m + 1));
            const int P = (int)(q | (m == 0 ? 2u : 1u));
            const float c = lane < 31u ? w.cS[P] + w.cS[s ^ P] : INFINITY;
            const uint32_t best = __reduce_min_sync(0xFFFFFFFFu, __float_as_uint(c));
            const uint32_t bp = __reduce_max_sync(0xFFFFFFFFu, lane < 31u && __float_as_uint(c) == best ? (uint32_t)P : 1u);
            if (lane == 0u) {
                w.cS[s] = kCi * w.aS[s] + __uint_as_float(best);
                w.pS[s] = (uint8_t)bp;
            }
        }
        __syncwarp();
    }
    if (nl == 7) {
        // all seven: 63 partitions, the larger of a lane's two on a tie
        const int P0 = (int)(lane << 1) | 1, P1 = P0 + 64;
        const float c0 = w.cS[P0] + w.cS[127 ^ P0], c1 = lane < 31u ? w.cS[P1] + w.cS[127 ^ P1] : INFINITY;
        const uint32_t best = __reduce_min_sync(0xFFFFFFFFu, __float_as_uint(fminf(c0, c1)));
        const uint32_t p = lane < 31u && __float_as_uint(c1) == best ? (uint32_t)P1
                                                                       : (__float_as_uint(c0) == best ? (uint32_t)P0 : 1u);
        const uint32_t bp = __reduce_max_sync(0xFFFFFFFFu, p);
        if (lane == 0u) {
            w.cS[127] = kCi * w.aS[127] + __uint_as_float(best);
            w.pS[127] = (uint8_t)bp;
        }
        __syncwarp();
    }
    const int full = nsub - 1;
    if (!(w.cS[full] < cost_r)) {
        if (lane == 0u) T.cost[r] = cost_r;
        return;
    }
    // pre-order walk of the chosen partitions (every lane the same); lane k keeps the k-th node
    int my_s = 0, sp = 1, next = 0, np = 0;
    uint32_t my_n = 0, my_k0 = 0, my_k1 = 0;
    int S = full;
    uint32_t node = r;
    for (;;) {
        const int P = w.pS[S], Q = S ^ P;
        const bool one0 = (P & (P - 1)) == 0, one1 = (Q & (Q - 1)) == 0;
        const uint32_t k0 = one0 ? w.leaves[__ffs(P) - 1] : w.internals[next];
        next += one0 ? 0 : 1;
        const uint32_t k1 = one1 ? w.leaves[__ffs(Q) - 1] : w.internals[next];
        next += one1 ? 0 : 1;
        if ((int)lane == np) {
            my_s = S;
            my_n = node;
            my_k0 = k0;
            my_k1 = k1;
        }
        ++np;
        if (!one0) {
            if (!one1) {
                w.st_s[sp] = Q;
                w.st_n[sp] = k1;
                ++sp;
            }
            S = P;
            node = k0;
        } else if (!one1) {
            S = Q;
            node = k1;
        } else {
            if (sp == 1) break;
            --sp;
            S = w.st_s[sp];
            node = w.st_n[sp];
        }
    }
    if ((int)lane < np) {
        Box b{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
        uint32_t cnt = 0;
        for (int j = 0; j < nl; ++j)
            if (my_s & (1 << j)) {
                const float4 lo = w.lo[j], hi = w.hi[j];
                b = merge(b, Box{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}});
                cnt += w.count[j];
            }
        T.nbox[2 * (size_t)my_n] = make_float4(b.lo[0], b.lo[1], b.lo[2], __uint_as_float(my_k0));
        T.nbox[2 * (size_t)my_n + 1] = make_float4(b.hi[0], b.hi[1], b.hi[2], __uint_as_float(my_k1));
        T.count[my_n] = cnt;
        T.cost[my_n] = w.cS[my_s];
        if (my_k0 & LEAF) T.leaf_parent[my_k0 & ~LEAF] = my_n; else T.parent[my_k0] = my_n;
        if (my_k1 & LEAF) T.leaf_parent[my_k1 & ~LEAF] = my_n; else T.parent[my_k1] = my_n;
    }
}

// Bottom-up pass over the tree, a warp starting from `per` leaves: a lane goes
// on to a node's parent only on the node's second arrival (both subtrees final);
// the nodes of at least `gamma` leaves that the lanes reach in a step are
// restructured one after another by the whole warp.
//
// A block is one warp, so that its place is free as soon as its climb ends
// (climbs differ in length by the tree's depth), and 64 registers let the 32
// blocks of an SM run at once: with the subsets' cells by one addition and leaves
// and nodes read by the same loads, two builds of a 4.2M-triangle mesh, one with
// three rounds, 11.7 -> 10.6 ms (blocks of two warps 10.7, of four 11.1; left at
// 89 registers 11.9).
__global__ void __launch_bounds__(32, 32) k_treelet(Tree T, uint32_t n, uint32_t *__restrict__ visits, uint32_t gamma,
                                                    uint32_t per) {
    __shared__ TreeletWork s_w;
    __shared__ uint8_t s_subsets[112];
    const uint32_t lane = threadIdx.x;
    for (uint32_t i = lane; i < 112u; i += 32u) s_subsets[i] = kSubsets.s[i];
    __syncwarp();
    const uint32_t j = blockIdx.x * per + lane;
    uint32_t x = lane < per && j < n ? __ldcg(&T.leaf_parent[j]) : NONE;
    bool active = x != NONE;
    while (__any_sync(0xFFFFFFFFu, active)) {
        bool need = false;
        uint32_t up = NONE, left = 0u, right = 0u;
        float node_area = 0.0f;
        if (active) {
            // the node's own record is final (only its parent's treelets will change it), so it is
            // read while the arrival is under way
            up = __ldcg(&T.parent[x]);
            const uint32_t count = __ldcg(&T.count[x]);
            const float4 lo = __ldcg(&T.nbox[2 * (size_t)x]), hi = __ldcg(&T.nbox[2 * (size_t)x + 1]);
            left = __float_as_uint(lo.w);
            right = __float_as_uint(hi.w);
            node_area = area3(hi.x - lo.x, hi.y - lo.y, hi.z - lo.z);
            active = arrive(&visits[x]) != 0u;
            need = active && count >= gamma;
        }
        uint32_t m;
        while ((m = __ballot_sync(0xFFFFFFFFu, need)) != 0u) {
            const int leader = __ffs(m) - 1;
            const uint32_t r = __shfl_sync(0xFFFFFFFFu, x, leader);
            const uint32_t rl = __shfl_sync(0xFFFFFFFFu, left, leader), rr = __shfl_sync(0xFFFFFFFFu, right, leader);
            const float ra = __shfl_sync(0xFFFFFFFFu, node_area, leader);
            __syncwarp();
            optimize_treelet(T, r, rl, rr, ra, s_w, s_subsets);
            __syncwarp(); // the lanes' writes come before the owner's arrival; the working set is free again
            if ((int)lane == leader) need = false;
        }
        if (active) {
            x = up;
            if (x == NONE) active = false;
        }
    }
}

// ----------------------------------------------------------------- collapse
// The wide BVH is laid out level by level.  What a level needs of the one
// before is only its nodes in order, so a level runs two small kernels without
// the host: k_level_open chooses each node's children (greedy expansion of the
// largest area) and their octant codes, eight lanes to a node, and k_level_link
// numbers the level's children and triangles.  Between the two and the final
// kernel a node's record holds its children in binary-tree terms (NodeDraft);
// k_emit then quantizes and writes all nodes and triangle slots at once.  (A
// thread per node took 45 to 200 us a level for the chain of its own steps, two
// single-block scans and a host synchronisation beside it: with the merged
// bottom-up pass and the row scans of the sort, two builds of a 4.2M-triangle
// mesh 21.6 -> 14.5 ms, 10,007 triangles with three treelet rounds 1.12 -> 0.68;
// octant scores compared as keys, made once a node, 8.87 -> 8.66 by then.)
struct Collapse {
    Tree T;
    const float *verts;  // the BVH's own triangles (model-local indexing)
    const uint32_t *mat_idx; // material of each triangle, for slot_nm
    float4 *slot_nm;     // per triangle slot {geometric normal, material bits}, or null
    uint8_t *wide;       // this BVH's first node
    float4 *tris;        // triangle slot array
    uint32_t W, leaf_max, node_bytes;
    uint32_t node_base, node_cap; // index of the BVH's first node in the whole array; nodes there are room for
    uint32_t slot_base;  // index of its first triangle slot
    uint32_t prim_base;  // added to the primitive index stored in a triangle slot (scene-global ids)
};

// Progress of the collapse: the level about to be laid out.
struct LevelState {
    uint32_t count;      // its nodes (0: done)
    uint32_t node_start; // its first node: all nodes so far
    uint32_t tri_start;  // triangle slots taken by the levels before
    uint32_t depth;      // levels laid out
    uint32_t overflow;   // the next level would not fit: the collapse stopped
};

// A node's record until k_emit: words [0, W) its children (binary node or LEAF |
// leaf), bytes of words W and W + 1 their codes (kNoChild: none; bit 3: a leaf
// slot, its triangle count in bits 4-5), word W + 2 its first child's index,
// W + 3 its first triangle slot.  4 W + 16 bytes: 48 / 32 / 24 of 80 / 64 / 48.
constexpr uint32_t kNoChild = 0xFFu, kLeafSlot = 8u;

constexpr uint32_t kLevelThreads = 256, kLevelBlocks = 608;

__global__ void k_collapse_start(uint32_t *level, LevelState *st, uint32_t root) {
    if (threadIdx.x != 0) return;
    level[0] = root;
    st[0] = LevelState{1u, 0u, 0u, 0u, 0u};
}

// Nodes [first, last) of a level that block b lays out.
__device__ __forceinline__ void level_share(uint32_t count, uint32_t &first, uint32_t &last) {
    const uint32_t share = (count + gridDim.x - 1) / gridDim.x;
    first = min(count, blockIdx.x * share);
    last = min(count, first + share);
}

// Largest `key` of the lane's group of eight and the first lane that has it.
__device__ __forceinline__ uint32_t group_top(uint32_t key, uint32_t &who) {
    uint32_t top = key;
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, off, 8));
    const uint32_t eq = __ballot_sync(0xFFFFFFFFu, key == top);
    who = (uint32_t)__ffs((eq >> (threadIdx.x & 24u)) & 0xFFu) - 1u;
    return top;
}

// Box of a group's children, lane i holding child i.  The corners' minima and maxima
// may be taken in any order unless one is a NaN, which the next child replaces: then
// the children are merged one after the other, as the CPU form does.
__device__ __forceinline__ Box group_merge(Box b, bool child) {
    bool nan = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) nan = nan || b.lo[a] != b.lo[a] || b.hi[a] != b.hi[a];
    if (__any_sync(0xFFFFFFFFu, child && nan)) {
        Box r = b;
        for (int j = 0; j < 8; ++j) {
            Box o;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                o.lo[a] = __shfl_sync(0xFFFFFFFFu, b.lo[a], j, 8);
                o.hi[a] = __shfl_sync(0xFFFFFFFFu, b.hi[a], j, 8);
            }
            if (__shfl_sync(0xFFFFFFFFu, child, j, 8)) r = j ? merge(r, o) : o;
        }
        return r;
    }
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            b.lo[a] = fmn(b.lo[a], __shfl_xor_sync(0xFFFFFFFFu, b.lo[a], off, 8));
            b.hi[a] = fmx(b.hi[a], __shfl_xor_sync(0xFFFFFFFFu, b.hi[a], off, 8));
        }
    return b;
}

struct LevelChild {
    uint32_t ref, left, right, count;
    Box b;
};
__device__ __forceinline__ LevelChild level_child(const Tree &T, uint32_t ref) {
    const size_t j = ref & ~LEAF;
    const float4 *p = (ref & LEAF) ? T.lbox : T.nbox;
    const float4 lo = p[2 * j], hi = p[2 * j + 1];
    LevelChild c;
    c.ref = ref;
    c.left = __float_as_uint(lo.w);
    c.right = __float_as_uint(hi.w);
    c.count = (ref & LEAF) ? 1u : T.count[j];
    c.b = Box{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}};
    return c;
}

__global__ void __launch_bounds__(kLevelThreads) k_level_open(Collapse C, const LevelState *__restrict__ st,
                                                              const uint32_t *__restrict__ level, uint32_t *__restrict__ nic,
                                                              unsigned long long *__restrict__ bsum) {
    __shared__ unsigned long long s_sum;
    const LevelState ls = *st;
    uint32_t first, last;
    level_share(ls.count, first, last);
    if (threadIdx.x == 0) s_sum = 0ull;
    __syncthreads();
    const uint32_t c = threadIdx.x & 7u;
    unsigned long long mine = 0ull;
    for (uint32_t k0 = first; k0 < last; k0 += kLevelThreads / 8u) {
        const uint32_t k = k0 + (threadIdx.x >> 3);
        const bool live = k < last;
        const uint32_t r = live ? level[k] : LEAF;
        uint32_t m = 0; // the group's children so far: lane i holds child i
        LevelChild e{};
        e.b = Box{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
        if (live) {
            m = (r & LEAF) ? 1u : 2u;
            if (r & LEAF) {
                if (c == 0u) e = level_child(C.T, r);
            } else if (c < 2u) {
                e = level_child(C.T, __float_as_uint(C.T.nbox[2 * (size_t)r + c].w));
            }
        }
        for (uint32_t it = 2; it < C.W; ++it) {
            // open the internal child of largest area (the first of equals; NaN never)
            const float a = area(e.b);
            uint32_t who;
            const uint32_t top = group_top(c < m && !(e.ref & LEAF) && a >= 0.0f ? __float_as_uint(a) + 1u : 0u, who);
            const uint32_t xl = __shfl_sync(0xFFFFFFFFu, e.left, (int)who, 8), xr = __shfl_sync(0xFFFFFFFFu, e.right, (int)who, 8);
            if (top != 0u) {
                if (c == who || c == m) e = level_child(C.T, c == who ? xl : xr);
                ++m;
            }
        }
        const bool child = c < m;
        // octant codes: repeatedly the largest projection of a child's centre (seen from the
        // node's) on a free octant's diagonal; the first child, then the first code, of equals
        const Box nb = group_merge(e.b, child);
        float off[3];
        uint32_t score[8]; // by order-preserving key; 0: not a number
#pragma unroll
        for (int a = 0; a < 3; ++a) off[a] = (e.b.lo[a] + e.b.hi[a]) * 0.5f - (nb.lo[a] + nb.hi[a]) * 0.5f;
        bool nan = false;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float sx = (q & 4) ? -1.0f : 1.0f, sy = (q & 2) ? -1.0f : 1.0f, sz = (q & 1) ? -1.0f : 1.0f;
            const float s = (off[0] * sx + off[1] * sy) + off[2] * sz;
            score[q] = s == s ? f2key(s + 0.0f) : 0u; // + 0: no negative zero
            nan = nan || s != s;
        }
        const bool odd = __any_sync(0xFFFFFFFFu, child && nan);
        uint32_t used = 0u, code = 0u;
        bool placed = !child;
        for (uint32_t it = 0; it < C.W; ++it) {
            uint32_t bs = 0u, bc = 0u;
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q)
                if (!(used & (1u << q)) && score[q] > bs) {
                    bs = score[q];
                    bc = q;
                }
            if (odd) {
                // the first child's first code stands against any other if it is not a number
                const uint32_t open = __ballot_sync(0xFFFFFFFFu, !placed) >> (threadIdx.x & 24u) & 0xFFu;
                const uint32_t q0 = (uint32_t)__ffs(~used) - 1u;
                bool none = false;
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) none = none || (q == q0 && score[q] == 0u);
                if (none && (open & (0u - open)) == 1u << c) {
                    bs = 0xFFFFFFFFu;
                    bc = q0;
                }
            }
            uint32_t who;
            const uint32_t top = group_top(placed ? 0u : bs, who);
            const uint32_t q = __shfl_sync(0xFFFFFFFFu, bc, (int)who, 8);
            if (top != 0u) {
                used |= 1u << q;
                if (c == who) {
                    code = q;
                    placed = true;
                }
            }
        }
        const bool leafslot = child && ((e.ref & LEAF) || e.count <= C.leaf_max);
        const uint32_t gshift = threadIdx.x & 24u;
        const uint32_t ni = (uint32_t)__popc((__ballot_sync(0xFFFFFFFFu, child && !leafslot) >> gshift) & 0xFFu);
        uint32_t nt = leafslot ? e.count : 0u;
#pragma unroll
        for (int o = 4; o >= 1; o >>= 1) nt += __shfl_xor_sync(0xFFFFFFFFu, nt, o, 8);
        if (live) {
            uint8_t *rec = C.wide + (size_t)(ls.node_start + k) * C.node_bytes;
            if (c < C.W) reinterpret_cast<uint32_t *>(rec)[c] = e.ref;
            rec[4 * C.W + c] = (uint8_t)(child ? code | (leafslot ? kLeafSlot | e.count << 4 : 0u) : kNoChild);
            if (c == 0u) {
                nic[k] = ni | nt << 8;
                mine += (unsigned long long)ni | (unsigned long long)nt << 32;
            }
        }
    }
    if (mine) atomicAdd(&s_sum, mine);
    __syncthreads();
    if (threadIdx.x == 0) bsum[blockIdx.x] = s_sum;
}

__global__ void __launch_bounds__(kLevelThreads) k_level_link(Collapse C, const LevelState *__restrict__ st, LevelState *next_st,
                                                              const uint32_t *__restrict__ nic,
                                                              const unsigned long long *__restrict__ bsum,
                                                              uint32_t *__restrict__ next_level) {
    __shared__ uint32_t sums[8];
    const LevelState ls = *st;
    uint32_t first, last;
    level_share(ls.count, first, last);
    // children and triangles of the blocks before
    uint32_t at_n = 0, at_t = 0;
    {
        uint32_t sn = 0, stt = 0;
        for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kLevelThreads) {
            const unsigned long long v = bsum[b];
            sn += (uint32_t)v;
            stt += (uint32_t)(v >> 32);
        }
        block_prefix(sn, sums, &at_n);
        block_prefix(stt, sums, &at_t);
    }
    const uint32_t next_start = ls.node_start + ls.count;
    for (uint32_t k0 = first; k0 < last; k0 += kLevelThreads) {
        const uint32_t k = k0 + threadIdx.x;
        const uint32_t v = k < last ? nic[k] : 0u;
        uint32_t tot_n, tot_t;
        const uint32_t cn = at_n + block_prefix(v & 0xFFu, sums, &tot_n), ct = at_t + block_prefix(v >> 8, sums, &tot_t);
        if (k < last) {
            uint32_t *rec = reinterpret_cast<uint32_t *>(C.wide + (size_t)(ls.node_start + k) * C.node_bytes);
            const unsigned long long codes = (unsigned long long)rec[C.W] | (unsigned long long)rec[C.W + 1] << 32;
            uint32_t imask = 0;
            for (uint32_t i = 0; i < C.W; ++i) {
                const uint32_t q = (uint32_t)(codes >> (8 * i)) & 0xFFu;
                if (q != kNoChild && !(q & kLeafSlot)) imask |= 1u << (q & 7u);
            }
            for (uint32_t i = 0; i < C.W; ++i) {
                const uint32_t q = (uint32_t)(codes >> (8 * i)) & 0xFFu;
                if (q != kNoChild && !(q & kLeafSlot)) next_level[cn + __popc(imask & ((1u << (q & 7u)) - 1u))] = rec[i];
            }
            rec[C.W + 2] = C.node_base + next_start + cn;
            rec[C.W + 3] = C.slot_base + ls.tri_start + ct;
        }
        at_n += tot_n;
        at_t += tot_t;
    }
    if (blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) {
        LevelState nx = ls;
        if (ls.count) {
            nx.node_start = next_start;
            nx.tri_start += at_t;
            nx.depth += 1u;
            // the next level would write nodes [next_start, next_start + at_n)
            nx.overflow = at_n > C.node_cap - next_start ? 1u : 0u;
            nx.count = nx.overflow ? 0u : at_n;
        }
        *next_st = nx;
    }
}

__device__ __forceinline__ int ceil_log2(double x) {
    int k;
    const double m = frexp(x, &k);
    return (m == 0.5) ? k - 1 : k;
}
__device__ __forceinline__ int floor_log2(double x) {
    int k;
    frexp(x, &k);
    return k - 1;
}

// ceil(log2(ext / 252)) with the quotient rounded to double, for ext > 0, without
// the division: with ext = m 2^e it is e - 7 for m <= 252/128, else e - 6 (the
// doubles next to 252 2^k lie further from it than the quotient's rounding can
// close).  Double arithmetic runs at a sixty-fourth of the float rate here.
__device__ __forceinline__ int ceil_log2_252nd(double ext) {
    const uint32_t hi = (uint32_t)__double2hiint(ext), lo = (uint32_t)__double2loint(ext);
    const uint32_t e = hi >> 20, m = hi & 0xFFFFFu;
    if (e - 1u >= 0x7FEu) return ceil_log2(ext / 252.0); // infinite, NaN or subnormal
    return (int)e - 1023 - (m > 0xF8000u || (m == 0xF8000u && lo != 0u) ? 6 : 7);
}

// Quantized planes of a node's frame: floor((x - p) / 2^e) - 1, at least 0, and
// ceil((x - p) / 2^e) + 1, at most 255, of the quotient in double, as the CPU form
// takes them.  x - p is at least a quantum and below 2^9 of them, so its float
// value decides the whole number unless it is one itself and the exact difference
// is not; only then is the difference formed in double.
template <bool HI>
__device__ __forceinline__ uint32_t quantum_of(float x, float p, float inv_quantum, int e) {
    const float d = x - p, bb = d - x; // two-sum of x and -p: err is exactly what d dropped
    const float err = (x - (d - bb)) + (-p - bb);
    const float q = d * inv_quantum, fl = floorf(q);
    if (q >= 1.0f && q < 512.0f && (fl != q || err == 0.0f)) {
        if (HI) return (uint32_t)fminf(ceilf(q) + 1.0f, 255.0f);
        return (uint32_t)(fl - 1.0f);
    }
    const double v = ((double)x - (double)p) * ldexp(1.0, -e);
    if (HI) {
        double qh = ceil(v) + 1.0;
        if (qh > 255.0) qh = 255.0;
        return (uint32_t)qh;
    }
    double ql = floor(v) - 1.0;
    if (ql < 0.0) ql = 0.0;
    return (uint32_t)ql;
}

// Quantizes and writes every node and the triangle slots, eight lanes to a node.
__global__ void __launch_bounds__(kLevelThreads) k_emit(Collapse C, const LevelState *__restrict__ st) {
    __shared__ __align__(16) uint8_t s_node[kLevelThreads / 8][80];
    const LevelState ls = *st;
    if (ls.count != 0u || ls.overflow) return; // levels are still to come, or the collapse stopped
    const uint32_t n_wide = ls.node_start, W = C.W;
    const uint32_t c = threadIdx.x & 7u, gshift = threadIdx.x & 24u;
    uint8_t *buf = s_node[threadIdx.x >> 3];
    for (uint32_t k0 = blockIdx.x * (kLevelThreads / 8u); k0 < n_wide; k0 += gridDim.x * (kLevelThreads / 8u)) {
        const uint32_t k = k0 + (threadIdx.x >> 3);
        const bool live = k < n_wide;
        uint8_t *rec = C.wide + (size_t)(live ? k : 0u) * C.node_bytes;
        const uint32_t *rw = reinterpret_cast<const uint32_t *>(rec);
        const uint32_t q = live && c < W ? rec[4 * W + c] : kNoChild;
        const uint32_t ref = q != kNoChild ? rw[c] : LEAF;
        const uint32_t cbase = live ? rw[W + 2] : 0u, tbase = live ? rw[W + 3] : 0u;
        const bool child = q != kNoChild, leafslot = child && (q & kLeafSlot);
        const uint32_t code = q & 7u, cnt = leafslot ? q >> 4 : 0u;
        Box b{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
        if (child) b = level_child(C.T, ref).b;
        const Box nb = group_merge(b, child);
        // the frame of axis a, on lane a
        int ex = 0;
        float pf = 0.0f;
        if (live && c < 3u) {
            const double lo = c == 0u ? nb.lo[0] : c == 1u ? nb.lo[1] : nb.lo[2];
            const double hi = c == 0u ? nb.hi[0] : c == 1u ? nb.hi[1] : nb.hi[2];
            const double ext = hi - lo;
            const double mag = fmax(fabs(lo), fabs(hi));
            int eh = -126;
            if (ext > 0.0) eh = max(eh, ceil_log2_252nd(ext));
            if (mag > 0.0) eh = max(eh, floor_log2(mag) - 21);
            if (eh > 100) eh = 100;
            ex = eh;
            const double pd = lo - ldexp(1.0, eh);
            pf = __double2float_rd(pd);
        }
        int e3[3];
        float p3[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            e3[a] = __shfl_sync(0xFFFFFFFFu, ex, a, 8);
            p3[a] = __shfl_sync(0xFFFFFFFFu, pf, a, 8);
        }
        // slots: by code in a node of eight, else the codes in use closed up
        uint32_t valid = child ? 1u << code : 0u, imask = child && !leafslot ? 1u << code : 0u, toff = 0u;
#pragma unroll
        for (int o = 4; o >= 1; o >>= 1) {
            valid |= __shfl_xor_sync(0xFFFFFFFFu, valid, o, 8);
            imask |= __shfl_xor_sync(0xFFFFFFFFu, imask, o, 8);
        }
        for (int j = 0; j < 8; ++j) {
            const uint32_t oc = __shfl_sync(0xFFFFFFFFu, code, j, 8), on = __shfl_sync(0xFFFFFFFFu, cnt, j, 8);
            toff += oc < code ? on : 0u;
        }
        const uint32_t slot = W == 8u ? code : (uint32_t)__popc(valid & ((1u << code) - 1u));
        const uint32_t slots = W == 8u ? valid : (1u << __popc(valid)) - 1u;
        if (c < W && !((slots >> c) & 1u)) { // empty slot: inverted box (lo 255, hi 0) fails every slab test
            buf[24 + c] = 0;
            for (uint32_t a = 0; a < 3; ++a) {
                buf[24 + W + a * W + c] = 255;
                buf[24 + 4 * W + a * W + c] = 0;
            }
        }
        if (c >= 3u) // padding behind the planes (48 and 64 byte nodes: 10 and 12 bytes)
            for (uint32_t o = 24 + 7 * W + (c - 3u); o < C.node_bytes; o += 5u) buf[o] = 0;
        if (child) {
            buf[24 + slot] = (uint8_t)(leafslot ? (((1u << cnt) - 1u) << 5) | toff : 0x20u | (24u + code));
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float inv_quantum = __uint_as_float((uint32_t)(127 - e3[a]) << 23);
                buf[24 + W + a * W + slot] = (uint8_t)quantum_of<false>(b.lo[a], p3[a], inv_quantum, e3[a]);
                buf[24 + 4 * W + a * W + slot] = (uint8_t)quantum_of<true>(b.hi[a], p3[a], inv_quantum, e3[a]);
            }
        }
        if (c == 0u) {
            uint32_t *h = reinterpret_cast<uint32_t *>(buf);
            h[0] = __float_as_uint(p3[0]);
            h[1] = __float_as_uint(p3[1]);
            h[2] = __float_as_uint(p3[2]);
            h[3] = (uint32_t)(e3[0] + 127) | ((uint32_t)(e3[1] + 127) << 8) | ((uint32_t)(e3[2] + 127) << 16) | (imask << 24);
            h[4] = cbase;
            h[5] = tbase;
        }
        __syncwarp(); // the record is read and the node complete before it is written
        if (live)
            for (uint32_t v = c; v < C.node_bytes / 16u; v += 8u)
                reinterpret_cast<uint4 *>(rec)[v] = reinterpret_cast<const uint4 *>(buf)[v];
        if (leafslot) {
            uint32_t stack[4], at = tbase + toff;
            int sp = 0;
            stack[sp++] = ref;
            while (sp > 0) {
                const uint32_t y = stack[--sp];
                if (!(y & LEAF)) { // at most three leaves below: at most two on the stack
                    stack[sp++] = right_of(C.T, y);
                    stack[sp++] = left_of(C.T, y);
                    continue;
                }
                const uint32_t prim = C.T.order[y & ~LEAF];
                const float *v = C.verts + (size_t)prim * 9;
                float4 *t = C.tris + (size_t)at * 3;
                t[0] = make_float4(v[0], v[1], v[2], __uint_as_float(prim + C.prim_base));
                t[1] = make_float4(v[3], v[4], v[5], 0.0f);
                t[2] = make_float4(v[6], v[7], v[8], 0.0f);
                if (C.slot_nm) { // the normal as the shading forms it from the vertices
                    const v3 a = mk(v[0], v[1], v[2]);
                    const v3 nrm = normalize(cross(sub(mk(v[3], v[4], v[5]), a), sub(mk(v[6], v[7], v[8]), a)));
                    C.slot_nm[at] = make_float4(nrm.x, nrm.y, nrm.z, __uint_as_float(C.mat_idx[prim]));
                }
                ++at;
            }
        }
        __syncwarp(); // the group's buffer is free again
    }
}

inline uint32_t grid_for(uint64_t n, uint32_t threads, uint32_t cap = 152 * 32) {
    uint64_t g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (uint32_t)g;
}

// Where a build's scratch arrays come from: stream-ordered allocations for
// crg_scene_build, a fixed device array for crg_build_bvh_noalloc.  get()
// returns a 256-byte aligned block, or nullptr when none is available.
struct ScratchSource {
    virtual void *get(size_t bytes) = 0;
    virtual ~ScratchSource() = default;
};

// Scratch owned for the duration of one build (stream-ordered allocations).
struct AsyncScratch final : ScratchSource {
    cudaStream_t st;
    std::vector<void *> ptrs;
    cudaError_t err = cudaSuccess;
    explicit AsyncScratch(cudaStream_t s) : st(s) {}
    void *get(size_t bytes) override {
        void *p = nullptr;
        if (fault_injected()) {
            err = cudaErrorMemoryAllocation;
            return nullptr;
        }
        const cudaError_t e = cudaMallocAsync(&p, bytes + 16, st);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            err = e;
            return nullptr;
        }
        ptrs.push_back(p);
        return p;
    }
    ~AsyncScratch() override {
        for (void *p : ptrs) cudaFreeAsync(p, st);
    }
};

// One BVH of n triangles written into a region of a scene's node arrays.
struct BvhTarget {
    const float *verts;  // float[n*9], the BVH's triangles
    uint32_t n;
    float4 *nbox;        // binary nodes float4[2*max(1, n-1)]; nullptr = take them from the scratch
    uint32_t *order;     // uint32[n]: sorted primitive order (BVH-local indices)
    const uint32_t *mat_idx; // uint32[n]: material of each triangle (with slot_nm)
    float4 *slot_nm;     // normal and material per triangle slot; nullptr = not wanted
    uint8_t *wide;       // node array; this BVH's nodes start at node_base
    float4 *tris;        // triangle slot array; this BVH's slots start at slot_base
    uint32_t node_base, node_cap; // region of the node array reserved for this BVH
    uint32_t slot_base, prim_base;
};

struct BvhResult {
    uint32_t n_wide = 0, depth = 0;
    float sah = 0.0f;
};

// The build pipeline of this file's header comment, for one BVH.  Synchronises
// the stream once, or once more for every eight levels of an unusually deep tree.  On failure *msg names the failing step.
crg_status build_pipeline(const BvhTarget &t, const crg_build_opts &o, ScratchSource &src, cudaStream_t st,
                          BvhResult &res, std::string *msg) {
    const uint32_t n = t.n;
    res = BvhResult{};
    if (n == 0) return CRG_OK;
    const uint32_t nint = n >= 2 ? n - 1 : 1;
    const uint32_t node_bytes = ((24 + 7 * o.width) + 15) / 16 * 16;
    const uint32_t nblk = sort_blocks(n);
    auto fail = [&](crg_status s, const std::string &m) {
        if (msg) *msg = m;
        return s;
    };
    auto cuda_fail = [&](cudaError_t e, const char *what) {
        (void)cudaGetLastError();
        return fail(e == cudaErrorMemoryAllocation ? CRG_ERR_OOM : CRG_ERR_CUDA,
                    std::string(what) + ": " + cudaGetErrorString(e));
    };
#define BP_CHECK(call)                                                                                                 \
    do {                                                                                                               \
        const cudaError_t e_ = (call);                                                                                 \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call);                                                            \
    } while (0)
    auto take = [&](size_t bytes) { return src.get((bytes + 255) / 256 * 256); };
    float4 *tbox = (float4 *)take(sizeof(float4) * 2 * (size_t)n);
    float4 *lbox = (float4 *)take(sizeof(float4) * 2 * (size_t)n);
    float4 *nbox = t.nbox ? t.nbox : (float4 *)take(sizeof(float4) * 2 * (size_t)nint);
    uint32_t *cb = (uint32_t *)take(sizeof(uint32_t) * 8);
    uint32_t *k0 = (uint32_t *)take(sizeof(uint32_t) * n), *v0 = (uint32_t *)take(sizeof(uint32_t) * n);
    uint32_t *k1 = (uint32_t *)take(sizeof(uint32_t) * n), *v1 = (uint32_t *)take(sizeof(uint32_t) * n);
    uint32_t *hist = (uint32_t *)take(sizeof(uint32_t) * 256 * (size_t)nblk), *digit_sum = (uint32_t *)take(sizeof(uint32_t) * 256);
    uint32_t *parent = (uint32_t *)take(sizeof(uint32_t) * nint), *leaf_parent = (uint32_t *)take(sizeof(uint32_t) * n);
    uint32_t *count = (uint32_t *)take(sizeof(uint32_t) * nint), *visits = (uint32_t *)take(sizeof(uint32_t) * nint);
    float *cost = (float *)take(sizeof(float) * nint);
    uint32_t *lvl0 = (uint32_t *)take(sizeof(uint32_t) * (n + 1)), *lvl1 = (uint32_t *)take(sizeof(uint32_t) * (n + 1));
    uint32_t *nic = (uint32_t *)take(sizeof(uint32_t) * (n + 1));
    unsigned long long *bsum = (unsigned long long *)take(sizeof(unsigned long long) * kLevelBlocks);
    LevelState *lv = (LevelState *)take(sizeof(LevelState) * 2);
    if (!tbox || !lbox || !nbox || !cb || !k0 || !v0 || !k1 || !v1 || !hist || !digit_sum || !parent || !leaf_parent || !count ||
        !visits || !cost || !lvl0 || !lvl1 || !nic || !bsum || !lv)
        return fail(CRG_ERR_OOM, "BVH build: no room for the build's scratch arrays");

    // centroid bounds start at the identities of min / max
    BP_CHECK(cudaMemsetAsync(cb, 0xFF, 3 * sizeof(uint32_t), st));
    BP_CHECK(cudaMemsetAsync(cb + 3, 0x00, 3 * sizeof(uint32_t), st));
    const uint32_t T = 256;
    k_bounds<<<grid_for(n, T, 152 * 8), T, 0, st>>>(t.verts, n, tbox, cb);
    k_morton<<<grid_for(n, T), T, 0, st>>>(tbox, n, cb, k0, v0);
    // 4 passes: k0/v0 -> k1/v1 -> k0/v0 -> k1/v1 -> k0/v0: the sorted data ends in k0 / v0
    {
        uint32_t *ki = k0, *vi = v0, *ko = k1, *vo = v1;
        for (int pass = 0; pass < 4; ++pass) {
            if (n <= kSmallSort) k_hist<2><<<nblk, kSortThreads, 0, st>>>(ki, n, pass * 8, hist);
            else k_hist<16><<<nblk, kSortThreads, 0, st>>>(ki, n, pass * 8, hist);
            k_scan_rows<<<256, 256, 0, st>>>(hist, nblk, digit_sum);
            if (n <= kSmallSort) k_scatter<2><<<nblk, kSortThreads, 0, st>>>(ki, vi, n, pass * 8, hist, digit_sum, ko, vo);
            else k_scatter<16><<<nblk, kSortThreads, 0, st>>>(ki, vi, n, pass * 8, hist, digit_sum, ko, vo);
            std::swap(ki, ko);
            std::swap(vi, vo);
        }
        k_gather<<<grid_for(n, T), T, 0, st>>>(tbox, v0, n, t.order, lbox);
    }
    Tree Tr{lbox, t.order, nbox, parent, leaf_parent, count, cost};
    if (n >= 2) {
        k_karras<<<grid_for(n - 1, T), T, 0, st>>>(k0, (int)n, nbox, parent, leaf_parent);
        BP_CHECK(cudaMemsetAsync(visits, 0, sizeof(uint32_t) * nint, st));
        k_bottom_up<<<(n + kClimbLeaves - 1) / kClimbLeaves, kClimbLeaves, 0, st>>>(Tr, n, visits);
        if (o.treelet) {
            // a warp takes 32 leaves where that still makes as many warps as run at once, and down to two
            // where it does not: its treelets wait for one another, those of different warps do not.
            // Three rounds over 10,007 triangles and the rest of the build 574 us with 32 leaves, 540 with
            // 8, 511 with 2, 517 with 1; 33,282 triangles, two builds, 1.355 ms with 32, 1.300 with 4;
            // 163,282 triangles 1.71 ms with 32, 1.72 with 16, 1.76 with 8.  (152 SMs x 32 warps: the GPU that
            // this was measured on; any value gives the same tree.)
            uint32_t gamma = 7, per = 32;
            while (per > 2u && n / per < 152u * 32u) per /= 2u;
            for (uint32_t round = 0; round < o.treelet_rounds; ++round) {
                BP_CHECK(cudaMemsetAsync(visits, 0, sizeof(uint32_t) * nint, st));
                k_treelet<<<(n + per - 1) / per, 32, 0, st>>>(Tr, n, visits, gamma, per);
                gamma *= 2;
            }
            // every node's cost is its children's and its area's still: a node of at least gamma leaves
            // took it in the last round, a smaller one has not changed since
        }
    }
    BP_CHECK(cudaGetLastError());

    // collapse into the target region: levels are enqueued ahead without knowing their sizes (an
    // empty one costs two short launches); the tree is rarely more than three levels deeper than a
    // complete one of its width, and what is left then is found by reading the state back
    Collapse Cc{Tr, t.verts, t.mat_idx, t.slot_nm, t.wide + (size_t)t.node_base * node_bytes, t.tris, o.width, o.leaf_max,
                node_bytes, t.node_base, t.node_cap - t.node_base, t.slot_base, t.prim_base};
    k_collapse_start<<<1, 32, 0, st>>>(lvl0, lv, n >= 2 ? 0u : LEAF);
    uint32_t *cur = lvl0, *nxt = lvl1;
    uint32_t level = 0, ahead = 3;
    for (uint64_t full = 1; full < n; full *= o.width) ++ahead;
    LevelState h{};
    float c0 = 0.0f;
    float4 r[2] = {};
    uint64_t bound = 1; // most nodes the level can have
    for (;;) {
        for (uint32_t k = 0; k < ahead; ++k, ++level) {
            const uint32_t blocks = grid_for(bound, kLevelThreads / 8, kLevelBlocks);
            k_level_open<<<blocks, kLevelThreads, 0, st>>>(Cc, lv + (level & 1u), cur, nic, bsum);
            k_level_link<<<blocks, kLevelThreads, 0, st>>>(Cc, lv + (level & 1u), lv + ((level + 1) & 1u), nic, bsum, nxt);
            std::swap(cur, nxt);
            bound = std::min<uint64_t>(bound * o.width, n);
        }
        k_emit<<<grid_for(nint, kLevelThreads / 8, 152 * 8), kLevelThreads, 0, st>>>(Cc, lv + (level & 1u));
        BP_CHECK(cudaGetLastError());
        BP_CHECK(cudaMemcpyAsync(&h, lv + (level & 1u), sizeof(h), cudaMemcpyDeviceToHost, st));
        if (n >= 2) {
            BP_CHECK(cudaMemcpyAsync(&c0, cost, sizeof(float), cudaMemcpyDeviceToHost, st));
            BP_CHECK(cudaMemcpyAsync(r, nbox, sizeof(r), cudaMemcpyDeviceToHost, st));
        }
        BP_CHECK(cudaStreamSynchronize(st));
        BP_CHECK(cudaGetLastError());
        if (h.overflow) return fail(CRG_ERR_DEVICE, "wide BVH node count exceeded capacity");
        if (h.count == 0) break;
        ahead = 8;
    }
    if (h.tri_start != n) return fail(CRG_ERR_DEVICE, "wide BVH triangle count mismatch");
    res.n_wide = h.node_start;
    res.depth = h.depth;
    if (n >= 2) {
        const float dx = r[1].x - r[0].x, dy = r[1].y - r[0].y, dz = r[1].z - r[0].z;
        const float ra = 2.0f * ((dx * dy + dy * dz) + dz * dx);
        res.sah = ra > 0.0f ? c0 / ra : 0.0f;
    }
#undef BP_CHECK
    (void)node_bytes;
    return CRG_OK;
}

// Grows b to `bytes`, keeping its first `keep` bytes (device to device).
crg_status grow_keep(crg_context *ctx, DevBuf &b, size_t bytes, size_t keep, cudaStream_t st) {
    if (b.ptr && b.bytes >= bytes) return CRG_OK;
    DevBuf nb;
    crg_status rc = dev_alloc(ctx, nb, bytes);
    if (rc != CRG_OK) return rc;
    if (b.ptr && keep) {
        const cudaError_t e = cudaMemcpyAsync(nb.ptr, b.ptr, std::min(keep, b.bytes), cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess) (void)cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            dev_free(nb);
            return cuda_error(ctx, e, "cudaMemcpyAsync(grow)");
        }
    }
    dev_free(b);
    b = nb;
    return CRG_OK;
}

} // namespace

crg_status build_bvh(crg_scene *s, const crg_build_opts &o, cudaStream_t st) {
    crg_context *ctx = s->ctx;
    const bool same = s->opts.width == o.width && s->opts.treelet == o.treelet && s->opts.leaf_max == o.leaf_max &&
                      s->opts.treelet_rounds == o.treelet_rounds;
    if (!same)
        for (crg_model_rec &m : s->models) m.built = false;
    s->built = false;
    s->opts = o;
    s->width = o.width;
    s->node_bytes = ((24 + 7 * o.width) + 15) / 16 * 16;
    // node arrays: each model's region at node_base (fixed by the triangle counts)
    uint32_t cap = 0;
    for (const crg_model_rec &m : s->models) cap = std::max(cap, m.node_base + m.node_cap);
    const uint32_t old_cap = s->node_cap;
    const size_t keep_nodes = same ? old_cap : 0;
    crg_status rc;
    if (s->ntri > 0) {
        if ((rc = grow_keep(ctx, s->bvh2, sizeof(float4) * 2 * (size_t)cap, sizeof(float4) * 2 * keep_nodes, st)) != CRG_OK)
            return rc;
        if ((rc = grow_keep(ctx, s->wide, (size_t)s->node_bytes * cap, (size_t)s->node_bytes * keep_nodes, st)) != CRG_OK)
            return rc;
        size_t kept_prims = 0;
        for (const crg_model_rec &m : s->models)
            if (m.built) kept_prims = std::max<size_t>(kept_prims, (size_t)m.first + m.ntri);
        if ((rc = grow_keep(ctx, s->order, sizeof(uint32_t) * s->ntri, sizeof(uint32_t) * kept_prims, st)) != CRG_OK)
            return rc;
        if ((rc = grow_keep(ctx, s->tris, sizeof(float4) * 3 * s->ntri, sizeof(float4) * 3 * kept_prims, st)) != CRG_OK)
            return rc;
        if ((rc = grow_keep(ctx, s->slot_nm, sizeof(float4) * s->ntri, sizeof(float4) * kept_prims, st)) != CRG_OK)
            return rc;
        if (cap > old_cap || !same) // unused node slots read as zero (deterministic downloads)
            CRG_CUDA(ctx, cudaMemsetAsync((uint8_t *)s->wide.ptr + (size_t)s->node_bytes * keep_nodes, 0,
                                          (size_t)s->node_bytes * (cap - keep_nodes), st));
    }
    s->node_cap = cap;
    for (crg_model_rec &m : s->models) {
        if (m.built) continue;
        BvhTarget t{(const float *)s->verts.ptr + (size_t)m.first * 9,
                    m.ntri,
                    (float4 *)s->bvh2.ptr + 2 * (size_t)m.node_base,
                    (uint32_t *)s->order.ptr + m.first,
                    (const uint32_t *)s->mat_idx.ptr + m.first,
                    (float4 *)s->slot_nm.ptr,
                    (uint8_t *)s->wide.ptr,
                    (float4 *)s->tris.ptr,
                    m.node_base,
                    m.node_base + m.node_cap,
                    m.first,
                    m.first};
        AsyncScratch src(st);
        BvhResult res;
        std::string msg;
        rc = build_pipeline(t, o, src, st, res, &msg);
        if (rc != CRG_OK) {
            if (src.err != cudaSuccess) return cuda_error(ctx, src.err, "cudaMallocAsync(build scratch)");
            return set_error(ctx, rc, msg);
        }
        m.n_wide = res.n_wide;
        m.depth = res.depth;
        m.sah = res.sah;
        m.built = true;
    }
    // whole-scene figures: the single model's, or the sums / maxima over the models
    s->n_wide = 0;
    s->depth = 0;
    s->sah = 0.0f;
    for (const crg_model_rec &m : s->models) {
        s->depth = std::max(s->depth, m.depth);
        s->sah += m.sah;
    }
    s->n_wide = s->models.size() == 1 ? s->models[0].n_wide : cap;
    s->built = true;
    return CRG_OK;
}

} // namespace crg

// ----------------------------------------------------------------- build without allocation
// crg_build_bvh_noalloc: build_pipeline with its scratch carved from one
// file-scope __device__ array sized for CRG_NOALLOC_MAX_TRIS triangles; every
// GPU that loads this library holds it until the process exits.
namespace crg {
namespace {

constexpr size_t kNaN = CRG_NOALLOC_MAX_TRIS; // max triangles
constexpr size_t kNaBlk = sort_blocks(kNaN);
constexpr size_t na_round(size_t b) { return (b + 255) / 256 * 256; }
// the blocks build_pipeline takes for kNaN triangles, each rounded to 256 bytes
constexpr size_t kNaBytes = 3 * na_round(sizeof(float4) * 2 * kNaN) +    // triangle boxes in both orders, binary nodes
                            na_round(sizeof(uint32_t) * 8) +               // centroid bounds
                            4 * na_round(sizeof(uint32_t) * kNaN) +        // sort keys and values
                            na_round(sizeof(uint32_t) * 256 * kNaBlk) +    // digit histograms
                            5 * na_round(sizeof(uint32_t) * kNaN) +        // parent, leaf parent, count, visits, cost
                            3 * na_round(sizeof(uint32_t) * (kNaN + 1)) +  // collapse levels, children and triangles per node
                            na_round(sizeof(uint32_t) * 256) +             // digit sums
                            na_round(sizeof(unsigned long long) * kLevelBlocks) + // level sums by block
                            na_round(sizeof(LevelState) * 2);              // level state

__device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

// Device address of g_noalloc_scratch per device, fetched once with that
// device current (in host code the symbol's name is only a stand-in).
constexpr int kNaMaxDevices = 64;
unsigned char *g_noalloc_ptr[kNaMaxDevices] = {nullptr};
std::mutex g_noalloc_mutex;

crg_status noalloc_scratch(unsigned char **out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNaMaxDevices) {
        (void)cudaGetLastError();
        return CRG_ERR_CUDA;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
            (void)cudaGetLastError();
            return CRG_ERR_CUDA;
        }
        g_noalloc_ptr[dev] = (unsigned char *)p;
    }
    *out = g_noalloc_ptr[dev];
    return CRG_OK;
}

// Bump allocation over the fixed array; never more than kNaBytes.
struct FixedScratch final : ScratchSource {
    unsigned char *base;
    size_t used = 0;
    explicit FixedScratch(unsigned char *b) : base(b) {}
    void *get(size_t bytes) override {
        if (bytes > kNaBytes - used) return nullptr;
        void *p = base + used;
        used += bytes;
        return p;
    }
};

// Message of this thread's last failed crg_build_bvh_noalloc call.
thread_local std::string g_noalloc_error;

crg_status noalloc_fail(crg_status s, const std::string &m) {
    g_noalloc_error = m;
    return s;
}

} // namespace

void noalloc_prepare() {
    unsigned char *p = nullptr;
    (void)noalloc_scratch(&p);
}

} // namespace crg

extern "C" const char *crg_noalloc_last_error(void) { return crg::g_noalloc_error.c_str(); }

extern "C" crg_status crg_build_bvh_noalloc(const float *d_verts, uint32_t ntri, const crg_build_opts *opts,
                                            void *d_wide, size_t wide_bytes, float *d_tris, uint32_t *d_order,
                                            crg_bvh_info *info, crg_stream stream) {
    using namespace crg;
    g_noalloc_error.clear();
    crg_build_opts o{8, 0, 3, 3};
    if (opts) o = *opts;
    if (!((o.width == 2 || o.width == 4 || o.width == 8) && o.leaf_max >= 1 && o.leaf_max <= 3 && o.treelet_rounds <= 8))
        return noalloc_fail(CRG_ERR_INVALID_ARG, "build options: width 2/4/8, leaf_max 1..3, treelet_rounds <= 8");
    if (ntri > CRG_NOALLOC_MAX_TRIS)
        return noalloc_fail(CRG_ERR_INVALID_ARG, "more triangles than CRG_NOALLOC_MAX_TRIS");
    const uint32_t n = ntri;
    const uint32_t node_bytes = ((24 + 7 * o.width) + 15) / 16 * 16;
    const uint32_t nint = n >= 2 ? n - 1 : 1;
    if (n > 0 && (!d_verts || !d_wide || !d_tris || !d_order)) return noalloc_fail(CRG_ERR_INVALID_ARG, "null buffer");
    if (n > 0 && wide_bytes < (size_t)node_bytes * nint)
        return noalloc_fail(CRG_ERR_INVALID_ARG, "node buffer smaller than node_bytes * max(1, ntri - 1)");
    if (info) {
        *info = crg_bvh_info{};
        info->ntri = n;
        info->width = o.width;
        info->leaf_max = o.leaf_max;
        info->treelet = o.treelet;
        info->node_bytes = node_bytes;
        info->n_bvh2_nodes = n >= 2 ? n - 1 : 0;
        info->n_tri_slots = n;
    }
    if (n == 0) return CRG_OK;
    unsigned char *base = nullptr;
    if (noalloc_scratch(&base) != CRG_OK) return noalloc_fail(CRG_ERR_CUDA, "cudaGetSymbolAddress(scratch array) failed");
    // an error left pending by the caller's earlier work is not this call's
    (void)cudaGetLastError();
    cudaStream_t st = (cudaStream_t)stream;
    FixedScratch src(base);
    BvhTarget t{d_verts, n, nullptr, d_order, nullptr, nullptr, (uint8_t *)d_wide, (float4 *)d_tris, 0, nint, 0, 0};
    BvhResult res;
    std::string msg;
    const crg_status rc = build_pipeline(t, o, src, st, res, &msg);
    if (rc != CRG_OK) {
        // kernels queued before the failure may still use the shared array:
        // let them finish so the caller's next call does not race with them
        (void)cudaStreamSynchronize(st);
        (void)cudaGetLastError();
        return noalloc_fail(rc, msg);
    }
    if (info) {
        info->n_wide_nodes = res.n_wide;
        info->depth = res.depth;
        info->sah_cost = res.sah;
    }
    return CRG_OK;
}
