// bvh_build.cu -- GPU LBVH build collapsed to the 8-wide compressed BVH.
//
// Replaces the driver-built bottom/top-level acceleration structures of the
// reference (ApplicationRT.cpp:186-258, XVKBLGeometry.cpp:8-38,
// XVKAccelerationStructure.cpp:15-96: one opaque BLAS per model, identity
// instances).  Steps, all on the context stream:
//   1. per-triangle bounds, scene centroid bounds (block reductions + atomics)
//   2. 63-bit Morton codes of the box centres (21 bits per axis)
//   3. stable LSD radix sort of (code, primitive) pairs, 8 passes of 8 bits (up to 2048
//      pairs: one block)
//   4. the binary tree: PLOC clustering (below), or with XR_BVH_BUILDER=lbvh and for
//      instances Karras, "Maximizing Parallelism in the Construction of BVHs, Octrees and
//      k-d Trees" (HPG 2012), whose radix tree splits equal codes by index and gets its
//      bounds bottom-up, the second arrival at a node computing its box
//   5. the SAH decisions of the collapse, bottom-up
//   6. top-down collapse, one level per launch, eight lanes per wide node: the children the
//      decisions give, children of <= 3 triangles become leaves, children and slots are paired
//      by how far the child's centre lies towards the slot's octant so that a ray visits near
//      children first, boxes are quantised to 8 bits (rounded outwards, plus the slack of
//      kBoxSlackCells).
// The kernels hand their counts on through device words (BuildWords); the host waits once
// per batch of clustering rounds and once per batch of levels.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "device_math.cuh"
#include "xr_internal.h"

namespace xr {
namespace {

constexpr uint32_t kLeafBit = 0x80000000u;
// Slack of the quantised child boxes, per side: the larger of kBoxSlackCells of the
// node's cell and one cell of the finest grid (2^emin >= 2^-17 of the largest
// coordinate).  The first covers the box test's own rounding (the plane constants
// of traversal are rounded at 32768 cells, 2^-9 of a cell, and the quantisation
// below adds 2^-16 of a cell); the second covers the watertight triangle
// test, whose hits can lie a few ulps of |v - o| (<= 2^-21 of the largest
// coordinate) outside the exact triangle.  The box test also widens every far t by
// a relative 2e-6, so a box is never rejected while it can hold a reported hit.
constexpr float kBoxSlackCells = 1.0f / 32.0f;

__device__ __forceinline__ uint32_t f2o(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float o2f(uint32_t u) {
    uint32_t v = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
#ifdef __CUDA_ARCH__
    return __uint_as_float(v);
#else
    float f;
    memcpy(&f, &v, 4);
    return f;
#endif
}

// Words of one build on the device: what the kernels share and the host reads back once.
constexpr uint32_t kMaxLevels = 200;               // wide levels of a tree
constexpr uint32_t kBuildLevels = kMaxLevels + 8;
struct BuildWords {
    uint32_t bounds[8];        // [0..2] centroid min, [3..5] centroid max (ordered), [6] largest |coordinate|
    uint32_t counters[4];      // [0] wide nodes, [1] triangle slots, [3] inconsistencies found
    uint32_t clusters[2];      // clusters left, by parity of the clustering round
    uint32_t made;             // binary nodes made by the clustering
    uint32_t stalled;          // a round of it has merged few clusters
    uint32_t root;             // root of the binary tree
    uint32_t level_count[kBuildLevels];   // wide nodes of each level
};

__global__ void k_build_init(BuildWords* w, uint32_t n, uint32_t root) {
    for (uint32_t i = threadIdx.x; i < sizeof(BuildWords) / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(w)[i] = 0u;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 0; k < 3; k++) w->bounds[k] = 0xFFFFFFFFu;
        w->counters[0] = 1u;
        w->clusters[0] = n;
        w->root = root;
        w->level_count[0] = 1u;
    }
}

// Primitive boxes: triangles from their vertices, or given boxes (box_lo non-null).  The
// bounds are reduced per block before the atomics: one set per warp serialised on seven
// addresses (1M triangles: 144 us; 152 x 4 blocks: 13 us).
constexpr int kPrepBlock = 256;
__global__ void __launch_bounds__(kPrepBlock) k_tri_prep(const uint4* __restrict__ tri_idx, const float4* __restrict__ vpos,
                                                         uint32_t ntri, const float4* __restrict__ box_lo,
                                                         const float4* __restrict__ box_hi, float4* __restrict__ tri_lo,
                                                         float4* __restrict__ tri_hi, uint32_t* __restrict__ bounds) {
    __shared__ float part[kPrepBlock / 32][7];
    float v[7] = {INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, 0.0f};   // min, -max, -(-amax)
    for (uint32_t t = blockIdx.x * kPrepBlock + threadIdx.x; t < ntri; t += gridDim.x * kPrepBlock) {
        float3 lo, hi;
        if (box_lo) {
            lo = xyz(box_lo[t]);
            hi = xyz(box_hi[t]);
        } else {
            uint4 id = tri_idx[t];
            float4 a = vpos[id.x], b = vpos[id.y], c = vpos[id.z];
            lo = f3(fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)));
            hi = f3(fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)));
        }
        tri_lo[t] = make_float4(lo.x, lo.y, lo.z, 0.0f);
        tri_hi[t] = make_float4(hi.x, hi.y, hi.z, 0.0f);
        const float c[3] = {(lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f};
        for (int k = 0; k < 3; k++) {
            v[k] = fminf(v[k], c[k]);
            v[3 + k] = fminf(v[3 + k], -c[k]);
        }
        const float amax = fmaxf(fmaxf(fmaxf(fabsf(lo.x), fabsf(lo.y)), fmaxf(fabsf(lo.z), fabsf(hi.x))),
                                 fmaxf(fabsf(hi.y), fabsf(hi.z)));
        v[6] = fminf(v[6], -amax);
    }
#pragma unroll
    for (int k = 0; k < 7; k++)
        for (int off = 16; off > 0; off >>= 1) v[k] = fminf(v[k], __shfl_xor_sync(0xFFFFFFFFu, v[k], off));
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 7; k++) part[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 7) {
        const int k = threadIdx.x;
        float m = part[0][k];
        for (int w = 1; w < kPrepBlock / 32; w++) m = fminf(m, part[w][k]);
        if (k == 6) atomicMax(&bounds[6], __float_as_uint(fabsf(m)));   // -m of +0 would be the largest word
        else if (m < INFINITY) {
            if (k < 3) atomicMin(&bounds[k], f2o(m));
            else atomicMax(&bounds[k], f2o(-m));
        }
    }
}

__device__ __forceinline__ uint64_t spread21(uint32_t v) {
    uint64_t x = v & 0x1FFFFFu;
    x = (x | (x << 32)) & 0x1F00000000FFFFull;
    x = (x | (x << 16)) & 0x1F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

__global__ void k_morton(const float4* __restrict__ tri_lo, const float4* __restrict__ tri_hi, uint32_t ntri,
                         const uint32_t* __restrict__ bounds, uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntri) return;
    float4 lo = tri_lo[t], hi = tri_hi[t];
    float c[3] = {(lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f};
    uint32_t q[3];
    for (int k = 0; k < 3; k++) {
        float mn = o2f(bounds[k]), mx = o2f(bounds[3 + k]);
        float ext = mx - mn;
        float u = ext > 0.0f ? (c[k] - mn) / ext : 0.5f;
        u = fminf(fmaxf(u, 0.0f), 1.0f);
        q[k] = min((uint32_t)(u * 2097152.0f), 2097151u);
    }
    keys[t] = spread21(q[0]) | (spread21(q[1]) << 1) | (spread21(q[2]) << 2);
    vals[t] = t;
}

// ---- stable LSD radix sort, 8 bits per pass ----
constexpr int kSortThreads = 256;

__global__ void k_sort_hist(const uint64_t* __restrict__ keys, uint32_t n, uint32_t chunk, int shift,
                            uint32_t* __restrict__ hist, uint32_t nblocks) {
    __shared__ uint32_t h[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    uint32_t b = blockIdx.x, beg = b * chunk, end = min(n, beg + chunk);
    for (uint32_t i = beg + threadIdx.x; i < end; i += blockDim.x)
        atomicAdd(&h[(uint32_t)(keys[i] >> shift) & 0xFFu], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i * nblocks + b] = h[i];
}

// Exclusive scan of each digit's row of block counts (one block per digit); the row's
// total goes to tot[digit], whose scan is left to the scatter (one block scanning all rows
// took 54 us a pass at 1M keys, this 5).
__global__ void __launch_bounds__(kSortThreads) k_sort_rows(uint32_t* __restrict__ hist, uint32_t* __restrict__ tot,
                                                            uint32_t nblocks) {
    __shared__ uint32_t wsum[kSortThreads / 32];
    uint32_t* row = hist + (size_t)blockIdx.x * nblocks;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t run = 0;
    for (uint32_t base = 0; base < nblocks; base += kSortThreads) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t v = i < nblocks ? row[i] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
            if ((int)lane >= d) x += y;
        }
        if (lane == 31u) wsum[warp] = x;
        __syncthreads();
        uint32_t before = run, all = 0;
        for (uint32_t w = 0; w < kSortThreads / 32; w++) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (i < nblocks) row[i] = before + x - v;
        run += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) tot[blockIdx.x] = run;
}

__global__ void __launch_bounds__(kSortThreads) k_sort_scatter(const uint64_t* __restrict__ kin,
                                                               const uint32_t* __restrict__ vin, uint64_t* __restrict__ kout,
                                                               uint32_t* __restrict__ vout, uint32_t n, uint32_t chunk, int shift,
                                                               const uint32_t* __restrict__ hist,
                                                               const uint32_t* __restrict__ tot, uint32_t nblocks) {
    __shared__ uint32_t base[256];
    __shared__ uint32_t wcnt[kSortThreads / 32][256];
    __shared__ uint32_t wsum[kSortThreads / 32];
    const uint32_t b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {   // thread d: where digit d starts, and in it this block's share
        const uint32_t v = tot[threadIdx.x];
        uint32_t x = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
            if ((int)lane >= d) x += y;
        }
        if (lane == 31u) wsum[warp] = x;
        __syncthreads();
        uint32_t before = 0;
        for (uint32_t w = 0; w < warp; w++) before += wsum[w];
        base[threadIdx.x] = before + x - v + hist[threadIdx.x * nblocks + b];
    }
    const uint32_t beg = b * chunk, end = min(n, beg + chunk);
    for (uint32_t tile = beg; tile < end; tile += kSortThreads) {
        for (int i = threadIdx.x; i < (kSortThreads / 32) * 256; i += blockDim.x) (&wcnt[0][0])[i] = 0;
        __syncthreads();
        uint32_t i = tile + threadIdx.x;
        bool valid = i < end;
        uint64_t key = valid ? kin[i] : 0ull;
        uint32_t val = valid ? vin[i] : 0u;
        uint32_t digit = valid ? ((uint32_t)(key >> shift) & 0xFFu) : 256u + lane;   // invalid lanes never match
        uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
        uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank == 0) wcnt[warp][digit] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t before = 0;
            for (uint32_t w = 0; w < warp; w++) before += wcnt[w][digit];
            uint32_t pos = base[digit] + before + rank;
            kout[pos] = key;
            vout[pos] = val;
        }
        __syncthreads();
        for (int d = threadIdx.x; d < 256; d += blockDim.x) {
            uint32_t tot = 0;
            for (int w = 0; w < kSortThreads / 32; w++) tot += wcnt[w][d];
            base[d] += tot;
        }
        __syncthreads();
    }
}

// Up to kSmallSort keys in one block (bitonic, ties by index like the stable radix sort):
// the top-level tree of a few hundred instances would otherwise spend 24 launches on it.
constexpr uint32_t kSmallSort = 2048;
__global__ void __launch_bounds__(1024) k_sort_small(uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n) {
    __shared__ uint64_t k[kSmallSort];
    __shared__ uint32_t v[kSmallSort];
    uint32_t size = 2;
    while (size < n) size <<= 1;
    for (uint32_t i = threadIdx.x; i < size; i += blockDim.x) {
        k[i] = i < n ? keys[i] : ~0ull;      // Morton codes have 63 bits
        v[i] = i;
    }
    __syncthreads();
    for (uint32_t span = 2; span <= size; span <<= 1)
        for (uint32_t step = span >> 1; step; step >>= 1) {
            for (uint32_t t = threadIdx.x; t < size / 2; t += blockDim.x) {
                const uint32_t a = 2u * t - (t & (step - 1u)), b = a + step;
                const uint64_t ka = k[a], kb = k[b];
                const uint32_t va = v[a], vb = v[b];
                const bool up = (a & span) == 0u, more = ka > kb || (ka == kb && va > vb);
                if (more == up) { k[a] = kb; k[b] = ka; v[a] = vb; v[b] = va; }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        keys[i] = k[i];
        vals[i] = v[i];
    }
}

// ---- Karras radix tree ----
__device__ __forceinline__ int delta(const uint64_t* keys, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    uint64_t a = keys[i], b = keys[j];
    if (a == b) return 64 + __clz((uint32_t)(i ^ j));
    return __clzll(a ^ b);
}

__global__ void k_karras(const uint64_t* __restrict__ keys, int n, uint32_t* __restrict__ left, uint32_t* __restrict__ right,
                         uint32_t* __restrict__ parent_int, uint32_t* __restrict__ parent_leaf,
                         uint32_t* __restrict__ count) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(keys, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int lo = min(i, j), hi = max(i, j);
    uint32_t lc = (lo == gamma) ? ((uint32_t)gamma | kLeafBit) : (uint32_t)gamma;
    uint32_t rc = (hi == gamma + 1) ? ((uint32_t)(gamma + 1) | kLeafBit) : (uint32_t)(gamma + 1);
    left[i] = lc;
    right[i] = rc;
    count[i] = (uint32_t)(hi - lo + 1);
    if (lc & kLeafBit) parent_leaf[lc & ~kLeafBit] = (uint32_t)i; else parent_int[lc] = (uint32_t)i;
    if (rc & kLeafBit) parent_leaf[rc & ~kLeafBit] = (uint32_t)i; else parent_int[rc] = (uint32_t)i;
}

__device__ __forceinline__ void ref_box(uint32_t ref, const float4* nlo, const float4* nhi, const float4* tlo,
                                        const float4* thi, const uint32_t* sorted, float4* lo, float4* hi) {
    if (ref & kLeafBit) {
        uint32_t p = sorted[ref & ~kLeafBit];
        *lo = tlo[p]; *hi = thi[p];
    } else {
        *lo = __ldcg(nlo + ref); *hi = __ldcg(nhi + ref);
    }
}

__global__ void k_bounds(int n, const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                         const uint32_t* __restrict__ parent_int, const uint32_t* __restrict__ parent_leaf,
                         const uint32_t* __restrict__ sorted, const float4* __restrict__ tlo, const float4* __restrict__ thi,
                         float4* nlo, float4* nhi, uint32_t* flags) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    uint32_t node = parent_leaf[j];
    // the radix tree of 64-bit keys split by 32-bit index is at most 96 levels deep
    for (int guard = 0; node != kInvalid; guard++) {
        if (guard > 128 || node >= (uint32_t)(n - 1)) { atomicOr(&flags[n - 1], 1u); return; }
        __threadfence();
        if (atomicAdd(&flags[node], 1u) == 0u) return;
        __threadfence();
        float4 al, ah, bl, bh;
        ref_box(left[node], nlo, nhi, tlo, thi, sorted, &al, &ah);
        ref_box(right[node], nlo, nhi, tlo, thi, sorted, &bl, &bh);
        __stcg(nlo + node, make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), 0.0f));
        __stcg(nhi + node, make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.0f));
        node = parent_int[node];
    }
}

struct CollapseArgs {
    const uint32_t* left; const uint32_t* right; const uint32_t* count;   // binary tree, primitives per node
    const float4* nlo; const float4* nhi; const float4* tlo; const float4* thi;
    const uint32_t* sorted;           // sorted primitive ids
    const uint4* tri_idx; const float4* vpos;
    const float4* records;            // non-null: leaves copy 4 float4 per primitive from here (instances)
    const uint8_t* dec;               // non-null: wide nodes follow the SAH decisions of k_sah_dp
    const uint32_t* ref_prim;         // non-null: primitives are triangle pieces; the triangle of each
    const uint32_t* task_in; const uint32_t* task_wide_in;
    uint32_t* task_out; uint32_t* task_wide_out;
    BuildWords* words;
    WideNode* nodes; float4* tris;
    int emin_floor;                   // lower bound of the finest grid exponent
    uint32_t max_nodes, n_prims;      // allocation bounds
};

__device__ __forceinline__ uint32_t ref_count(uint32_t ref, const uint32_t* count) {
    return (ref & kLeafBit) ? 1u : count[ref];
}
__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
    float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}
__device__ __forceinline__ int ceil_log2f(float v) {   // smallest e with 2^e >= v (v > 0)
    int e;
    float m = frexpf(v, &e);                           // v = m 2^e, m in [0.5, 1)
    return (m == 0.5f) ? e - 1 : e;
}

// ---- SAH-optimal collapse (Ylitie, Karras and Laine, HPG 2017, section 3.2) ----
// For every binary node n and every i in 1..8, cost(n, i) is the smallest SAH cost
// of representing n's subtree by at most i children of a wide node:
//   cost(n, 1) = min(leaf: A(n) ct count(n) if count(n) <= 3,
//                    wide node: A(n) cn + min_{j=2..8} D(n, j)),
//   cost(n, i) = min(cost(n, i - 1), D(n, i)),  D(n, i) = min_k cost(l, k) + cost(r, i - k);
// a primitive costs A ct for every i.  Computed bottom-up (the second thread to
// reach a node evaluates it); the decisions -- the best j with its split, and per i the
// split k (0: i - 1 children suffice) -- drive the top-down collapse.  A wide node's own
// subtree is always split: where every cost is 0 or infinite (primitives without area, or
// too large for it) no split is ever cheaper, and the node would be its own only child.
#ifndef XR_SAH_TRI
#define XR_SAH_TRI 1.2f
#endif
constexpr float kSahNode = 1.0f, kSahTri = XR_SAH_TRI;
constexpr uint32_t kDecStride = 16;   // bytes per binary node: [0] split of j*, [1] j*, [i] split of i (2..8)

__global__ void k_parents(uint32_t nint, const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                          uint32_t* __restrict__ parent_int, uint32_t* __restrict__ parent_leaf, const uint32_t* made) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nint || i >= *made) return;   // nodes a clustering without progress left out are not there
    const uint32_t lc = left[i], rc = right[i];
    if (lc & kLeafBit) parent_leaf[lc & ~kLeafBit] = i; else parent_int[lc] = i;
    if (rc & kLeafBit) parent_leaf[rc & ~kLeafBit] = i; else parent_int[rc] = i;
}

__device__ __forceinline__ void child_costs(uint32_t ref, const float* cost, const uint32_t* sorted, const float4* tlo,
                                            const float4* thi, float c[9]) {
    if (ref & kLeafBit) {
        const uint32_t p = sorted[ref & ~kLeafBit];
        const float4 lo = tlo[p], hi = thi[p];
        const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
        const float v = (dx * dy + dy * dz + dz * dx) * kSahTri;
        for (int i = 1; i <= 8; i++) c[i] = v;
    } else {
        const float4 a = __ldcg(reinterpret_cast<const float4*>(cost + 8u * (size_t)ref));
        const float4 b = __ldcg(reinterpret_cast<const float4*>(cost + 8u * (size_t)ref) + 1);
        c[1] = a.x; c[2] = a.y; c[3] = a.z; c[4] = a.w;
        c[5] = b.x; c[6] = b.y; c[7] = b.z; c[8] = b.w;
    }
}

__global__ void k_sah_dp(int n, const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                         const uint32_t* __restrict__ count, const uint32_t* __restrict__ parent_int,
                         const uint32_t* __restrict__ parent_leaf, const uint32_t* __restrict__ sorted,
                         const float4* __restrict__ tlo, const float4* __restrict__ thi, const float4* __restrict__ nlo,
                         const float4* __restrict__ nhi, float* cost, uint8_t* __restrict__ dec, uint32_t* flags) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    uint32_t node = parent_leaf[j];
    for (int guard = 0; node != kInvalid; guard++) {
        if (guard >= n || node >= (uint32_t)(n - 1)) { atomicOr(&flags[n - 1], 1u); return; }
        __threadfence();
        if (atomicAdd(&flags[node], 1u) == 0u) return;   // the sibling's thread evaluates it
        __threadfence();
        float cl[9], cr[9];
        child_costs(left[node], cost, sorted, tlo, thi, cl);
        child_costs(right[node], cost, sorted, tlo, thi, cr);
        float D[9];
        uint32_t ks[9];
#pragma unroll
        for (int i = 2; i <= 8; i++) {
            D[i] = INFINITY;
            ks[i] = 1u;
#pragma unroll
            for (int k = 1; k < i; k++) {
                const float v = cl[k] + cr[i - k];
                if (v < D[i]) { D[i] = v; ks[i] = (uint32_t)k; }
            }
        }
        uint32_t jstar = 2u, kstar = ks[2];
        float dbest = D[2];
#pragma unroll
        for (int i = 3; i <= 8; i++)
            if (D[i] < dbest) { dbest = D[i]; jstar = (uint32_t)i; kstar = ks[i]; }
        const float4 lo = __ldcg(nlo + node), hi = __ldcg(nhi + node);
        const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
        const float A = dx * dy + dy * dz + dz * dx;
        const uint32_t cnt = count[node];
        const float c_leaf = cnt <= 3u ? A * kSahTri * (float)cnt : INFINITY;
        const float c_int = A * kSahNode + dbest;
        // 16 decision bytes and 8 costs, each written as whole words
        uint32_t d[4] = {kstar | (jstar << 8), 0u, 0u, 0u};
        float c[9];
        c[1] = fminf(c_leaf, c_int);
#pragma unroll
        for (int i = 2; i <= 8; i++) {
            const bool less = D[i] < c[i - 1];
            c[i] = less ? D[i] : c[i - 1];
            if (less) d[i >> 2] |= ks[i] << (8 * (i & 3));
        }
        *reinterpret_cast<uint4*>(dec + (size_t)kDecStride * node) = make_uint4(d[0], d[1], d[2], d[3]);
        __stcg(reinterpret_cast<float4*>(cost + 8u * (size_t)node), make_float4(c[1], c[2], c[3], c[4]));
        __stcg(reinterpret_cast<float4*>(cost + 8u * (size_t)node) + 1, make_float4(c[5], c[6], c[7], c[8]));
        node = parent_int[node];
    }
}

// Quantisation grid of a node over its box: p = lo - one cell, cells of 2^e per
// axis with extent / 2^e <= 250 (at least 2^emin).
__device__ __forceinline__ void node_grid(float4 plo, float4 phi, int emin, float p3[3], int e[3]) {
    const float lo3[3] = {plo.x, plo.y, plo.z}, hi3[3] = {phi.x, phi.y, phi.z};
    for (int k = 0; k < 3; k++) {
        const float ext = hi3[k] - lo3[k];
        int ek = ext > 0.0f ? ceil_log2f(ext / 250.0f) : emin;
        ek = max(ek, emin);
        e[k] = ek;
        p3[k] = lo3[k] - ldexpf(1.0f, ek);
    }
}
// A child box on its parent's grid, rounded outwards plus the slack of kBoxSlackCells.
__device__ __forceinline__ void child_q(float4 clo, float4 chi, const float p3[3], const int e[3], int emin,
                                        uint8_t ql[3], uint8_t qh[3]) {
    const float cl[3] = {clo.x, clo.y, clo.z}, ch[3] = {chi.x, chi.y, chi.z};
    for (int k = 0; k < 3; k++) {
        const float inv = ldexpf(1.0f, -e[k]);
        const float slack = fmaxf(kBoxSlackCells, ldexpf(1.0f, emin - e[k]));
        const float l = floorf((cl[k] - p3[k]) * inv - slack);
        const float h = ceilf((ch[k] - p3[k]) * inv + slack);
        ql[k] = (uint8_t)fminf(fmaxf(l, 0.0f), 255.0f);
        qh[k] = (uint8_t)fminf(fmaxf(h, 0.0f), 255.0f);
    }
}
__device__ __forceinline__ void pack_q(const uint8_t ql[3][8], const uint8_t qh[3][8], uint32_t q[12]) {
    for (int k = 0; k < 3; k++) {
        q[2 * k] = ql[k][0] | (ql[k][1] << 8) | (ql[k][2] << 16) | ((uint32_t)ql[k][3] << 24);
        q[2 * k + 1] = ql[k][4] | (ql[k][5] << 8) | (ql[k][6] << 16) | ((uint32_t)ql[k][7] << 24);
        q[6 + 2 * k] = qh[k][0] | (qh[k][1] << 8) | (qh[k][2] << 16) | ((uint32_t)qh[k][3] << 24);
        q[6 + 2 * k + 1] = qh[k][4] | (qh[k][5] << 8) | (qh[k][6] << 16) | ((uint32_t)qh[k][7] << 24);
    }
}

// Finest grid exponent: cells of at least 2^-17 of the largest coordinate.
__host__ __device__ __forceinline__ int finest_exponent(float amax, int floor_e) {
    int e;
    frexpf(fmaxf(amax, 1e-20f), &e);
    e -= 17;
    return e > floor_e ? e : floor_e;
}

// Of *total, v for each calling lane (first lanes of groups of eight), with one atomic for
// those of a warp that call together: all nodes of a level add to the same words (the 20
// levels sent for 1M triangles 443 -> 400 us).
__device__ __forceinline__ uint32_t take_range(uint32_t* total, uint32_t v) {
    const uint32_t act = __activemask(), lane = threadIdx.x & 31u;
    uint32_t before = 0u, all = 0u;
    for (uint32_t l = 0; l < 32u; l += 8u) {
        if (!((act >> l) & 1u)) continue;
        const uint32_t x = __shfl_sync(act, v, (int)l);
        if (l < lane) before += x;
        all += x;
    }
    const int first = __ffs(act) - 1;
    uint32_t base = 0u;
    if ((int)lane == first && all) base = atomicAdd(total, all);
    return __shfl_sync(act, base, first) + before;
}

// One level of wide nodes, eight lanes per node, lane c holding child c (one thread per
// node left each level waiting ~70 us on that thread's chain of loads, whatever its size:
// 13 levels of the 1M-triangle scene took 0.96 ms, now 0.38).  What is left is that chain,
// shorter, for as many nodes as fit the SMs at a time (76 us for the widest level).  The level's node count is read
// on the device, so the host launches several levels without waiting for them.
__global__ void __launch_bounds__(128) k_collapse(CollapseArgs a, uint32_t level) {
    const uint32_t n_tasks = a.words->level_count[level];
    const uint32_t c = threadIdx.x & 7u, g0 = threadIdx.x & 24u;   // child, first lane of the group
    const uint32_t gm = 0xFFu << g0, upto = (2u << c) - 1u;
    const int emin = finest_exponent(__uint_as_float(a.words->bounds[6]), a.emin_floor);
    for (uint32_t task = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; task < n_tasks; task += (gridDim.x * blockDim.x) >> 3) {
        const uint32_t bref = level ? a.task_in[task] : a.words->root;
        const uint32_t widx = level ? a.task_wide_in[task] : 0u;
        uint32_t ref = kInvalid;
        if (bref & kLeafBit) {
            if (c == 0u) ref = bref;
        } else if (a.dec) {
            // The children the SAH decisions give, left to right: lane c may hold a subtree x
            // that takes the lanes c .. c + i - 1; splitting it sends its right part to lane
            // c + k.
            uint32_t x = bref, i = c == 0u ? a.dec[(size_t)kDecStride * bref + 1] : 0u;
            while (true) {
                const bool open = i > 1u && !(x & kLeafBit);
                uint32_t k = 0u, r = 0u, l = 0u;
                if (open) {
                    k = a.dec[(size_t)kDecStride * x + (x == bref ? 0u : i)];
                    l = a.left[x];
                    r = a.right[x];
                }
                const uint32_t holders = (__ballot_sync(gm, i > 0u) >> g0) & 0xFFu;
                if (!__any_sync(gm, open)) break;
                const uint32_t from = 31u - __clz(holders & upto);   // lane 0 always holds one
                const uint32_t fk = __shfl_sync(gm, k, g0 + from), fi = __shfl_sync(gm, i, g0 + from);
                const uint32_t fr = __shfl_sync(gm, r, g0 + from);
                if (open) {
                    if (k) { x = l; i = k; }
                    else i--;
                } else if (i == 0u && fk && from + fk == c) {
                    x = fr;
                    i = fi - fk;
                }
            }
            if (i) ref = x;
        } else {
            // greedy widening, the same in every lane of the group
            uint32_t refs[8];
            int nc = 0;
            refs[nc++] = a.left[bref];
            refs[nc++] = a.right[bref];
            while (nc < 8) {
                int best = -1;
                float best_area = -1.0f;
                for (int phase = 0; phase < 2 && best < 0; phase++) {
                    for (int j = 0; j < nc; j++) {
                        uint32_t r = refs[j];
                        if (r & kLeafBit) continue;
                        uint32_t cnt = ref_count(r, a.count);
                        if (phase == 0 ? cnt <= 3u : cnt > 3u) continue;
                        float ar = half_area(a.nlo[r], a.nhi[r]);
                        if (ar > best_area) { best_area = ar; best = j; }
                    }
                }
                if (best < 0) break;
                uint32_t r = refs[best];
                refs[best] = a.left[r];
                refs[nc++] = a.right[r];
            }
            if ((int)c < nc) ref = refs[c];
        }
        const bool there = ref != kInvalid;
        // boxes, parent box
        float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0), hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0);
        uint32_t cnt = 0u;
        if (there) {
            ref_box(ref, a.nlo, a.nhi, a.tlo, a.thi, a.sorted, &lo, &hi);
            cnt = ref_count(ref, a.count);
        }
        float4 plo = lo, phi = hi;
        for (int d = 1; d < 8; d <<= 1) {
            plo = make_float4(fminf(plo.x, __shfl_xor_sync(gm, plo.x, d)), fminf(plo.y, __shfl_xor_sync(gm, plo.y, d)),
                              fminf(plo.z, __shfl_xor_sync(gm, plo.z, d)), 0);
            phi = make_float4(fmaxf(phi.x, __shfl_xor_sync(gm, phi.x, d)), fmaxf(phi.y, __shfl_xor_sync(gm, phi.y, d)),
                              fmaxf(phi.z, __shfl_xor_sync(gm, phi.z, d)), 0);
        }
        // Slot assignment: of the pairs of child and free slot the one whose centre lies furthest
        // from the parent's towards the slot's corner, until every child has a slot (the greedy
        // form of the assignment of Ylitie, Karras and Laine, section 3.3).  The first child of an
        // octant taking its slot and the others the nearest free ones visits 0.5% more nodes for
        // random rays and costs camera paths over 1M triangles 1.4% of the frame.
        const float cx = (lo.x + hi.x) - (plo.x + phi.x), cy = (lo.y + hi.y) - (plo.y + phi.y), cz = (lo.z + hi.z) - (plo.z + phi.z);
        uint32_t slot = 8u, used = 0u;
        for (uint32_t left = __popc((__ballot_sync(gm, there) >> g0) & 0xFFu); left; left--) {
            float best = -INFINITY;
            uint32_t at = 8u;
            if (there && slot == 8u) {
                for (uint32_t t = 0; t < 8u; t++) {
                    // a sum that is not a number counts as the least: the pairs stay ordered
                    const float d = fmaxf(((t & 1u) ? cx : -cx) + ((t & 2u) ? cy : -cy) + ((t & 4u) ? cz : -cz), -3.402823466e+38f);
                    if (!((used >> t) & 1u) && (at == 8u || d > best)) { best = d; at = t; }
                }
            }
            // the group's best pair; ties go to the lowest lane
            uint32_t who = at < 8u ? c : 8u;
            float bd = best;
            for (int d = 1; d < 8; d <<= 1) {
                const float od = __shfl_xor_sync(gm, bd, d);
                const uint32_t ow = __shfl_xor_sync(gm, who, d);
                if (ow < 8u && (who == 8u || od > bd || (od == bd && ow < who))) { bd = od; who = ow; }
            }
            const uint32_t st = __shfl_sync(gm, at, g0 + (who & 7u));
            if (c == who) slot = st;
            used |= 1u << st;
        }
        // internal children and leaf triangle counts
        const bool internal = there && !(ref & kLeafBit) && cnt > 3u;
        const bool leaf = there && !internal;
        const uint32_t imask = __reduce_or_sync(gm, internal ? 1u << slot : 0u), n_int = __popc(imask);
        const uint32_t n_tris = __reduce_add_sync(gm, leaf ? cnt : 0u);
        uint32_t child_base = 0u, tri_base = 0u, task_base = 0u;
        if (c == 0u) {
            child_base = take_range(&a.words->counters[0], n_int);
            tri_base = take_range(&a.words->counters[1], n_tris);
        }
        child_base = __shfl_sync(gm, child_base, g0);
        tri_base = __shfl_sync(gm, tri_base, g0);
        if (child_base + n_int > a.max_nodes || tri_base + n_tris > a.n_prims) {
            if (c == 0u) atomicOr(&a.words->counters[3], 1u);   // inconsistent tree: reported by the host, nothing written
            continue;
        }
        if (c == 0u) task_base = take_range(&a.words->level_count[level + 1u], n_int);
        task_base = __shfl_sync(gm, task_base, g0);
        int e[3];
        float p3[3];
        node_grid(plo, phi, emin, p3, e);
        uint8_t ql[3] = {0, 0, 0}, qh[3] = {0, 0, 0};
        if (there) child_q(lo, hi, p3, e, emin, ql, qh);
        // leaf triangles in slot order
        const uint32_t children = (imask << 24) | __reduce_or_sync(gm, leaf ? ((1u << cnt) - 1u) << (3u * slot) : 0u);
        const uint32_t off = __popc(children & ((1u << (3u * slot)) - 1u));   // used by leaves (slot < 8)
        // the node: every lane's bytes at its slot
        const uint32_t sh = 8u * (slot & 3u);
        const bool w0 = there && slot < 4u, w1 = there && slot >= 4u;
        uint32_t q[12];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            q[2 * k] = __reduce_or_sync(gm, w0 ? (uint32_t)ql[k] << sh : 0u);
            q[2 * k + 1] = __reduce_or_sync(gm, w1 ? (uint32_t)ql[k] << sh : 0u);
            q[6 + 2 * k] = __reduce_or_sync(gm, w0 ? (uint32_t)qh[k] << sh : 0u);
            q[6 + 2 * k + 1] = __reduce_or_sync(gm, w1 ? (uint32_t)qh[k] << sh : 0u);
        }
        uint4* dst = reinterpret_cast<uint4*>(a.nodes + widx);
        WideNode cells;
        set_cells(cells, e);
        if (c == 0u)
            dst[0] = make_uint4(__float_as_uint(p3[0]), __float_as_uint(p3[1]), __float_as_uint(p3[2]), cells.cell_xy);
        else if (c == 1u) dst[1] = make_uint4(child_base, tri_base, children, cells.cell_z);
        else if (c == 2u) dst[2] = make_uint4(q[0], q[1], q[2], q[3]);
        else if (c == 3u) dst[3] = make_uint4(q[4], q[5], q[6], q[7]);
        else if (c == 4u) dst[4] = make_uint4(q[8], q[9], q[10], q[11]);
        if (internal) {
            const uint32_t rank = __popc(imask & ((1u << slot) - 1u));
            a.task_out[task_base + rank] = ref;
            a.task_wide_out[task_base + rank] = child_base + rank;
        } else if (leaf) {
            // the (at most 3) primitives of the subtree, left to right
            uint32_t prims[3], np = 0, dfs[4], dsp = 0;
            dfs[dsp++] = ref;
            while (dsp) {
                uint32_t x = dfs[--dsp];
                if (x & kLeafBit) {
                    if (np < 3u) prims[np] = a.sorted[x & ~kLeafBit];
                    np++;
                } else if (dsp + 2u <= 4u) {
                    dfs[dsp++] = a.right[x];
                    dfs[dsp++] = a.left[x];
                }
            }
            if (np != cnt) { atomicOr(&a.words->counters[3], 2u); cnt = min(np, 3u); }
            for (uint32_t j = 0; j < cnt; j++) {
                uint32_t prim = prims[j];
                if (a.records) {   // an instance record: world-to-object rows, {instance, root}
                    float4* rec = a.tris + 4u * (tri_base + off + j);
                    for (int w = 0; w < 4; w++) rec[w] = a.records[4u * prim + w];
                    continue;
                }
                if (a.ref_prim) prim = a.ref_prim[prim];
                uint4 id = a.tri_idx[prim];
                float4 v0 = a.vpos[id.x], v1 = a.vpos[id.y], v2 = a.vpos[id.z];
                float4* tri = a.tris + 3u * (tri_base + off + j);
                tri[0] = make_float4(v0.x, v0.y, v0.z, __uint_as_float(prim));
                tri[1] = make_float4(v1.x, v1.y, v1.z, 0.0f);
                tri[2] = make_float4(v2.x, v2.y, v2.z, 0.0f);
            }
        }
    }
}

// ---- refit: new vertex positions under the same topology ----
// Triangle slots [first, first + n) take their primitive's current vertex positions.
__global__ void k_refit_slots(float4* __restrict__ tris, uint32_t first, uint32_t n, const uint4* __restrict__ tri_idx,
                              const float4* __restrict__ vpos) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4* t = tris + 3u * ((size_t)first + i);
    const float w = t[0].w;
    const uint4 id = tri_idx[__float_as_uint(w)];
    const float4 v0 = vpos[id.x], v1 = vpos[id.y], v2 = vpos[id.z];
    t[0] = make_float4(v0.x, v0.y, v0.z, w);
    t[1] = make_float4(v1.x, v1.y, v1.z, 0.0f);
    t[2] = make_float4(v2.x, v2.y, v2.z, 0.0f);
}

// Nodes [first, first + n), one level, deepest level first: each child's exact box
// (a leaf child from its triangle slots, an internal child from the box the launch
// of the level below wrote), the node's box, then its grid and child boxes
// requantised as the build does; topology, slots and metadata are kept.
__global__ void k_refit_level(WideNode* __restrict__ nodes, uint32_t first, uint32_t n, const float4* __restrict__ tris,
                              float4* __restrict__ box_lo, float4* __restrict__ box_hi, int emin) {
    const uint32_t w = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= first + n) return;
    WideNode nd = nodes[w];
    const uint32_t imask = nd.children >> 24;
    float4 clo[8], chi[8];
    float4 plo = make_float4(INFINITY, INFINITY, INFINITY, 0), phi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0);
    uint32_t present = 0;
    for (int s = 0; s < 8; s++) {
        const uint32_t bits = (nd.children >> (3 * s)) & 7u;
        if (!((imask >> s) & 1u) && (bits == 0u)) continue;
        present |= 1u << s;
        if (imask & (1u << s)) {
            const uint32_t c = nd.child_base + __popc(imask & ((1u << s) - 1u));
            clo[s] = box_lo[c];
            chi[s] = box_hi[c];
        } else {
            float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0), hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0);
            const uint32_t off = __popc(nd.children & ((1u << (3 * s)) - 1u)), cnt = __popc(bits);
            for (uint32_t j = 0; j < cnt; j++)
                for (int v = 0; v < 3; v++) {
                    const float4 q = tris[3u * ((size_t)nd.tri_base + off + j) + v];
                    lo = make_float4(fminf(lo.x, q.x), fminf(lo.y, q.y), fminf(lo.z, q.z), 0);
                    hi = make_float4(fmaxf(hi.x, q.x), fmaxf(hi.y, q.y), fmaxf(hi.z, q.z), 0);
                }
            clo[s] = lo;
            chi[s] = hi;
        }
        plo = make_float4(fminf(plo.x, clo[s].x), fminf(plo.y, clo[s].y), fminf(plo.z, clo[s].z), 0);
        phi = make_float4(fmaxf(phi.x, chi[s].x), fmaxf(phi.y, chi[s].y), fmaxf(phi.z, chi[s].z), 0);
    }
    box_lo[w] = plo;
    box_hi[w] = phi;
    int e[3];
    float p3[3];
    node_grid(plo, phi, emin, p3, e);
    uint8_t ql[3][8], qh[3][8];
    for (int s = 0; s < 8; s++) {
        uint8_t cql[3] = {0, 0, 0}, cqh[3] = {0, 0, 0};
        if (present & (1u << s)) child_q(clo[s], chi[s], p3, e, emin, cql, cqh);
        for (int k = 0; k < 3; k++) { ql[k][s] = cql[k]; qh[k][s] = cqh[k]; }
    }
    nd.px = p3[0]; nd.py = p3[1]; nd.pz = p3[2];
    set_cells(nd, e);
    pack_q(ql, qh, nd.q);
    nodes[w] = nd;
}

// ---- early split clipping (Ernst and Greiner, "Early Split Clipping for Bounding
// Volume Hierarchies", RT 2007) ----
// A triangle whose box diagonal exceeds kEscMult times the mean is referenced by
// several pieces: its box is halved at the midpoint of the longest axis, the
// triangle clipped to each half (Sutherland-Hodgman against the one new plane; the
// crossing point of an edge is computed once per edge, so both halves share it),
// and halves larger than the threshold are split again, at most kEscMaxDepth
// times.  Each piece keeps the bounds of its clipped polygon; the BVH is built over
// the pieces and every leaf slot holds the whole triangle, so a ray meeting any
// piece tests the same triangle and finds the same hit.
#ifndef XR_ESC_MULT
#define XR_ESC_MULT 4.0f
#endif
constexpr float kEscMult = XR_ESC_MULT;
constexpr int kEscMaxDepth = 6;   // up to 64 pieces per triangle

struct EscPoly {
    float3 v[9];   // a triangle clipped by up to six axis-aligned planes
    int n;
};

__device__ __forceinline__ void esc_clip(const EscPoly& in, int axis, float c, bool below, EscPoly& out) {
    out.n = 0;
    for (int k = 0; k < in.n; k++) {
        const float3 a = in.v[k], b = in.v[k + 1 == in.n ? 0 : k + 1];
        const float da = sel3(a, axis) - c, db = sel3(b, axis) - c;
        const bool ina = below ? da <= 0.0f : da >= 0.0f;
        const bool inb = below ? db <= 0.0f : db >= 0.0f;
        if (ina && out.n < 9) out.v[out.n++] = a;
        if (ina != inb && (da != 0.0f && db != 0.0f) && out.n < 9) {
            const float t = da / (da - db);
            float3 q = a + (b - a) * t;
            if (axis == 0) q.x = c; else if (axis == 1) q.y = c; else q.z = c;
            out.v[out.n++] = q;
        }
    }
}

// Pieces of one triangle in a fixed depth-first order; EMIT writes them at `base`.
template <bool EMIT>
__device__ uint32_t esc_pieces(float3 v0, float3 v1, float3 v2, float thr, uint32_t prim, uint32_t base,
                               float4* __restrict__ rlo, float4* __restrict__ rhi, uint32_t* __restrict__ rprim) {
    EscPoly st[kEscMaxDepth + 2];
    int dep[kEscMaxDepth + 2];
    int sp = 0;
    st[0].v[0] = v0; st[0].v[1] = v1; st[0].v[2] = v2; st[0].n = 3;
    dep[0] = 0;
    sp = 1;
    uint32_t cnt = 0;
    while (sp > 0) {
        sp--;
        const EscPoly p = st[sp];
        const int d = dep[sp];
        float3 lo = p.v[0], hi = p.v[0];
        for (int k = 1; k < p.n; k++) {
            lo = f3(fminf(lo.x, p.v[k].x), fminf(lo.y, p.v[k].y), fminf(lo.z, p.v[k].z));
            hi = f3(fmaxf(hi.x, p.v[k].x), fmaxf(hi.y, p.v[k].y), fmaxf(hi.z, p.v[k].z));
        }
        const float3 e = hi - lo;
        if (d < kEscMaxDepth && length(e) > thr && sp + 2 <= kEscMaxDepth + 2) {
            const int axis = (e.x >= e.y && e.x >= e.z) ? 0 : (e.y >= e.z ? 1 : 2);
            const float c = 0.5f * (sel3(lo, axis) + sel3(hi, axis));
            EscPoly a, b;
            esc_clip(p, axis, c, true, a);
            esc_clip(p, axis, c, false, b);
            if (b.n >= 3) { st[sp] = b; dep[sp] = d + 1; sp++; }
            if (a.n >= 3) { st[sp] = a; dep[sp] = d + 1; sp++; }
        } else {
            if (EMIT) {
                rlo[base + cnt] = make_float4(lo.x, lo.y, lo.z, 0.0f);
                rhi[base + cnt] = make_float4(hi.x, hi.y, hi.z, 0.0f);
                rprim[base + cnt] = prim;
            }
            cnt++;
        }
    }
    return cnt;
}

__global__ void k_esc_diag(const uint4* __restrict__ tri_idx, const float4* __restrict__ vpos, uint32_t n,
                           double* __restrict__ sum) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    float d = 0.0f;
    if (t < n) {
        const uint4 id = tri_idx[t];
        const float4 a = vpos[id.x], b = vpos[id.y], c = vpos[id.z];
        const float ex = fmaxf(a.x, fmaxf(b.x, c.x)) - fminf(a.x, fminf(b.x, c.x));
        const float ey = fmaxf(a.y, fmaxf(b.y, c.y)) - fminf(a.y, fminf(b.y, c.y));
        const float ez = fmaxf(a.z, fmaxf(b.z, c.z)) - fminf(a.z, fminf(b.z, c.z));
        d = sqrtf(ex * ex + ey * ey + ez * ez);
    }
    for (int off = 16; off > 0; off >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, off);
    if ((threadIdx.x & 31) == 0 && d != 0.0f) atomicAdd(sum, (double)d);
}

template <bool EMIT>
__global__ void k_esc(const uint4* __restrict__ tri_idx, const float4* __restrict__ vpos, uint32_t n, float thr,
                      uint32_t* __restrict__ count, const uint32_t* __restrict__ offset, const uint32_t* __restrict__ sums,
                      float4* __restrict__ rlo, float4* __restrict__ rhi, uint32_t* __restrict__ rprim) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const uint4 id = tri_idx[t];
    const float3 a = xyz(vpos[id.x]), b = xyz(vpos[id.y]), c = xyz(vpos[id.z]);
    if (EMIT) esc_pieces<true>(a, b, c, thr, t, offset[t] + sums[t >> 10], rlo, rhi, rprim);
    else count[t] = esc_pieces<false>(a, b, c, thr, t, 0u, nullptr, nullptr, nullptr);
}

// ---- PLOC: Meister and Bittner, "Parallel Locally-Ordered Clustering for
// Bounding Volume Hierarchy Construction" (TVCG 2018).  Clusters stay in
// Morton order; each finds the cluster within +-kPlocRadius positions whose
// merged box has the smallest surface area, mutual pairs merge into a new
// internal node at the lower position, the array is compacted, and rounds repeat
// until one cluster is left.  Of equal areas the pairs go by their indices: the globally
// best pair is always mutual, so every round merges.  Boxes that coincide or stand in a
// regular row have so many equal areas that a round merges next to nothing (256 equal
// boxes: one pair a round, a chain of 255 nodes; a row of 256: 135 rounds).  From the first
// round on that merges few clusters (ploc_few) the partner (positions 2k and 2k + 1) comes
// first among equals, which keeps the best pair mutual and halves such boxes in a round;
// trees whose rounds never stall are those of the indices alone.
#ifndef XR_PLOC_RADIUS
#define XR_PLOC_RADIUS 64
#endif
constexpr int kPlocRadius = XR_PLOC_RADIUS;
constexpr int kPlocBlock = 256;       // k_ploc_nn: two clusters per thread
constexpr uint32_t kPlocWide = 1u << 16;   // up to this many: several lanes per cluster
constexpr uint32_t kPlocTail = 2048;  // clusters that one block takes to the end
// Few of n clusters merged in a round: boxes in random places lose about one in six, equal
// boxes one pair, a row of boxes or boxes inside one another one in 64.
__host__ __device__ __forceinline__ bool ploc_few(uint32_t n, uint32_t merged) {
    return n > 16u && merged < (n < 64u ? 2u : n / 32u);
}

// A cluster: {lo, reference}, {hi, primitives}.
__global__ void k_ploc_init(uint32_t n, const uint32_t* __restrict__ sorted, const float4* __restrict__ tlo,
                            const float4* __restrict__ thi, float4* __restrict__ clo, float4* __restrict__ chi) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t p = sorted[i];
    const float4 lo = tlo[p], hi = thi[p];
    clo[i] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(i | kLeafBit));
    chi[i] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(1u));
}

__device__ __forceinline__ float merged_area(float4 alo, float4 ahi, float4 blo, float4 bhi) {
    float dx = fmaxf(ahi.x, bhi.x) - fminf(alo.x, blo.x);
    float dy = fmaxf(ahi.y, bhi.y) - fminf(alo.y, blo.y);
    float dz = fmaxf(ahi.z, bhi.z) - fminf(alo.z, blo.z);
    return dx * dy + dy * dz + dz * dx;
}
// What stands for a position outside the array: its merged area is infinite, so it never wins.
__device__ __forceinline__ float4 nowhere(float s) { return make_float4(s * INFINITY, s * INFINITY, s * INFINITY, 0.0f); }

// Nearest neighbours.  Candidates are taken in ascending order with a strict comparison:
// of equal areas the lowest position wins, which orders pairs by area, lower index, upper
// index; once rounds have stalled the partner is taken before.  A thread searches for two
// adjacent clusters, so that each candidate read from shared memory serves two (reading it
// was the bound: 128 x 32 B per cluster); even and odd positions are stored apart, so that
// the threads' reads are consecutive.  SPLIT > 1:
// that many lanes share a pair's candidates, for counts that leave the chip idle and the
// search a serial chain (2048 .. 64K clusters: 10.5 us a round with one lane, 5.5 with 8).
template <int SPLIT>
__global__ void __launch_bounds__(kPlocBlock) k_ploc_nn(const uint32_t* n_ptr, const uint32_t* stalled,
                                                        const float4* __restrict__ clo, const float4* __restrict__ chi,
                                                        uint32_t* __restrict__ nn) {
    constexpr int R = kPlocRadius, kPairs = kPlocBlock / SPLIT, kHalf = kPairs + R;
    static_assert(R % 2 == 0, "even and odd candidates are stored apart");
    __shared__ float4 slo[2][kHalf], shi[2][kHalf];
    const int n = (int)*n_ptr;
    const int first = (int)blockIdx.x * 2 * kPairs;
    if (first >= n) return;
    for (int k = threadIdx.x; k < 2 * kHalf; k += kPlocBlock) {
        const int j = first - R + k;
        const bool in = j >= 0 && j < n;
        slo[k & 1][k >> 1] = in ? clo[j] : nowhere(-1.0f);
        shi[k & 1][k >> 1] = in ? chi[j] : nowhere(1.0f);
    }
    __syncthreads();
    const int t = threadIdx.x / SPLIT, i0 = first + 2 * t;
    const float4 alo = slo[0][t + R / 2], ahi = shi[0][t + R / 2], blo = slo[1][t + R / 2], bhi = shi[1][t + R / 2];
    float best0 = INFINITY, best1 = INFINITY;
    int m0 = 2 * R + 2, m1 = 2 * R + 2;   // candidate's place: twice the step plus the parity (none: beyond the last)
    if (*stalled) {
        const float a = merged_area(alo, ahi, blo, bhi);
        if (a < INFINITY) { best0 = best1 = a; m0 = R + 1; m1 = R; }
    }
    // positions i0 - R .. i0 + R + 1: the first is out of the second cluster's reach, the
    // last out of the first's, and neither is its own neighbour
    auto step = [&](int m, bool e0, bool e1, bool o0, bool o1) {
        const float4 elo = slo[0][t + m], ehi = shi[0][t + m];
        if (e0) { const float a = merged_area(alo, ahi, elo, ehi); if (a < best0) { best0 = a; m0 = 2 * m; } }
        if (e1) { const float a = merged_area(blo, bhi, elo, ehi); if (a < best1) { best1 = a; m1 = 2 * m; } }
        const float4 olo = slo[1][min(t + m, kHalf - 1)], ohi = shi[1][min(t + m, kHalf - 1)];
        if (o0) { const float a = merged_area(alo, ahi, olo, ohi); if (a < best0) { best0 = a; m0 = 2 * m + 1; } }
        if (o1) { const float a = merged_area(blo, bhi, olo, ohi); if (a < best1) { best1 = a; m1 = 2 * m + 1; } }
    };
    if (SPLIT == 1) {
        step(0, true, false, true, true);
#pragma unroll 4
        for (int m = 1; m < R / 2; m++) step(m, true, true, true, true);
        step(R / 2, false, true, true, false);
#pragma unroll 4
        for (int m = R / 2 + 1; m < R; m++) step(m, true, true, true, true);
        step(R, true, true, false, true);
    } else {
        for (int m = (int)threadIdx.x % SPLIT; m <= R; m += SPLIT) step(m, m != R / 2, m != 0, m != R, m != R / 2);
#pragma unroll
        for (int d = 1; d < SPLIT; d <<= 1) {
            const float a0 = __shfl_xor_sync(0xFFFFFFFFu, best0, d), a1 = __shfl_xor_sync(0xFFFFFFFFu, best1, d);
            const int p0 = __shfl_xor_sync(0xFFFFFFFFu, m0, d), p1 = __shfl_xor_sync(0xFFFFFFFFu, m1, d);
            if (a0 < best0 || (a0 == best0 && p0 < m0)) { best0 = a0; m0 = p0; }
            if (a1 < best1 || (a1 == best1 && p1 < m1)) { best1 = a1; m1 = p1; }
        }
        if (threadIdx.x % SPLIT) return;
    }
    if (i0 < n) nn[i0] = (uint32_t)(m0 > 2 * R + 1 ? i0 : i0 - R + m0);
    if (i0 + 1 < n) nn[i0 + 1] = (uint32_t)(m1 > 2 * R + 1 ? i0 + 1 : i0 - R + m1);
}

struct PlocTree {   // the binary tree being made
    uint32_t* left; uint32_t* right; uint32_t* count;
    float4* nlo; float4* nhi;
    uint32_t max_nodes;
};
// Node k over two clusters; returns the merged cluster in alo, ahi.
__device__ __forceinline__ void ploc_node(const PlocTree& T, uint32_t k, float4& alo, float4& ahi, float4 blo, float4 bhi) {
    const uint32_t cnt = __float_as_uint(ahi.w) + __float_as_uint(bhi.w);
    if (k < T.max_nodes) {
        T.left[k] = __float_as_uint(alo.w);
        T.right[k] = __float_as_uint(blo.w);
        T.count[k] = cnt;
    }
    alo = make_float4(fminf(alo.x, blo.x), fminf(alo.y, blo.y), fminf(alo.z, blo.z), __uint_as_float(k));
    ahi = make_float4(fmaxf(ahi.x, bhi.x), fmaxf(ahi.y, bhi.y), fmaxf(ahi.z, bhi.z), __uint_as_float(cnt));
    if (k < T.max_nodes) {
        T.nlo[k] = make_float4(alo.x, alo.y, alo.z, 0.0f);
        T.nhi[k] = make_float4(ahi.x, ahi.y, ahi.z, 0.0f);
    }
}

// Merges the mutual pairs of 1024 positions; the clusters that stay go to the start of the
// block's 1024 places of (olo, ohi), in order, and their number to sums[block].
__global__ void __launch_bounds__(1024) k_ploc_merge(const uint32_t* n_ptr, const uint32_t* __restrict__ nn,
                                                     const float4* __restrict__ clo, const float4* __restrict__ chi,
                                                     float4* __restrict__ olo, float4* __restrict__ ohi,
                                                     uint32_t* __restrict__ sums, uint32_t* made, PlocTree T) {
    __shared__ uint32_t wsum[32];
    const uint32_t n = *n_ptr, i = blockIdx.x * 1024u + threadIdx.x, lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    if (blockIdx.x * 1024u >= n) return;
    bool keep = false;
    float4 lo, hi;
    if (i < n) {
        const uint32_t j = n > 1u ? nn[i] : i;
        const bool mutual = j != i && nn[j] == i;
        keep = !(mutual && i > j);   // else merged into position j
        if (keep) {
            lo = clo[i];
            hi = chi[i];
            if (mutual) ploc_node(T, atomicAdd(made, 1u), lo, hi, clo[j], chi[j]);
        }
    }
    const uint32_t kept = __ballot_sync(0xFFFFFFFFu, keep);
    if (lane == 0u) wsum[w] = __popc(kept);
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (uint32_t v = 0; v < 32u; v++) {
        if (v < w) before += wsum[v];
        all += wsum[v];
    }
    if (keep) {
        const uint32_t at = blockIdx.x * 1024u + before + __popc(kept & ((1u << lane) - 1u));
        olo[at] = lo;
        ohi[at] = hi;
    }
    if (threadIdx.x == 0u) sums[blockIdx.x] = all;
}

// Closes the gaps between the blocks' clusters; each block adds up the counts before its own.
__global__ void __launch_bounds__(256) k_ploc_compact(const uint32_t* n_ptr, uint32_t* n_next, uint32_t* stalled,
                                                      const uint32_t* __restrict__ sums, const float4* __restrict__ olo,
                                                      const float4* __restrict__ ohi, float4* __restrict__ clo,
                                                      float4* __restrict__ chi) {
    __shared__ uint32_t wsum[8];
    const uint32_t nb = (*n_ptr + 1023u) / 1024u, b = blockIdx.x;
    if (b >= nb) return;
    uint32_t s = 0;
    for (uint32_t i = threadIdx.x; i < b; i += 256u) s += sums[i];
    s = __reduce_add_sync(0xFFFFFFFFu, s);
    if ((threadIdx.x & 31u) == 0u) wsum[threadIdx.x >> 5] = s;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < 8; w++) before += wsum[w];
    const uint32_t cnt = sums[b];
    for (uint32_t i = threadIdx.x; i < cnt; i += 256u) {
        clo[before + i] = olo[b * 1024u + i];
        chi[before + i] = ohi[b * 1024u + i];
    }
    if (b == nb - 1u && threadIdx.x == 0u) {
        *n_next = before + cnt;
        if (ploc_few(*n_ptr, *n_ptr - (before + cnt))) *stalled = 1u;
    }
}

// The last rounds, from at most kPlocTail clusters to one, in one block: at 1M primitives
// 45 of the 75 rounds have fewer, and three launches each would cost more than their work.
// As clusters get fewer, more lanes share the search of one.
constexpr size_t kPlocTailSmem = kPlocTail * (2 * sizeof(float4) + sizeof(uint32_t));
__global__ void __launch_bounds__(1024) k_ploc_tail(uint32_t* n_ptr, const float4* __restrict__ clo,
                                                    const float4* __restrict__ chi, BuildWords* words, PlocTree T,
                                                    bool may_stop) {
    extern __shared__ float4 tail_mem[];
    float4 *lo = tail_mem, *hi = tail_mem + kPlocTail;
    uint32_t* nn = reinterpret_cast<uint32_t*>(tail_mem + 2 * kPlocTail);
    __shared__ uint32_t wsum[32], made;
    const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5;
    uint32_t n = *n_ptr;
    if (n > kPlocTail) return;   // not the host's promise: `made` will not match
    for (uint32_t i = t; i < n; i += 1024u) { lo[i] = clo[i]; hi[i] = chi[i]; }
    if (t == 0u) made = words->made;
    bool stalled = words->stalled != 0u;   // the same in all threads
    __syncthreads();
    while (n > 1u) {
        uint32_t share = 1u;   // lanes per cluster
        while (share < 32u && n * share * 2u <= 1024u) share <<= 1;
        const uint32_t sub = t & (share - 1u);
        for (uint32_t base = 0; base < n; base += 1024u / share) {
            const uint32_t c = base + t / share;
            float best = INFINITY;
            uint32_t bj = kInvalid;
            if (c < n) {
                const float4 alo = lo[c], ahi = hi[c];
                if (stalled && (c ^ 1u) < n) {
                    const float a = merged_area(alo, ahi, lo[c ^ 1u], hi[c ^ 1u]);
                    if (a < best) { best = a; bj = c ^ 1u; }
                }
                const int end = min((int)c + kPlocRadius, (int)n - 1);
                int j = (int)c - kPlocRadius + (int)sub;
                if (j < 0) j += (-j + (int)share - 1) / (int)share * (int)share;
                for (; j <= end; j += (int)share) {
                    const float a = merged_area(alo, ahi, lo[j], hi[j]);
                    if (a < best && j != (int)c) { best = a; bj = (uint32_t)j; }
                }
            }
            for (uint32_t d = 1; d < share; d <<= 1) {
                const float oa = __shfl_xor_sync(0xFFFFFFFFu, best, d);
                const uint32_t oj = __shfl_xor_sync(0xFFFFFFFFu, bj, d);
                if (oa < best || (oa == best && oj < bj)) { best = oa; bj = oj; }
            }
            if (c < n && sub == 0u) nn[c] = bj == kInvalid ? c : bj;
        }
        __syncthreads();
        // merge and close the gaps, 1024 positions at a time: writes go at or before the
        // positions read in the same step, after all of its reads
        uint32_t out = 0u;
        for (uint32_t base = 0; base < n; base += 1024u) {
            const uint32_t i = base + t;
            bool keep = false;
            float4 al, ah;
            if (i < n) {
                const uint32_t j = nn[i];
                const bool mutual = j != i && nn[j] == i;
                keep = !(mutual && i > j);
                if (keep) {
                    al = lo[i];
                    ah = hi[i];
                    if (mutual) ploc_node(T, atomicAdd(&made, 1u), al, ah, lo[j], hi[j]);
                }
            }
            const uint32_t kept = __ballot_sync(0xFFFFFFFFu, keep);
            if (lane == 0u) wsum[w] = __popc(kept);
            __syncthreads();
            uint32_t before = 0, all = 0;
            for (uint32_t v = 0; v < 32u; v++) {
                if (v < w) before += wsum[v];
                all += wsum[v];
            }
            if (keep) {
                const uint32_t at = out + before + __popc(kept & ((1u << lane) - 1u));
                lo[at] = al;
                hi[at] = ah;
            }
            out += all;
            __syncthreads();
        }
        if (out == n) break;   // no progress (infinite areas): `made` will not match
        if (ploc_few(n, n - out)) {
            if (stalled && may_stop) break;   // the same
            stalled = true;
        }
        n = out;
    }
    if (t == 0u) {
        words->made = made;
        words->root = __float_as_uint(lo[0].w);
        *n_ptr = n;
    }
}

// exclusive scan in blocks of 1024 (block sums to `sums`)
__global__ void __launch_bounds__(1024) k_scan_local(const uint32_t* __restrict__ in, uint32_t n,
                                                     uint32_t* __restrict__ out, uint32_t* __restrict__ sums) {
    __shared__ uint32_t warp_sums[32];
    const uint32_t i = blockIdx.x * 1024u + threadIdx.x, lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t v = i < n ? in[i] : 0u;
    uint32_t x = v;
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if ((int)lane >= off) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t s = warp_sums[lane];
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, off);
            if ((int)lane >= off) s += y;
        }
        warp_sums[lane] = s;
    }
    __syncthreads();
    const uint32_t before = (w ? warp_sums[w - 1] : 0u) + x - v;
    if (i < n) out[i] = before;
    if (threadIdx.x == 1023) sums[blockIdx.x] = warp_sums[31];
}

// exclusive scan of the block sums (one block); sums[nb] receives the total
__global__ void k_scan_top(uint32_t* sums, uint32_t nb) {
    if (threadIdx.x != 0) return;
    uint32_t acc = 0;
    for (uint32_t b = 0; b < nb; b++) { uint32_t v = sums[b]; sums[b] = acc; acc += v; }
    sums[nb] = acc;
}

template <typename T>
xr_status dalloc(Context* ctx, T** p, size_t count) {
    return cuda_check(ctx, cudaMalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T)), "cudaMalloc (bvh)");
}
// Scratch of a build: stream-ordered allocations from the context's pool
// (rebuilding a top-level BVH every frame would otherwise spend a millisecond in
// cudaMalloc / cudaFree, each of which also waits for the device).
template <typename T>
xr_status salloc(Context* ctx, T** p, size_t count) {
    return pool_alloc(ctx, p, count, "bvh scratch");
}
inline void sfree(Context* ctx, void* p) { pool_free(ctx, p); }

}  // namespace

// `declined` non-null: a clustering that makes little progress or gives a tree deeper than
// B.max_depth sets it, and nothing is built.
static xr_status build_tree(Context* ctx, WideBuild& B, bool* declined) {
    cudaStream_t st = ctx->stream;
    const uint32_t n = B.n;
    const bool records = B.records != nullptr;
    const uint32_t slot_words = records ? 4u : 3u;
    B.nodes = nullptr; B.slots = nullptr;
    B.n_nodes = 0; B.n_slots = 0; B.depth = 0; B.emin = 0; B.ms = 0.0f;
    B.level_off.clear();
    if (n == 0) return XR_OK;

    cudaEvent_t e0, e1;
    cudaEventCreate(&e0); cudaEventCreate(&e1);
    cudaEventRecord(e0, st);

    float4 *tlo = nullptr, *thi = nullptr, *nlo = nullptr, *nhi = nullptr;
    uint64_t *k0 = nullptr, *k1 = nullptr;
    uint32_t *v0 = nullptr, *v1 = nullptr, *hist = nullptr;
    uint32_t *left = nullptr, *right = nullptr, *pint = nullptr, *pleaf = nullptr, *flags = nullptr;
    uint32_t* range = nullptr;   // primitives below each binary internal node
    uint32_t *ta = nullptr, *tb = nullptr, *wa = nullptr, *wb = nullptr;
    BuildWords* words = nullptr;
    WideNode* nodes_tmp = nullptr;
    float* sah_cost = nullptr;     // SAH collapse: 8 costs and kDecStride decision bytes per binary node
    uint8_t* sah_dec = nullptr;
    uint32_t* sah_flags = nullptr;
    // clustering: clusters, their next round's, nearest neighbours, block counts
    float4 *clo = nullptr, *chi = nullptr, *olo = nullptr, *ohi = nullptr;
    uint32_t *nn = nullptr, *sums = nullptr;
    void* scratch = nullptr;
    BuildWords back;
    xr_status s = XR_OK;
    const uint32_t nint = n > 1 ? n - 1 : 1;
    const uint32_t chunk = 1024;   // keys per sort block: 4096 left a third of the chip idle at 1M (54 + 28 + 11 us a pass with one block scanning, now 5 + 19 + 6)
    const uint32_t nblk = (n + chunk - 1) / chunk;
    const char* builder = getenv("XR_BVH_BUILDER");
    const bool use_lbvh = B.builder == 2 || (B.builder == 0 && builder && strcmp(builder, "lbvh") == 0);
    const bool ploc = n > 1 && !use_lbvh;
    const char* coll = getenv("XR_BVH_COLLAPSE");   // greedy: the area-greedy widening instead of the SAH decisions
    const bool sah = n > 1 && !(coll && strcmp(coll, "greedy") == 0);
    const uint32_t np = ploc ? n : 0u, nd = sah ? nint : 0u;
    {   // One stream-ordered allocation holds all scratch.  Mapping and returning it takes a
        // microsecond or more a megabyte, a fifth of a 1M-triangle build, so arrays share memory
        // where one's last use comes before the other's first, in stream order: sort and clustering
        // with what follows them, the costs of the SAH decisions with the collapse (328 -> 212 bytes
        // a primitive).
        struct Item { void** dst; size_t bytes; };
        std::vector<Item> items;
        auto add = [&](auto** dst, size_t count) { items.push_back({(void**)dst, count * sizeof(**dst)}); };
        // the offset behind the items added since the last call, laid out from `off`
        char* base = nullptr;
        auto place = [&](size_t off) {
            for (const Item& it : items) {
                if (base) *it.dst = base + off;
                off += (it.bytes + 255u) & ~size_t(255u);
            }
            items.clear();
            return off;
        };
        auto layout = [&]() {
            add(&tlo, n); add(&thi, n); add(&v0, n); add(&left, nint); add(&right, nint); add(&pint, nint); add(&pleaf, n);
            add(&flags, (size_t)nint + 1); add(&range, nint); add(&nlo, nint); add(&nhi, nint); add(&words, 1);
            const size_t all = place(0);
            add(&k0, n); add(&k1, n); add(&v1, n); add(&hist, 256 * ((size_t)nblk + 1));
            add(&clo, np); add(&chi, np); add(&olo, np); add(&ohi, np); add(&nn, np); add(&sums, np / 1024 + 1);
            const size_t tree = place(all);
            add(&sah_dec, kDecStride * (size_t)nd); add(&sah_flags, (size_t)nd + 1);
            const size_t decided = place(all);
            add(&sah_cost, 8 * (size_t)nd);
            const size_t deciding = place(decided);
            add(&ta, n); add(&tb, n); add(&wa, n); add(&wb, n); add(&nodes_tmp, nint);
            const size_t collapse = place(decided);
            return std::max(tree, std::max(deciding, collapse));
        };
        if ((s = pool_alloc_bytes(ctx, &scratch, layout(), "bvh scratch"))) goto done;
        base = (char*)scratch;
        layout();
    }
    if (!B.slots_into && (s = dalloc(ctx, &B.slots, (size_t)slot_words * n))) goto done;
    if (B.slots_into) B.slots = B.slots_into;
    {
        const uint32_t blocks = (n + 255) / 256;
        k_build_init<<<1, 256, 0, st>>>(words, n, n == 1 ? kLeafBit : 0u);
        k_tri_prep<<<std::min<uint32_t>((n + kPrepBlock - 1) / kPrepBlock, 4u * (uint32_t)ctx->sm_count), kPrepBlock, 0, st>>>(
            B.tri_idx, B.vpos, n, B.box_lo, B.box_hi, tlo, thi, words->bounds);
        k_morton<<<blocks, 256, 0, st>>>(tlo, thi, n, words->bounds, k0, v0);
        if (n <= kSmallSort) {
            k_sort_small<<<1, 1024, 0, st>>>(k0, v0, n);
        } else {
            uint32_t* tot = hist + 256 * (size_t)nblk;
            for (int pass = 0; pass < 8; pass++) {
                int shift = pass * 8;
                k_sort_hist<<<nblk, 256, 0, st>>>(k0, n, chunk, shift, hist, nblk);
                k_sort_rows<<<256, kSortThreads, 0, st>>>(hist, tot, nblk);
                k_sort_scatter<<<nblk, kSortThreads, 0, st>>>(k0, v0, k1, v1, n, chunk, shift, hist, tot, nblk);
                std::swap(k0, k1);
                std::swap(v0, v1);
            }
        }
        cudaMemsetAsync(pint, 0xFF, nint * 4, st);
        cudaMemsetAsync(pleaf, 0xFF, (size_t)n * 4, st);
        cudaMemsetAsync(flags, 0, (nint + 1) * 4, st);
        if (n > 1 && use_lbvh) {
            k_karras<<<(n - 1 + 255) / 256, 256, 0, st>>>(k0, (int)n, left, right, pint, pleaf, range);
            k_bounds<<<blocks, 256, 0, st>>>((int)n, left, right, pint, pleaf, v0, tlo, thi, nlo, nhi, flags);
        } else if (ploc) {
            const PlocTree T{left, right, range, nlo, nhi, nint};
            k_ploc_init<<<blocks, 256, 0, st>>>(n, v0, tlo, thi, clo, chi);
            // Rounds until one block can take the rest.  The kernels read the cluster count on
            // the device, so the host sends several rounds (a round keeps about five sixths)
            // with the count of the batch's start and waits once per batch.
            uint32_t cnt = n, side = 0;
            while (cnt > kPlocTail && !s) {
                uint32_t rounds = 1;
                for (uint32_t c = cnt; c > kPlocTail && rounds < 8; c -= c / 6) rounds++;
                for (uint32_t r = 0; r < rounds; r++, side ^= 1u) {
                    uint32_t *cur = &words->clusters[side], *next = &words->clusters[side ^ 1u];
                    if (cnt > kPlocWide)
                        k_ploc_nn<1><<<(cnt + 2 * kPlocBlock - 1) / (2 * kPlocBlock), kPlocBlock, 0, st>>>(cur, &words->stalled, clo, chi, nn);
                    else
                        k_ploc_nn<8><<<(cnt + kPlocBlock / 4 - 1) / (kPlocBlock / 4), kPlocBlock, 0, st>>>(cur, &words->stalled, clo, chi, nn);
                    k_ploc_merge<<<(cnt + 1023) / 1024, 1024, 0, st>>>(cur, nn, clo, chi, olo, ohi, sums, &words->made, T);
                    k_ploc_compact<<<(cnt + 1023) / 1024, 256, 0, st>>>(cur, next, &words->stalled, sums, olo, ohi, clo, chi);
                }
                uint32_t left_over = 0;
                cudaMemcpyAsync(&left_over, &words->clusters[side], 4, cudaMemcpyDeviceToHost, st);
                if ((s = cuda_check(ctx, cudaStreamSynchronize(st), "bvh: ploc"))) break;
                if (declined && ploc_few(cnt, cnt - left_over)) { *declined = true; goto done; }
                if (left_over >= cnt) s = fail(ctx, XR_ERR_STATE, "bvh: clustering made no progress");
                cnt = left_over;
            }
            if (s) goto done;
            if ((s = cuda_check(ctx, cudaFuncSetAttribute(k_ploc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                          (int)kPlocTailSmem), "bvh: ploc"))) goto done;
            k_ploc_tail<<<1, 1024, kPlocTailSmem, st>>>(&words->clusters[side], clo, chi, words, T,
                                                           declined != nullptr);
        }
        cudaMemsetAsync(sah_flags, 0, (nd + 1) * 4, st);
        if (sah) {
            if (!use_lbvh) k_parents<<<(nint + 255) / 256, 256, 0, st>>>(nint, left, right, pint, pleaf, &words->made);
            k_sah_dp<<<blocks, 256, 0, st>>>((int)n, left, right, range, pint, pleaf, v0, tlo, thi, nlo, nhi, sah_cost,
                                             sah_dec, sah_flags);
        }
        CollapseArgs ca;
        ca.left = left; ca.right = right; ca.count = range; ca.nlo = nlo; ca.nhi = nhi; ca.tlo = tlo; ca.thi = thi;
        ca.sorted = v0; ca.tri_idx = B.tri_idx; ca.vpos = B.vpos; ca.records = B.records;
        ca.dec = sah ? sah_dec : nullptr;
        ca.ref_prim = B.ref_prim;
        ca.words = words; ca.nodes = nodes_tmp; ca.tris = B.slots; ca.emin_floor = B.emin_floor;
        ca.max_nodes = nint; ca.n_prims = n;
        // Levels in batches: enough for a well-filled tree and a few more, then eight at a time.
        uint32_t level = 0, until = 5;
        for (uint32_t c = n; c > 1; c /= 8) until++;
        uint32_t bflag = 0, dflag = 0;
        while (true) {
            for (; level < until; level++) {
                // a level has at most 8 times the nodes of the one above
                const uint64_t most = level < 8 ? std::min<uint64_t>(1ull << (3 * level), nint) : nint;
                const uint32_t grid = (uint32_t)std::min<uint64_t>((most * 8 + 127) / 128, 16ull * (uint32_t)ctx->sm_count);
                ca.task_in = level & 1u ? tb : ta; ca.task_wide_in = level & 1u ? wb : wa;
                ca.task_out = level & 1u ? ta : tb; ca.task_wide_out = level & 1u ? wa : wb;
                k_collapse<<<grid, 128, 0, st>>>(ca, level);
            }
            cudaMemcpyAsync(&back, words, sizeof(back), cudaMemcpyDeviceToHost, st);
            cudaMemcpyAsync(&bflag, flags + nint, 4, cudaMemcpyDeviceToHost, st);
            cudaMemcpyAsync(&dflag, sah_flags + nd, 4, cudaMemcpyDeviceToHost, st);
            if ((s = cuda_check(ctx, cudaStreamSynchronize(st), "bvh: collapse"))) goto done;
            if (declined && ploc && (back.made != n - 1 || back.level_count[B.max_depth])) { *declined = true; goto done; }
            if (ploc && back.made != n - 1) {
                s = fail(ctx, XR_ERR_STATE, "bvh: clustering built the wrong number of nodes");
                goto done;
            }
            if (back.counters[3] || bflag || dflag) { s = fail(ctx, XR_ERR_STATE, "bvh: inconsistent radix tree"); goto done; }
            if (back.level_count[level] == 0u) break;
            if (level >= kMaxLevels) { s = fail(ctx, XR_ERR_OVERFLOW, "bvh: collapse did not terminate"); goto done; }
            until = std::min(level + 8u, kMaxLevels);
        }
        if (back.counters[1] != n) { s = fail(ctx, XR_ERR_STATE, "bvh: triangle slots do not match the primitive count"); goto done; }
        // the nodes each level allocated are the next level
        B.level_off.push_back(0u);
        uint32_t depth = 0;
        for (; back.level_count[depth]; depth++) B.level_off.push_back(B.level_off.back() + back.level_count[depth]);
        const uint32_t n_nodes = back.counters[0];
        if (B.nodes_into) B.nodes = B.nodes_into;
        else if ((s = dalloc(ctx, &B.nodes, n_nodes))) goto done;
        cudaMemcpyAsync(B.nodes, nodes_tmp, (size_t)n_nodes * sizeof(WideNode), cudaMemcpyDeviceToDevice, st);
        cudaEventRecord(e1, st);
        if ((s = cuda_check(ctx, cudaStreamSynchronize(st), "bvh: finish"))) goto done;
        float amax;
        memcpy(&amax, &back.bounds[6], 4);
        B.emin = finest_exponent(amax, B.emin_floor);
        B.n_nodes = n_nodes;
        B.n_slots = n;
        B.depth = depth;
        cudaEventElapsedTime(&B.ms, e0, e1);
    }
done:
    sfree(ctx, scratch);
    cudaEventDestroy(e0); cudaEventDestroy(e1);
    if (s != XR_OK || (declined && *declined)) {
        if (!B.slots_into) cudaFree(B.slots);
        if (!B.nodes_into) cudaFree(B.nodes);
        B.slots = nullptr; B.nodes = nullptr;
        B.level_off.clear();
    }
    return s;
}

xr_status build_wide(Context* ctx, WideBuild& B) {
    bool declined = false;
    xr_status s = build_tree(ctx, B, B.max_depth ? &declined : nullptr);
    if (!s && declined) {
        B.builder = 2;
        s = build_tree(ctx, B, nullptr);
    }
    return s;
}

xr_status build_bvh(Context* ctx) {
    NvtxRange nvtx_range("xr bvh build");
    if (ctx->d_nodes) { cudaFree(ctx->d_nodes); ctx->d_nodes = nullptr; }
    if (ctx->d_tris) { cudaFree(ctx->d_tris); ctx->d_tris = nullptr; }
    ctx->n_nodes = 0; ctx->n_tri_slots = 0; ctx->bvh_depth = 0;
    ctx->bvh_levels.clear();
    WideBuild wb;
    wb.n = ctx->ntri;
    wb.tri_idx = ctx->d_tri_idx;
    wb.vpos = ctx->d_vpos;
    float4 *rlo = nullptr, *rhi = nullptr;
    uint32_t *rprim = nullptr, *cnt = nullptr, *off = nullptr, *sums = nullptr;
    double* dsum = nullptr;
    xr_status s = XR_OK;
    // Off by default: on the benchmark scene the unsplit ground triangles sit near the
    // root, where almost every ray meets them first and gets an early closest t that
    // culls the rest; split into pieces deep in the tree they lose that role, and the
    // frame is slower (threshold 4 / 8 / 16 x the mean diagonal: 3.01 / 2.91 / 2.80 ms
    // against 2.68 ms), although triangle tests per camera ray drop from 4.7 to 3.4.
    const char* split_env = getenv("XR_BVH_SPLIT");
    const bool split = ctx->ntri > 1 && split_env && strcmp(split_env, "1") == 0;
    if (split) {
        // references: pieces of the large triangles, one box per piece
        const uint32_t n = ctx->ntri, nb = (n + 1023) / 1024;
        cudaStream_t st = ctx->stream;
        if ((s = salloc(ctx, &dsum, 1)) || (s = salloc(ctx, &cnt, n)) || (s = salloc(ctx, &off, n)) ||
            (s = salloc(ctx, &sums, nb + 1)))
            goto out;
        cudaMemsetAsync(dsum, 0, sizeof(double), st);
        k_esc_diag<<<(n + 255) / 256, 256, 0, st>>>(ctx->d_tri_idx, ctx->d_vpos, n, dsum);
        double total = 0.0;
        cudaMemcpyAsync(&total, dsum, sizeof(double), cudaMemcpyDeviceToHost, st);
        if ((s = cuda_check(ctx, cudaStreamSynchronize(st), "bvh: split threshold"))) goto out;
        const float thr = (float)(kEscMult * total / n);
        k_esc<false><<<(n + 127) / 128, 128, 0, st>>>(ctx->d_tri_idx, ctx->d_vpos, n, thr, cnt, nullptr, nullptr,
                                                       nullptr, nullptr, nullptr);
        k_scan_local<<<nb, 1024, 0, st>>>(cnt, n, off, sums);
        k_scan_top<<<1, 32, 0, st>>>(sums, nb);
        uint32_t nref = 0;
        cudaMemcpyAsync(&nref, sums + nb, 4, cudaMemcpyDeviceToHost, st);
        if ((s = cuda_check(ctx, cudaStreamSynchronize(st), "bvh: split count"))) goto out;
        if ((s = salloc(ctx, &rlo, nref)) || (s = salloc(ctx, &rhi, nref)) || (s = salloc(ctx, &rprim, nref))) goto out;
        k_esc<true><<<(n + 127) / 128, 128, 0, st>>>(ctx->d_tri_idx, ctx->d_vpos, n, thr, nullptr, off, sums, rlo, rhi,
                                                      rprim);
        wb.n = nref;
        wb.box_lo = rlo;
        wb.box_hi = rhi;
        wb.ref_prim = rprim;
    }
    s = build_wide(ctx, wb);
out:
    sfree(ctx, rlo); sfree(ctx, rhi); sfree(ctx, rprim); sfree(ctx, cnt);
    sfree(ctx, off); sfree(ctx, sums); sfree(ctx, dsum);
    // a scene build is a one-off: hand its scratch back to the device, but for what stages
    // the arrays of host calls (a pool grown again by the first 1000-ray query: 253 us, not 170)
    cudaStreamSynchronize(ctx->stream);
    cudaMemPoolTrimTo(ctx->pool, kStagePooled);
    if (s) return s;
    ctx->d_nodes = wb.nodes;
    ctx->d_tris = wb.slots;
    ctx->n_nodes = wb.n_nodes;
    ctx->n_tri_slots = wb.n_slots;
    ctx->bvh_depth = wb.depth;
    ctx->bvh_levels = wb.level_off;
    ctx->bvh_emin = wb.emin;
    ctx->ms_bvh = wb.ms;
    ctx->bvh_ready = true;
    return XR_OK;
}

void launch_refit_slots(float4* tris, uint32_t first, uint32_t n, const uint4* tri_idx, const float4* vpos,
                        cudaStream_t st) {
    if (n) k_refit_slots<<<(n + 255) / 256, 256, 0, st>>>(tris, first, n, tri_idx, vpos);
}
void launch_refit_level(WideNode* nodes, uint32_t first, uint32_t n, const float4* tris, float4* box_lo,
                        float4* box_hi, int emin, cudaStream_t st) {
    if (n) k_refit_level<<<(n + 127) / 128, 128, 0, st>>>(nodes, first, n, tris, box_lo, box_hi, emin);
}

}  // namespace xr
