// Device BVH builder: the compressed 8-wide BVH of device/traverse.cuh built
// on the GPU, in place of the host's binned-SAH build.
//
// The reference used Metal's closed acceleration-structure builder
// (ShapeBuilder.swift:7-94,302-319; EntityBuilder.swift:148-165); its
// algorithm is unknown, so this is a new design:
//
//  1. Triangle boxes and the centroid bounds (one pass).
//  2. 63-bit Morton codes of the centroids (21 bits per axis), sorted with
//     the triangle indices by an LSD radix sort of 8-bit digits: per pass a
//     tile histogram, an exclusive scan of the (digit, tile) counts and a
//     stable scatter that ranks a tile's keys warp by warp with match.any.
//  3. A binary tree by parallel locally-ordered clustering (Meister and
//     Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
//     Hierarchy Construction", TVCG 2018): clusters in Morton order, each
//     finds the neighbour within 16 positions whose union box has the
//     smallest surface area; mutual nearest neighbours merge; the survivors
//     are compacted by a scan, and the loop repeats until one cluster is
//     left.  Equal costs are ordered by a symmetric hash of the pair, so
//     regular geometry (grids of equal triangles) still merges in parallel;
//     an iteration that merges fewer than 1/16 of the clusters is replaced
//     by merging Morton neighbours pairwise, which bounds the iteration count.
//     One cooperative launch runs all iterations.
//  4. The SAH-optimal collapse into 8-wide nodes, as the host builder makes
//     it (Ylitie, Karras and Laine 2017, section 3.1): when it is made (its
//     children were made in earlier iterations), every binary node gets the
//     least surface-area cost of its subtree as at most 1..8 slots of its
//     parent (a leaf of at most 3
//     triangles, an inner node, or a spread over several slots) and the
//     choices that reach it.  Then level by level from the root, each node
//     collects its slots from those choices, places the children in octant
//     slots and quantises their boxes; scans of the children and leaf
//     triangles per node place the next level's nodes and the triangles.  A
//     tree the optimal collapse would make deeper than the traversal stack is
//     collapsed again greedily (open the inner child of largest area until a
//     node has 8 children).
//
// Every kernel's indexes are bounded by its element count; the host reads the
// clustering's result and one 8-byte total per tree level.
#include "bvh_gpu.h"

#include <cooperative_groups.h>

#include <cfloat>
#include <cmath>
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "bvh_build.h"
#include "device/traverse.cuh"

namespace rmd {
namespace {

constexpr int kRadius = 16;          // clustering search window (each side), by default
constexpr int kMaxRadius = 64;
constexpr uint32_t kLeafTris = 3;    // subtrees of at most this many triangles are leaves
constexpr uint32_t kMaxWideLevels = 32;  // the traversal kernels' stack holds one group per level
constexpr int kScanItems = 4;        // per thread
constexpr int kScanThreads = 1024;
constexpr uint32_t kScanTile = kScanItems * kScanThreads;  // 4096
constexpr int kSortThreads = 256;    // 8 warps
constexpr int kSortRounds = 16;      // 32 keys per warp per round
constexpr uint32_t kSortTile = kSortThreads * kSortRounds;  // 4096 keys

// -------------------------------------------------------------------- scan
__device__ __forceinline__ uint2 operator+(uint2 a, uint2 b) { return make_uint2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ uint2 operator-(uint2 a, uint2 b) { return make_uint2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ uint32_t shflUp(uint32_t v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ uint2 shflUp(uint2 v, int d) {
    return make_uint2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}

// Inclusive scan of one value per thread over a block of kScanThreads;
// `total` = the block's sum.
template <class T>
__device__ T blockInclusiveScan(T v, T &total) {
    __shared__ T warpSums[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T u = shflUp(inc, d);
        if (lane >= d) inc = inc + u;
    }
    if (lane == 31) warpSums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        T wi = warpSums[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T u = shflUp(wi, d);
            if (lane >= d) wi = wi + u;
        }
        warpSums[lane] = wi;
    }
    __syncthreads();
    total = warpSums[kScanThreads / 32 - 1];
    if (warp > 0) inc = inc + warpSums[warp - 1];
    __syncthreads();
    return inc;
}

// Exclusive scan of kScanItems consecutive values per thread, in place in v;
// returns the block's sum.
template <class T>
__device__ T blockExclusiveScanItems(T (&v)[kScanItems]) {
    T sum = v[0];
#pragma unroll
    for (int k = 1; k < kScanItems; k++) sum = sum + v[k];
    T total;
    T run = blockInclusiveScan(sum, total) - sum;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const T x = v[k];
        v[k] = run;
        run = run + x;
    }
    return total;
}

// tile-wise exclusive scan of in into out; partials[b] = tile b's sum
template <class T>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const T *in, T *out, uint32_t m, T *partials) {
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    T v[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; k++) v[k] = base + k < m ? in[base + k] : T{};
    const T total = blockExclusiveScanItems(v);
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        if (base + k < m) out[base + k] = v[k];
    if (threadIdx.x == 0) partials[blockIdx.x] = total;
}

// in-place exclusive scan of at most kScanTile partials by one block; *total = their sum
template <class T>
__global__ void __launch_bounds__(kScanThreads) k_scan_partials(T *partials, uint32_t m, T *total) {
    const uint32_t base = threadIdx.x * kScanItems;
    T v[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; k++) v[k] = base + k < m ? partials[base + k] : T{};
    const T all = blockExclusiveScanItems(v);
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        if (base + k < m) partials[base + k] = v[k];
    if (threadIdx.x == 0) *total = all;
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) k_scan_add(T *out, uint32_t m, const T *partials) {
    const uint32_t base = blockIdx.x * kScanTile;
    const T p = partials[blockIdx.x];
    for (uint32_t k = threadIdx.x; k < kScanTile; k += kScanThreads)
        if (base + k < m) out[base + k] = out[base + k] + p;
}

// ------------------------------------------------------------- primitives
__device__ __forceinline__ uint32_t orderedBits(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float orderedFloat(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ float3 load3(const float *p, uint32_t i) {
    return make_float3(p[3 * (size_t)i], p[3 * (size_t)i + 1], p[3 * (size_t)i + 2]);
}

// triangle boxes (lo.w = 1: the leaf's triangle count) and the centroid bounds
__global__ void k_bvh_prims(const float *v0, const float *v1, const float *v2, uint32_t n, float4 *lo, float4 *hi,
                            uint32_t *centroidBounds) {
    float cmin[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, cmax[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float3 a = load3(v0, i), b = load3(v1, i), c = load3(v2, i);
        const float3 l = make_float3(fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)));
        const float3 h = make_float3(fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)));
        lo[i] = make_float4(l.x, l.y, l.z, __uint_as_float(1u));
        hi[i] = make_float4(h.x, h.y, h.z, 0.0f);
        const float cc[3] = {0.5f * (l.x + h.x), 0.5f * (l.y + h.y), 0.5f * (l.z + h.z)};
        for (int k = 0; k < 3; k++) {
            cmin[k] = fminf(cmin[k], cc[k]);
            cmax[k] = fmaxf(cmax[k], cc[k]);
        }
    }
    for (int k = 0; k < 3; k++) {
        for (int d = 16; d > 0; d >>= 1) {
            cmin[k] = fminf(cmin[k], __shfl_xor_sync(0xffffffffu, cmin[k], d));
            cmax[k] = fmaxf(cmax[k], __shfl_xor_sync(0xffffffffu, cmax[k], d));
        }
    }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 3; k++) {
            atomicMin(&centroidBounds[k], orderedBits(cmin[k]));
            atomicMax(&centroidBounds[3 + k], orderedBits(cmax[k]));
        }
}

// 21 bits spread to every third bit of 63
__device__ __forceinline__ uint64_t spread21(uint32_t x) {
    uint64_t v = x & 0x1fffffu;
    v = (v | (v << 32)) & 0x001f00000000ffffull;
    v = (v | (v << 16)) & 0x001f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

__global__ void k_bvh_morton(const float4 *lo, const float4 *hi, uint32_t n, const uint32_t *centroidBounds,
                             uint64_t *keys, uint32_t *vals) {
    float cmin[3], scale[3];
    for (int k = 0; k < 3; k++) {
        cmin[k] = orderedFloat(centroidBounds[k]);
        const float ext = orderedFloat(centroidBounds[3 + k]) - cmin[k];
        scale[k] = ext > 0.0f ? 2097152.0f / ext : 0.0f;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 l = lo[i], h = hi[i];
        const float c[3] = {0.5f * (l.x + h.x), 0.5f * (l.y + h.y), 0.5f * (l.z + h.z)};
        uint32_t q[3];
        for (int k = 0; k < 3; k++) {
            const float t = (c[k] - cmin[k]) * scale[k];
            q[k] = t <= 0.0f ? 0u : (t >= 2097151.0f ? 2097151u : (uint32_t)t);
        }
        keys[i] = (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
        vals[i] = i;
    }
}

// ------------------------------------------------------------- radix sort
// counts[d * tiles + tile] = keys of the tile whose digit is d
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const uint64_t *keys, uint32_t n, int shift,
                                                              uint32_t *counts, uint32_t tiles) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t base = blockIdx.x * kSortTile;
    for (uint32_t k = threadIdx.x; k < kSortTile; k += kSortThreads) {
        const uint32_t i = base + k;
        if (i < n) atomicAdd(&h[(uint32_t)(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    counts[threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of one tile: warp w ranks its 512 keys (16 rounds of 32, in
// order) by digit with match.any, the warps' digit counts are prefixed in
// shared memory, and offsets (the scanned counts) place the tile.
__global__ void __launch_bounds__(kSortThreads) k_radix_scatter(const uint64_t *keysIn, const uint32_t *valsIn,
                                                                 uint64_t *keysOut, uint32_t *valsOut, uint32_t n,
                                                                 int shift, const uint32_t *offsets, uint32_t tiles) {
    __shared__ uint32_t wh[kSortThreads / 32][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int w = 0; w < kSortThreads / 32; w++) wh[w][threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t chunk = blockIdx.x * kSortTile + (uint32_t)warp * (32u * kSortRounds);
    const uint32_t lt = (1u << lane) - 1u;
    uint64_t key[kSortRounds];
    uint32_t val[kSortRounds], dig[kSortRounds], rank[kSortRounds];
#pragma unroll
    for (int r = 0; r < kSortRounds; r++) {
        const uint32_t i = chunk + (uint32_t)r * 32u + (uint32_t)lane;
        const bool valid = i < n;
        key[r] = valid ? keysIn[i] : 0ull;
        val[r] = valid ? valsIn[i] : 0u;
        const uint32_t d = valid ? ((uint32_t)(key[r] >> shift) & 255u) : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = valid ? wh[warp][d] : 0u;
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wh[warp][d] += (uint32_t)__popc(peers);
        __syncwarp();
        dig[r] = d;
        rank[r] = before + (uint32_t)__popc(peers & lt);
    }
    __syncthreads();
    {  // exclusive prefix over the warps, per digit
        uint32_t run = 0u;
        for (int w = 0; w < kSortThreads / 32; w++) {
            const uint32_t c = wh[w][threadIdx.x];
            wh[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortRounds; r++) {
        if (dig[r] < 256u) {
            const uint32_t pos = offsets[dig[r] * tiles + blockIdx.x] + wh[warp][dig[r]] + rank[r];
            keysOut[pos] = key[r];
            valsOut[pos] = val[r];
        }
    }
}

// -------------------------------------------------------------- clustering
__device__ __forceinline__ float unionArea(float4 al, float4 ah, float4 bl, float4 bh) {
    const float ex = fmaxf(ah.x, bh.x) - fminf(al.x, bl.x);
    const float ey = fmaxf(ah.y, bh.y) - fminf(al.y, bl.y);
    const float ez = fmaxf(ah.z, bh.z) - fminf(al.z, bl.z);
    return ex * ey + ey * ez + ez * ex;  // half the surface area
}

// symmetric tie order of the pair (i, j)
__device__ __forceinline__ uint32_t pairHash(uint32_t i, uint32_t j) {
    uint32_t a = min(i, j), b = max(i, j);
    uint32_t h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    return h;
}

// leaves: node k = sorted triangle k
__global__ void k_bvh_leaves(const uint32_t *sortedTri, uint32_t n, const float4 *triLo, const float4 *triHi,
                             float4 *nodeLo, float4 *nodeHi, int2 *nodeChild, uint32_t *cl, float4 *clLo,
                             float4 *clHi) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t t = sortedTri[k];
        const float4 l = triLo[t], h = triHi[t];
        nodeLo[k] = l;
        nodeHi[k] = h;
        nodeChild[k] = make_int2(-1, (int)t);
        cl[k] = k;
        clLo[k] = l;
        clHi[k] = h;
    }
}

// ------------------------------------------------------- optimal collapse
// cost[8 i + s - 1]: the least cost of node i's subtree given as at most s
// slots of its parent (leaf slot: area * triangles; inner node: area + its
// subtree as 8 slots); choice[8 i]: 1 if i as one slot is a leaf; choice[8 i +
// s - 1], s > 1: 0 if s - 1 slots do as well, else the left child's slots;
// split[i]: the left child's slots when i is an inner node.  Ties favour
// more slots (a shallower tree).  The host builder's recurrence.
__device__ __forceinline__ float boxArea(float4 l, float4 h) {
    const float ex = h.x - l.x, ey = h.y - l.y, ez = h.z - l.z;
    if (ex < 0.0f) return 0.0f;
    return 2.0f * (ex * ey + ey * ez + ez * ex);
}

__global__ void k_dp_leaves(const float4 *lo, const float4 *hi, uint32_t n, float *cost, uint8_t *choice) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float leaf = boxArea(lo[i], hi[i]);  // one triangle
        for (int k = 0; k < 8; k++) {
            cost[8 * (size_t)i + k] = leaf;
            choice[8 * (size_t)i + k] = k == 0 ? 1 : 0;
        }
    }
}

// node i's costs and choices from its children's
__device__ void dpNode(size_t i, int2 ch, float4 l, float4 h, float *cost, uint8_t *choice, uint8_t *split) {
    const uint32_t tris = __float_as_uint(l.w);
    const float area = boxArea(l, h);
    const float leaf = tris <= kLeafTris ? area * (float)tris : FLT_MAX;
    float cl[8], cr[8];
    for (int k = 0; k < 8; k++) {
        cl[k] = cost[8 * (size_t)ch.x + k];
        cr[k] = cost[8 * (size_t)ch.y + k];
    }
    float dist[9];
    uint8_t distK[9];
    for (int s = 2; s <= 8; s++) {
        dist[s] = FLT_MAX;
        distK[s] = 1;
        for (int k = 1; k < s; k++) {
            const float v = cl[k - 1] + cr[s - k - 1];
            if (v < dist[s]) {
                dist[s] = v;
                distK[s] = (uint8_t)k;
            }
        }
    }
    const float inner = area + dist[8];
    split[i] = distK[8];
    float c = fminf(leaf, inner);
    cost[8 * i] = c;
    choice[8 * i] = tris <= kLeafTris && leaf <= inner ? 1 : 0;
    for (int s = 2; s <= 8; s++) {
        if (dist[s] <= c) {
            c = dist[s];
            choice[8 * i + s - 1] = distK[s];
        } else {
            choice[8 * i + s - 1] = 0;
        }
        cost[8 * i + s - 1] = c;
    }
}

// ------------------------------------------------------------- clustering
constexpr uint32_t kClusterThreads = 256;
constexpr uint32_t kClusterWarps = kClusterThreads / 32;
constexpr uint32_t kAlone = 512;           // clusters from which one block goes on alone
constexpr uint32_t kMaxClusterIterations = 4096;

struct ClusterArgs {
    uint32_t *cl[2];            // binary node of each cluster, in Morton order; double buffered
    float4 *clLo[2], *clHi[2];  // its box
    uint32_t *nn;               // the position each cluster would merge with
    float4 *nodeLo, *nodeHi;
    int2 *nodeChild;
    float *dpCost;
    uint8_t *dpChoice, *dpSplit;
    uint2 *blockTotals;         // per block: surviving clusters, merges
    uint32_t *result;           // root, iterations, whether it converged
    uint32_t n;
    int radius;
};

struct ClusterFate {
    bool survives, leads;  // a merge
};
__device__ __forceinline__ ClusterFate clusterFate(const uint32_t *nn, uint32_t i, uint32_t n, bool pairwise) {
    if (pairwise) return {(i & 1u) == 0u, (i & 1u) == 0u && i + 1u < n};
    const uint32_t j = nn[i];
    const bool mutual = nn[j] == i;
    return {!(mutual && i > j), mutual && i < j};
}

// The whole clustering in one cooperative launch.  Each iteration every block
// takes a contiguous run of the clusters: finds their nearest neighbours
// within `radius` positions, counts its survivors and merges, and, with the
// other blocks' counts, moves the survivors to their places in the next
// iteration's arrays and makes the merged nodes, costs and choices of the
// optimal collapse included (the children's are there since an earlier
// iteration); grid barriers stand between.  The last kAlone clusters, half of
// the iterations, are one block's work with block barriers.
//
// Bound by latency: 852 k triangles take 61 iterations, and as five launches,
// a three-kernel scan and an 8-byte read by the host each they cost 3.4 ms of
// which the kernels ran 1.9.
__global__ void __launch_bounds__(kClusterThreads) k_cluster(ClusterArgs A) {
    __shared__ float4 sLo[kClusterThreads + 2 * kMaxRadius], sHi[kClusterThreads + 2 * kMaxRadius];
    __shared__ uint2 sums[kClusterWarps];
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const int radius = A.radius;
    uint32_t clusters = A.n, nodeBase = A.n, iterations = 0;
    int c = 0;
    while (clusters > 1u && iterations < kMaxClusterIterations) {
        iterations++;
        const bool alone = clusters <= kAlone;
        if (alone && blockIdx.x != 0u) return;
        const uint32_t blocks = alone ? 1u : gridDim.x;
        const uint32_t per = ((clusters + blocks - 1u) / blocks + kClusterThreads - 1u) / kClusterThreads * kClusterThreads;
        const uint32_t begin = min(blockIdx.x * per, clusters), end = min(begin + per, clusters);
        uint32_t *cl = A.cl[c];
        float4 *lo = A.clLo[c], *hi = A.clHi[c];
        // nearest neighbour of each cluster within `radius` positions
        for (uint32_t base = begin; base < end; base += kClusterThreads) {
            for (uint32_t k = tid; k < kClusterThreads + 2u * radius; k += kClusterThreads) {
                const int64_t j = (int64_t)base - radius + k;
                if (j >= 0 && j < (int64_t)clusters) {
                    sLo[k] = lo[j];
                    sHi[k] = hi[j];
                }
            }
            __syncthreads();
            const uint32_t i = base + tid;
            if (i < end) {
                const float4 al = sLo[tid + radius], ah = sHi[tid + radius];
                uint64_t best = ~0ull;
                uint32_t bestJ = 0u;
                for (int d = -radius; d <= radius; d++) {
                    const int64_t j = (int64_t)i + d;
                    if (d == 0 || j < 0 || j >= (int64_t)clusters) continue;
                    const float a = unionArea(al, ah, sLo[tid + radius + d], sHi[tid + radius + d]);
                    // cost >= 0, so its bits order like the float; the hash orders ties
                    const uint64_t key = ((uint64_t)__float_as_uint(fmaxf(a, 0.0f)) << 32) | pairHash(i, (uint32_t)j);
                    if (key < best) {
                        best = key;
                        bestJ = (uint32_t)j;
                    }
                }
                A.nn[i] = bestJ;
            }
            __syncthreads();
        }
        if (alone) __syncthreads();
        else grid.sync();
        // this block's survivors and merges
        uint32_t survivors = 0, merges = 0;
        for (uint32_t i = begin + tid; i < end; i += kClusterThreads) {
            const ClusterFate f = clusterFate(A.nn, i, clusters, false);
            survivors += f.survives;
            merges += f.leads;
        }
        survivors = __reduce_add_sync(0xffffffffu, survivors);
        merges = __reduce_add_sync(0xffffffffu, merges);
        if (lane == 0u) sums[warp] = make_uint2(survivors, merges);
        __syncthreads();
        if (tid == 0u) {
            uint2 t = make_uint2(0u, 0u);
            for (uint32_t w = 0; w < kClusterWarps; w++) t = t + sums[w];
            A.blockTotals[blockIdx.x] = t;
        }
        if (alone) __syncthreads();
        else grid.sync();
        // all blocks' totals, and those before this one
        uint2 before = make_uint2(0u, 0u), total = make_uint2(0u, 0u);
        for (uint32_t k = lane; k < blocks; k += 32u) {  // every warp sums all of them
            const uint2 t = A.blockTotals[k];
            total = total + t;
            if (k < blockIdx.x) before = before + t;
        }
        total = make_uint2(__reduce_add_sync(0xffffffffu, total.x), __reduce_add_sync(0xffffffffu, total.y));
        before = make_uint2(__reduce_add_sync(0xffffffffu, before.x), __reduce_add_sync(0xffffffffu, before.y));
        // too few mutual pairs: merge neighbours pairwise
        const bool pairwise = total.y < max(1u, clusters / 16u);
        if (pairwise) {
            total = make_uint2((clusters + 1u) / 2u, clusters / 2u);
            before = make_uint2((begin + 1u) / 2u, begin / 2u);
        }
        // survivors to their places; leaders make the merged node
        uint32_t *clOut = A.cl[c ^ 1];
        float4 *loOut = A.clLo[c ^ 1], *hiOut = A.clHi[c ^ 1];
        for (uint32_t base = begin; base < end; base += kClusterThreads) {
            const uint32_t i = base + tid;
            ClusterFate f = {false, false};
            if (i < end) f = clusterFate(A.nn, i, clusters, pairwise);
            const uint32_t keep = __ballot_sync(0xffffffffu, f.survives), lead = __ballot_sync(0xffffffffu, f.leads);
            __syncthreads();  // the previous use of sums
            if (lane == 0u) sums[warp] = make_uint2(__popc(keep), __popc(lead));
            __syncthreads();
            uint2 at = before;
            for (uint32_t w = 0; w < kClusterWarps; w++) {
                if (w < warp) at = at + sums[w];
                before = before + sums[w];
            }
            if (f.survives) {
                const uint32_t below = (1u << lane) - 1u;
                const uint32_t p = at.x + __popc(keep & below);
                if (f.leads) {
                    const uint32_t j = pairwise ? i + 1u : A.nn[i];
                    const float4 al = lo[i], ah = hi[i], bl = lo[j], bh = hi[j];
                    const uint32_t count = __float_as_uint(al.w) + __float_as_uint(bl.w);
                    const float4 l = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), __uint_as_float(count));
                    const float4 h = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.0f);
                    const uint32_t id = nodeBase + at.y + __popc(lead & below);
                    const int2 ch = make_int2((int)cl[i], (int)cl[j]);
                    A.nodeLo[id] = l;
                    A.nodeHi[id] = h;
                    A.nodeChild[id] = ch;
                    clOut[p] = id;
                    loOut[p] = l;
                    hiOut[p] = h;
                    dpNode(id, ch, l, h, A.dpCost, A.dpChoice, A.dpSplit);
                } else {
                    clOut[p] = cl[i];
                    loOut[p] = lo[i];
                    hiOut[p] = hi[i];
                }
            }
        }
        if (alone) __syncthreads();
        else grid.sync();
        nodeBase += total.y;
        clusters = total.x;
        c ^= 1;
    }
    if (blockIdx.x == 0u && tid == 0u) {
        A.result[0] = A.cl[c][0];
        A.result[1] = iterations;
        A.result[2] = clusters <= 1u ? 1u : 0u;
    }
}

// ---------------------------------------------------------------- collapse
struct Tree {
    const float4 *lo, *hi;
    const int2 *child;
    const uint8_t *choice, *split;  // the optimal collapse's choices; null: the greedy collapse
    __device__ uint32_t count(int i) const { return __float_as_uint(lo[i].w); }
    __device__ bool leaf(int i) const { return child[i].x < 0 || count(i) <= kLeafTris; }
    // whether binary node i, as one slot of its parent, is a leaf
    __device__ bool leafSlot(int i) const { return choice ? choice[8 * (size_t)i] == 1 : leaf(i); }
    __device__ float area(int i) const {
        const float4 l = lo[i], h = hi[i];
        const float ex = h.x - l.x, ey = h.y - l.y, ez = h.z - l.z;
        if (ex < 0.0f) return 0.0f;
        return 2.0f * (ex * ey + ey * ez + ez * ex);
    }
};

// Children of one 8-wide node by slot (-1: empty) and its (inner children,
// leaf triangles); the same choices as the host's greedy collapse.
__global__ void k_collapse_plan(Tree t, const uint2 *entries, uint32_t m, int *slots, uint2 *counts) {
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e += gridDim.x * blockDim.x) {
        const int root = (int)entries[e].x;
        int kids[8];
        int nk = 0;
        if (entries[e].y == 0u && t.count(root) <= kLeafTris) {
            kids[nk++] = root;  // the whole scene is one leaf
        } else if (t.choice) {
            // the slots of the optimal collapse: (subtree, slots it may take), left child first
            int stNode[16], stSlots[16];
            int top = 0;
            const int k0 = t.split[root];
            stNode[top] = t.child[root].y, stSlots[top++] = 8 - k0;
            stNode[top] = t.child[root].x, stSlots[top++] = k0;
            while (top > 0 && nk < 8) {
                const int x = stNode[--top];
                int sl = stSlots[top];
                const bool binLeaf = t.child[x].x < 0;
                while (sl > 1 && !binLeaf && t.choice[8 * (size_t)x + sl - 1] == 0) sl--;
                if (sl == 1 || binLeaf) {
                    kids[nk++] = x;
                } else if (top + 2 <= 16) {
                    const int k = t.choice[8 * (size_t)x + sl - 1];
                    stNode[top] = t.child[x].y, stSlots[top++] = sl - k;
                    stNode[top] = t.child[x].x, stSlots[top++] = k;
                }
            }
        } else {
            kids[nk++] = t.child[root].x;
            kids[nk++] = t.child[root].y;
        }
        while (!t.choice && nk < 8) {
            int best = -1;
            float bestArea = -1.0f;
            for (int i = 0; i < nk; i++)
                if (!t.leaf(kids[i])) {
                    const float a = t.area(kids[i]);
                    if (a > bestArea) {
                        bestArea = a;
                        best = i;
                    }
                }
            if (best < 0) break;
            const int k = kids[best];
            kids[best] = t.child[k].x;
            kids[nk++] = t.child[k].y;
        }
        float nlo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, nhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (int i = 0; i < nk; i++) {
            const float4 l = t.lo[kids[i]], h = t.hi[kids[i]];
            nlo[0] = fminf(nlo[0], l.x); nlo[1] = fminf(nlo[1], l.y); nlo[2] = fminf(nlo[2], l.z);
            nhi[0] = fmaxf(nhi[0], h.x); nhi[1] = fmaxf(nhi[1], h.y); nhi[2] = fmaxf(nhi[2], h.z);
        }
        float centre[3];
        for (int k = 0; k < 3; k++) centre[k] = 0.5f * (nlo[k] + nhi[k]);
        float score[8][8];
        for (int i = 0; i < nk; i++) {
            const float4 l = t.lo[kids[i]], h = t.hi[kids[i]];
            const float off[3] = {0.5f * (l.x + h.x) - centre[0], 0.5f * (l.y + h.y) - centre[1],
                                  0.5f * (l.z + h.z) - centre[2]};
            for (int sl = 0; sl < 8; sl++) {
                float v = 0.0f;
                for (int k = 0; k < 3; k++) v += ((sl >> k) & 1) ? off[k] : -off[k];
                score[i][sl] = v;
            }
        }
        int slotKid[8] = {-1, -1, -1, -1, -1, -1, -1, -1};
        bool kidDone[8] = {false, false, false, false, false, false, false, false};
        for (int round = 0; round < nk; round++) {
            int bi = -1, bs = -1;
            float bv = -FLT_MAX;
            for (int i = 0; i < nk; i++) {
                if (kidDone[i]) continue;
                for (int sl = 0; sl < 8; sl++)
                    if (slotKid[sl] < 0 && score[i][sl] > bv) {
                        bv = score[i][sl];
                        bi = i;
                        bs = sl;
                    }
            }
            if (bi < 0) break;  // scores are finite for finite boxes; guards non-finite input
            kidDone[bi] = true;
            slotKid[bs] = bi;
        }
        uint32_t inner = 0u, tris = 0u;
        for (int sl = 0; sl < 8; sl++) {
            const int node = slotKid[sl] >= 0 ? kids[slotKid[sl]] : -1;
            slots[8 * (size_t)e + sl] = node;
            if (node < 0) continue;
            if (t.leafSlot(node)) tris += t.count(node);
            else inner++;
        }
        counts[e] = make_uint2(inner, tris);
    }
}

// quantised child bounds, conservative in float (the host's rule)
__device__ void quantise(const float *nlo, const float *nhi, const float4 *klo, const float4 *khi, const bool *used,
                         rmdhost::GpuWideNode &w) {
    for (int k = 0; k < 3; k++) {
        const float lo = nlo[k], extent = nhi[k] - nlo[k];
        int e = -100;
        if (extent > 0.0f) {
            int ex;
            frexpf(extent / 255.0f, &ex);
            e = ex;
            while (lo + 255.0f * ldexpf(1.0f, e) < nhi[k]) e++;
        }
        e = max(-126, min(127, e));
        const float scale = ldexpf(1.0f, e);
        w.origin[k] = lo;
        w.exponent[k] = (uint8_t)(e + 127);
        for (int c = 0; c < 8; c++) {
            if (!used[c]) {
                w.qlo[k][c] = 255;
                w.qhi[k][c] = 0;
                continue;
            }
            const float cl = k == 0 ? klo[c].x : (k == 1 ? klo[c].y : klo[c].z);
            const float ch = k == 0 ? khi[c].x : (k == 1 ? khi[c].y : khi[c].z);
            int ql = (int)floorf((cl - lo) / scale);
            int qh = (int)ceilf((ch - lo) / scale);
            ql = max(0, min(255, ql));
            qh = max(0, min(255, qh));
            while (ql > 0 && lo + (float)ql * scale > cl) ql--;
            while (qh < 255 && lo + (float)qh * scale < ch) qh++;
            w.qlo[k][c] = (uint8_t)ql;
            w.qhi[k][c] = (uint8_t)qh;
        }
    }
}

// Writes the level's nodes, their leaf triangles and the next level's entries.
__global__ void k_collapse_emit(Tree t, const uint2 *entries, uint32_t m, const int *slots, const uint2 *offsets,
                                uint32_t nodeBase, uint32_t triBase, const float *v0, const float *v1, const float *v2,
                                const uint32_t *inst, const uint32_t *prim, rmdhost::GpuWideNode *nodes,
                                float4 *tris, uint2 *next) {
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e += gridDim.x * blockDim.x) {
        int kid[8];
        bool used[8];
        float4 klo[8], khi[8];
        float nlo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, nhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (int sl = 0; sl < 8; sl++) {
            kid[sl] = slots[8 * (size_t)e + sl];
            used[sl] = kid[sl] >= 0;
            if (!used[sl]) continue;
            klo[sl] = t.lo[kid[sl]];
            khi[sl] = t.hi[kid[sl]];
            nlo[0] = fminf(nlo[0], klo[sl].x); nlo[1] = fminf(nlo[1], klo[sl].y); nlo[2] = fminf(nlo[2], klo[sl].z);
            nhi[0] = fmaxf(nhi[0], khi[sl].x); nhi[1] = fmaxf(nhi[1], khi[sl].y); nhi[2] = fmaxf(nhi[2], khi[sl].z);
        }
        rmdhost::GpuWideNode w;
        memset(&w, 0, sizeof(w));
        quantise(nlo, nhi, klo, khi, used, w);
        const uint2 off = offsets[e];
        w.childBase = nodeBase + off.x;
        w.triBase = triBase + off.y;
        uint32_t innerAt = 0u, triAt = 0u;
        for (int sl = 0; sl < 8; sl++) {
            if (!used[sl]) continue;
            const int node = kid[sl];
            if (!t.leafSlot(node)) {
                w.imask |= (uint8_t)(1u << sl);
                next[off.x + innerAt] = make_uint2((uint32_t)node, w.childBase + innerAt);
                innerAt++;
                continue;
            }
            const uint32_t c = t.count(node);
            w.meta[sl] = (uint8_t)((((1u << c) - 1u) << 5) | triAt);
            // the leaf's triangles, depth first (at most kLeafTris, so a short stack)
            int stack[8];
            int sp = 0;
            stack[sp++] = node;
            while (sp > 0) {
                const int x = stack[--sp];
                const int2 ch = t.child[x];
                if (ch.x < 0) {
                    const uint32_t tri = (uint32_t)ch.y;
                    float4 *o = &tris[TRI_FLOAT4 * ((size_t)w.triBase + triAt)];
                    const float3 a = load3(v0, tri), b = load3(v1, tri), cc = load3(v2, tri);
                    const float wa = __uint_as_float(inst[tri]), wb = __uint_as_float(prim[tri]);
                    // the three rotated copies that traversal reads (device/traverse.cuh)
                    o[0] = make_float4(a.y, a.z, a.x, wa);
                    o[1] = make_float4(b.y, b.z, b.x, wb);
                    o[2] = make_float4(cc.y, cc.z, cc.x, 0.0f);
                    o[3] = make_float4(a.z, a.x, a.y, wa);
                    o[4] = make_float4(b.z, b.x, b.y, wb);
                    o[5] = make_float4(cc.z, cc.x, cc.y, 0.0f);
                    o[6] = make_float4(a.x, a.y, a.z, wa);
                    o[7] = make_float4(b.x, b.y, b.z, wb);
                    o[8] = make_float4(cc.x, cc.y, cc.z, 0.0f);
                    triAt++;
                } else if (sp + 2 <= 8) {
                    stack[sp++] = ch.y;
                    stack[sp++] = ch.x;
                }
            }
        }
        nodes[entries[e].y] = w;
    }
}

// --------------------------------------------------------------- host side
// The builder's workspace: one allocation, carved into arrays on 256 bytes.
// (As 45 allocations it cost more than the build: 25 ms, and up to 125 ms in a
// process that had freed large blocks before.)
struct Workspace {
    cudaStream_t stream;
    char *base = nullptr;
    size_t used = 0;
    size_t allocated = 0;
    const rmdhost::DeviceMemory &memory;
    Workspace(cudaStream_t s, const rmdhost::DeviceMemory &m) : stream(s), memory(m) {}
    ~Workspace() {
        if (!base) return;
        cudaStreamSynchronize(stream);  // after an error its kernels may still run
        memory.free(base, allocated);
    }
    template <class T>
    T *take(size_t count) {  // null while only sizes are counted
        T *p = base ? reinterpret_cast<T *>(base + used) : nullptr;
        used += (std::max<size_t>(1, count) * sizeof(T) + 255) & ~size_t(255);
        return p;
    }
};

#define BVH_TRY(x)                               \
    do {                                         \
        const cudaError_t e_ = (x);              \
        if (e_ != cudaSuccess) return e_;        \
    } while (0)

int gridFor(uint32_t n, int threads) { return (int)std::max<uint32_t>(1, std::min<uint32_t>((n + threads - 1) / threads, 148u * 16u)); }

template <class T>
cudaError_t exclusiveScan(const T *in, T *out, uint32_t m, T *partials, T *total, cudaStream_t s) {
    const uint32_t tiles = std::max<uint32_t>(1, (m + kScanTile - 1) / kScanTile);
    if (tiles > kScanTile) return cudaErrorInvalidValue;
    k_scan_tiles<T><<<tiles, kScanThreads, 0, s>>>(in, out, m, partials);
    k_scan_partials<T><<<1, kScanThreads, 0, s>>>(partials, tiles, total);
    k_scan_add<T><<<tiles, kScanThreads, 0, s>>>(out, m, partials);
    return cudaGetLastError();
}

template <class T>
cudaError_t readTotal(const T *d, T &h, cudaStream_t s) {
    BVH_TRY(cudaMemcpyAsync(&h, d, sizeof(T), cudaMemcpyDeviceToHost, s));
    return cudaStreamSynchronize(s);
}

}  // namespace
}  // namespace rmd

namespace rmdhost {

using namespace rmd;

cudaError_t buildWideBvhGpu(const float *v0, const float *v1, const float *v2, const uint32_t *inst,
                            const uint32_t *prim, uint32_t n, cudaStream_t s, const DeviceMemory &memory, GpuBvhResult &out) {
    out = GpuBvhResult();
    if (n == 0) return cudaSuccess;  // no nodes: everything misses
    if (n > kGpuBvhMaxTriangles) {
        out.error = "the device BVH builder takes at most 2^24 triangles";
        return cudaErrorInvalidValue;
    }
    Workspace S(s, memory);
    float4 *triLo, *triHi, *nodeLo, *nodeHi, *clLo[2], *clHi[2];
    int2 *nodeChild;
    uint64_t *keys[2];
    uint32_t *vals[2], *centroidBounds, *counts, *offsets, *countPartials, *countTotal, *cl[2], *nn, *result;
    uint2 *blockTotals, *entries[2], *plan, *planPos, *pairPartials, *pairTotal;
    float *dpCost;
    uint8_t *dpChoice, *dpSplit;
    int *slots;
    GpuWideNode *wide;
    const uint32_t tiles = (n + kSortTile - 1) / kSortTile;
    const size_t nodes2 = 2 * (size_t)n;
    int device = 0, sms = 0, perSm = 0;
    BVH_TRY(cudaGetDevice(&device));
    BVH_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    BVH_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k_cluster, kClusterThreads, 0));
    const uint32_t clusterBlocks = std::min<uint32_t>((uint32_t)std::max(1, perSm * sms), (n + kClusterThreads - 1) / kClusterThreads);
    const auto carve = [&] {
        S.used = 0;
        triLo = S.take<float4>(n);
        triHi = S.take<float4>(n);
        nodeLo = S.take<float4>(nodes2);
        nodeHi = S.take<float4>(nodes2);
        nodeChild = S.take<int2>(nodes2);
        dpCost = S.take<float>(8 * nodes2);
        dpChoice = S.take<uint8_t>(8 * nodes2);
        dpSplit = S.take<uint8_t>(nodes2);
        for (int b = 0; b < 2; b++) {
            keys[b] = S.take<uint64_t>(n);
            vals[b] = S.take<uint32_t>(n);
            cl[b] = S.take<uint32_t>(n);
            clLo[b] = S.take<float4>(n);
            clHi[b] = S.take<float4>(n);
        }
        centroidBounds = S.take<uint32_t>(6);
        counts = S.take<uint32_t>(256 * (size_t)tiles);
        offsets = S.take<uint32_t>(256 * (size_t)tiles);
        countPartials = S.take<uint32_t>(kScanTile);
        countTotal = S.take<uint32_t>(1);
        nn = S.take<uint32_t>(n);
        blockTotals = S.take<uint2>(clusterBlocks);
        result = S.take<uint32_t>(3);
        pairPartials = S.take<uint2>(kScanTile);
        pairTotal = S.take<uint2>(1);
        wide = S.take<GpuWideNode>(n);
        entries[0] = S.take<uint2>(n);
        entries[1] = S.take<uint2>(n);
        slots = S.take<int>(8 * (size_t)n);
        plan = S.take<uint2>(n);
        planPos = S.take<uint2>(n);
    };
    carve();
    S.allocated = S.used;
    BVH_TRY(memory.alloc(reinterpret_cast<void **>(&S.base), S.allocated));
    carve();
    BVH_TRY(memory.alloc(&out.tris, (size_t)n * TRI_FLOAT4 * sizeof(float4)));
    float4 *tris = static_cast<float4 *>(out.tris);

    // 1. boxes and centroid bounds
    const uint32_t initBounds[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    BVH_TRY(cudaMemcpyAsync(centroidBounds, initBounds, sizeof(initBounds), cudaMemcpyHostToDevice, s));
    k_bvh_prims<<<gridFor(n, 256), 256, 0, s>>>(v0, v1, v2, n, triLo, triHi, centroidBounds);
    // 2. Morton codes, sorted with the triangle indices (8 passes of 8 bits)
    k_bvh_morton<<<gridFor(n, 256), 256, 0, s>>>(triLo, triHi, n, centroidBounds, keys[0], vals[0]);
    BVH_TRY(cudaGetLastError());
    int cur = 0;
    for (int shift = 0; shift < 64; shift += 8) {
        k_radix_hist<<<tiles, kSortThreads, 0, s>>>(keys[cur], n, shift, counts, tiles);
        BVH_TRY(exclusiveScan<uint32_t>(counts, offsets, 256u * tiles, countPartials, countTotal, s));
        k_radix_scatter<<<tiles, kSortThreads, 0, s>>>(keys[cur], vals[cur], keys[cur ^ 1], vals[cur ^ 1], n, shift,
                                                      offsets, tiles);
        BVH_TRY(cudaGetLastError());
        cur ^= 1;
    }
    // 3. clustering: leaves are nodes 0..n-1 (sorted order), merges n..2n-2
    k_bvh_leaves<<<gridFor(n, 256), 256, 0, s>>>(vals[cur], n, triLo, triHi, nodeLo, nodeHi, nodeChild, cl[0],
                                                 clLo[0], clHi[0]);
    BVH_TRY(cudaGetLastError());
    k_dp_leaves<<<gridFor(n, 256), 256, 0, s>>>(nodeLo, nodeHi, n, dpCost, dpChoice);
    BVH_TRY(cudaGetLastError());
    // search radius: RMD_BVH_RADIUS overrides the default (1..64)
    int radius = kRadius;
    if (const char *env = std::getenv("RMD_BVH_RADIUS")) radius = std::max(1, std::min(kMaxRadius, std::atoi(env)));
    ClusterArgs ca = {{cl[0], cl[1]}, {clLo[0], clLo[1]}, {clHi[0], clHi[1]}, nn, nodeLo, nodeHi, nodeChild, dpCost,
                      dpChoice, dpSplit, blockTotals, result, n, radius};
    void *args[] = {&ca};
    BVH_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_cluster), dim3(clusterBlocks), dim3(kClusterThreads), args, 0, s));
    uint32_t found[3];
    BVH_TRY(cudaMemcpyAsync(found, result, sizeof(found), cudaMemcpyDeviceToHost, s));
    BVH_TRY(cudaStreamSynchronize(s));
    if (!found[2]) {
        out.error = "device BVH clustering did not converge";
        return cudaErrorInvalidValue;
    }
    const uint32_t root = found[0];
    out.clusterIterations = found[1];

    // 4. collapse, level by level; at most n wide nodes (each has >= 2 triangles below it or is the root)
    const uint2 first = make_uint2(root, 0u);
    Tree t{nodeLo, nodeHi, nodeChild, dpChoice, dpSplit};
    uint32_t level = 0, width = 0, wideCount = 0, triCount = 0;
    int e = 0;
    for (bool restart = true; restart;) {  // the optimal collapse, or the greedy one if that is too deep
        restart = false;
        BVH_TRY(cudaMemcpyAsync(entries[0], &first, sizeof(first), cudaMemcpyHostToDevice, s));
        level = 0, width = 1, wideCount = 1, triCount = 0, e = 0;
    while (width > 0) {
        if (++level > kMaxWideLevels) {
            if (t.choice) {
                t.choice = t.split = nullptr;
                restart = true;
                break;
            }
            out.error = "device BVH deeper than the traversal stack (32 levels)";
            return cudaErrorInvalidValue;
        }
        k_collapse_plan<<<gridFor(width, 128), 128, 0, s>>>(t, entries[e], width, slots, plan);
        BVH_TRY(exclusiveScan<uint2>(plan, planPos, width, pairPartials, pairTotal, s));
        k_collapse_emit<<<gridFor(width, 128), 128, 0, s>>>(t, entries[e], width, slots, planPos, wideCount, triCount,
                                                            v0, v1, v2, inst, prim, wide, tris, entries[e ^ 1]);
        BVH_TRY(cudaGetLastError());
        uint2 total;
        BVH_TRY(readTotal(pairTotal, total, s));
        wideCount += total.x;
        triCount += total.y;
        width = total.x;
        e ^= 1;
        if (wideCount > n + 1) {
            out.error = "device BVH collapse produced more nodes than triangles";
            return cudaErrorInvalidValue;
        }
    }
    }
    if (triCount != n) {
        out.error = "device BVH collapse placed " + std::to_string(triCount) + " of " + std::to_string(n) +
                    " triangles";
        return cudaErrorInvalidValue;
    }
    BVH_TRY(memory.alloc(&out.nodes, (size_t)wideCount * sizeof(GpuWideNode)));
    out.nodeCount = wideCount;
    BVH_TRY(cudaMemcpyAsync(out.nodes, wide, (size_t)wideCount * sizeof(GpuWideNode), cudaMemcpyDeviceToDevice, s));
    out.levels = level;
    return cudaStreamSynchronize(s);
}

}  // namespace rmdhost
