// Static sm_100a kernels of the wavefront: closest-hit and shadow traversal,
// film accumulation + path regeneration, frame set-up, the environment-map
// pyramid reductions, film read-out, and small test hooks.  The shading
// megakernel lives in the NVRTC module (device/integrator.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "device/traverse.cuh"
#include "device/wavefront.cuh"
#include "drive.h"
#include "kernels.h"
#include "sky.h"

namespace rmd {

// ------------------------------------------------------------- frame set-up
__global__ void k_frame_init(Counters *cnt, uint32_t capacity, uint64_t firstPath, uint64_t endPath) {
    cnt->nQ[0] = cnt->nQ[1] = 0;
    cnt->nF[0] = cnt->nF[1] = 0;
    cnt->nShadow = cnt->nShadowPrev = 0;
    cnt->traceWork = cnt->shadowWork = 0;
    cnt->errors = 0;
    cnt->capacity = capacity;
    cnt->nHit = cnt->nMiss = 0;  // numRecords / numSamples persist across frames (the renderer resets them)
    cnt->nextPath = cnt->handOut[0] = cnt->handOut[1] = firstPath;
    cnt->endPath = endPath;
    cnt->numPaths = endPath - firstPath;
    cnt->loopIterations = 0;
    cnt->pathsDone = 0;
    cnt->segments = 0;
    cnt->shadowRays = 0;
    cnt->rays = 0;
    cnt->invalid = 0;
    cnt->filmStart = cnt->traceStart = cnt->traceEnd = 0;
    cnt->nsFilm = cnt->nsTrace = cnt->nsShade = 0;
    cnt->traceClocks[0] = cnt->traceClocks[1] = 0;
}

// ------------------------------------------------------------- film + regeneration
// Adds the radiance of the paths in finish list f to the film (the film writes of intersection.metal:84-87,111-116,174-178 and
// shadow.metal:24-27, gathered per path) and appends the next camera samples
// (generate.metal:72-121) to S[p]: sample j takes path id nextPath + j and
// position nQ[p] + j, so no counter is contended.  BATCH: path ids run over
// the concatenated pixels of all views (fp.numPixels in total); each sample
// takes its view's camera, size and PCG stream (the view's own pixel index),
// so a view renders as it would alone.
template <bool BATCH>
__global__ void __launch_bounds__(256) k_film_regen(Context ctx, PathPool pool, FrameParams fp, Counters *cnt,
                                                    uint32_t p, uint32_t f) {
    waitForPreviousKernel();
    const uint32_t nFin = cnt->nF[f];
    const uint32_t base = cnt->nQ[p];
    const unsigned long long first = cnt->handOut[p];
    const uint32_t nNew = newPaths(cnt, p, first);
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // counters of later stages of this iteration
        cnt->nQ[p ^ 1u] = 0;
        cnt->nShadowPrev = cnt->nShadow;
        cnt->nShadow = 0;
        cnt->traceWork = 0;
        cnt->shadowWork = 0;
        cnt->nHit = 0;
        cnt->nMiss = 0;
        cnt->nextPath = first;
        cnt->handOut[p ^ 1u] = first + nNew;
        const unsigned long long t = deviceNs();
        if (cnt->traceEnd) {
            cnt->nsTrace += cnt->traceEnd - cnt->traceStart;
            cnt->nsShade += t - cnt->traceEnd;
            cnt->traceEnd = 0;
        }
        cnt->filmStart = t;
    }
    const PathState S = pool.s[p];
    const uint32_t n = max(nFin, nNew);
    uint32_t finished = 0, samples = 0;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        if (j < nFin) {
            const float4 L = __ldcs(&pool.finLists[f][j]);
            const uint32_t px = __float_as_uint(L.w);
            if (fp.filmFp64) {
                atomicAdd(&fp.film64[3 * (size_t)px + 0], (double)L.x);
                atomicAdd(&fp.film64[3 * (size_t)px + 1], (double)L.y);
                atomicAdd(&fp.film64[3 * (size_t)px + 2], (double)L.z);
            } else {
                atomicAdd(&fp.film[px], make_float4(L.x, L.y, L.z, 1.0f));
            }
            finished++;
            if (pool.records) {  // complete the path's guide training record
                const float4 r2 = __ldcs(&pool.finRecLists[f][4 * j + 2]);
                if (r2.w > 0.0f) {
                    samples++;  // a training sample; only nonzero targets are stored
                    const float4 r0 = __ldcs(&pool.finRecLists[f][4 * j + 0]), r1 = __ldcs(&pool.finRecLists[f][4 * j + 1]);
                    const float4 r3 = __ldcs(&pool.finRecLists[f][4 * j + 3]);
                    const float y = r2.w * r3.w * ((L.x - r3.x) + (L.y - r3.y) + (L.z - r3.z)) * (1.0f / 3.0f);
                    if (y > 0.0f && isfinite(y)) {
                        // a ring: the newest records replace the oldest
                        const uint32_t k = warpAppend(&cnt->numRecords) & (pool.recordCapacity - 1u);
                        GuideRecord g;
                        g.features[0] = r0.x; g.features[1] = r0.y; g.features[2] = r0.z; g.features[3] = r0.w;
                        g.features[4] = r1.x; g.features[5] = r1.y; g.features[6] = r1.z;
                        g.pdfBsdf = r1.w;
                        g.dir[0] = r2.x; g.dir[1] = r2.y; g.dir[2] = r2.z;
                        g.y = y;
                        pool.records[k] = g;
                    }
                }
            }
        }
        if (j < nNew) {
            const unsigned long long id = first + j;
            const uint32_t sample = (uint32_t)(id / fp.numPixels);
            const uint32_t r = (uint32_t)(id - (unsigned long long)sample * fp.numPixels);
            uint32_t x, y, pixel, sampleWord;
            PrngState prng;
            float3 org, dir;
            float nearClip, farClip;
            if constexpr (BATCH) {
                const uint32_t view = batchViewOf(pool.views, pool.numViews, r);
                const BatchView &bv = pool.views[view];
                FrameParams vf = fp;  // the view's frame
                vf.width = bv.width;
                vf.height = bv.height;
                vf.numPixels = bv.numPixels;
                blockLinearToPixel(r - bv.pixelOffset, bv.width, bv.height, x, y);
                cameraRay(bv.ctx, vf, x, y, sample, prng, org, dir);
                nearClip = bv.ctx.nearClip;
                farClip = bv.ctx.farClip;
                pixel = bv.pixelOffset + y * bv.width + x;
                sampleWord = (view << BATCH_SAMPLE_BITS) | sample;
            } else {
                blockLinearToPixel(r, fp.width, fp.height, x, y);
                cameraRay(ctx, fp, x, y, sample, prng, org, dir);
                nearClip = ctx.nearClip;
                farClip = ctx.farClip;
                pixel = y * fp.width + x;
                sampleWord = sample;
            }
            const uint32_t k = base + j;
            const uint2 rs = prng.pack();
            __stcs(&S.rayO[k], f4(org, nearClip));
            __stcs(&S.rayD[k], f4(dir, farClip));
            __stcs(&S.tp[k], make_float4(1.0f, 1.0f, 1.0f, inf_f()));
            __stcs(&S.L[k], make_float4(0.0f, 0.0f, 0.0f, __uint_as_float((uint32_t)RayFlagsCamera << 16)));
            __stcs(&S.id[k], make_uint4(pixel, sampleWord, rs.x, rs.y));
        }
    }
    blockAdd64(&cnt->pathsDone, finished);
    if (pool.records) {
        samples = __reduce_add_sync(0xffffffffu, samples);
        if ((threadIdx.x & 31) == 0 && samples) atomicAdd(&cnt->numSamples, samples);
    }
}

// ------------------------------------------------------------- traversal
template <bool BATCH>
__device__ __forceinline__ void closestRay(const PathPool &pool, const PathState &S, uint32_t idx, const WideNode *&nodes,
                                           const float4 *&tris, float4 &o, float4 &d) {
    if constexpr (BATCH) {
        const BatchView &bv = pool.views[__ldcg(&S.id[idx].y) >> BATCH_SAMPLE_BITS];
        nodes = static_cast<const WideNode *>(bv.nodes);
        tris = bv.tris;
    }
    o = __ldcs(&S.rayO[idx]);
    d = __ldcs(&S.rayD[idx]);
}
// a shadow ray: origin and tmax, direction and target (BATCH: the ray's view in bits 22-29 of the target)
template <bool BATCH>
__device__ __forceinline__ void shadowRay(const PathPool &pool, uint32_t idx, const WideNode *&nodes, const float4 *&tris,
                                          float4 &o, float4 &d) {
    o = __ldcs(&pool.shO[idx]);
    d = __ldcs(&pool.shD[idx]);
    if constexpr (BATCH) {
        const BatchView &bv = pool.views[(__float_as_uint(d.w) >> BATCH_TARGET_BITS) & 0xffu];
        nodes = static_cast<const WideNode *>(bv.nodes);
        tris = bv.tris;
    }
}
// handleShadowRays (shadow.metal:6-29): an unoccluded shadow ray adds its
// weight to its path's radiance, in S[q ^ 1] for a path that continues and in
// finish list q for one that ended.
template <bool BATCH>
__device__ __forceinline__ void unoccluded(const PathPool &pool, Counters *cnt, uint32_t q, uint32_t idx, uint32_t target) {
    if (target == 0xffffffffu) return;  // all ones: the path overflowed its queue
    const bool finished = (target & SHADOW_TO_FINISHED) != 0u;
    const uint32_t at = target & (BATCH ? BATCH_TARGET_MASK : SHADOW_TARGET_MASK);
    float4 *dst = finished ? &pool.finLists[q][at] : &pool.s[q ^ 1u].L[at];
    const float4 w = __ldcs(&pool.shW[idx]);
    float4 L = *dst;
    L.x += w.x;
    L.y += w.y;
    L.z += w.z;
    *dst = L;
    if (target & SHADOW_TO_RECORD) {  // light sample of the recorded vertex: not through its sampled direction
        float4 *rec = finished ? &pool.finRecLists[q][4 * at + 3] : &pool.s[q ^ 1u].rec[4 * at + 3];
        float4 r = *rec;
        r.x += w.x;
        r.y += w.y;
        r.z += w.z;
        *rec = r;
    }
    if (pool.shRec && w.w > 0.0f) {
        // a training record of the vertex's light sample: its direction,
        // target (MIS-weighted contribution / throughput) and features
        const float y = (w.x + w.y + w.z) * (1.0f / 3.0f) * w.w;
        if (y > 0.0f && isfinite(y)) {
            const uint32_t k = atomicAdd(&cnt->numRecords, 1u) & (pool.recordCapacity - 1u);
            const float4 r0 = __ldcs(&pool.shRec[2 * idx]), r1 = __ldcs(&pool.shRec[2 * idx + 1]);
            const float4 d = __ldcs(&pool.shD[idx]);
            GuideRecord g;
            g.features[0] = r0.x; g.features[1] = r0.y; g.features[2] = r0.z; g.features[3] = r0.w;
            g.features[4] = r1.x; g.features[5] = r1.y; g.features[6] = r1.z;
            g.pdfBsdf = r1.w;
            g.dir[0] = d.x; g.dir[1] = d.y; g.dir[2] = d.z;
            g.y = y;
            pool.records[k] = g;
        }
    }
}

constexpr uint32_t TRACE_THREADS = 128, TRACE_GROUPS = TRACE_THREADS / 8;

// the SM's clock in units of 256 cycles
__device__ __forceinline__ uint32_t clock256() { return (uint32_t)(clock64() >> 8); }

// One ray per group of 8 lanes: the block's closest-hit or shadow rays.  Out
// of line, so that it takes no registers from the loop of whole warps.
template <bool BATCH, bool CLOSEST, bool SHADOW>
__device__ __noinline__ void traceByGroups(const WideNode *__restrict__ sceneNodes, const float4 *__restrict__ sceneTris,
                                           const PathPool &pool, Counters *cnt, uint32_t p, uint32_t q,
                                           uint32_t nClosest, uint32_t nShadow, uint32_t *clocks) {
    __shared__ uint2 stacks[TRACE_GROUPS * TRAVERSAL_STACK];
    __shared__ uint32_t found[TRACE_GROUPS];  // per group: index << 1 | hit, or all ones
    const uint32_t closestWarps = (nClosest + 3u) / 4u, shadowWarps = (nShadow + 3u) / 4u;
    const uint32_t warp = blockIdx.x * (TRACE_THREADS / 32u) + (threadIdx.x >> 5);
    const uint32_t group = threadIdx.x >> 3, inWarp = group & 3u;
    const bool first = (threadIdx.x & 7u) == 0u;
    uint2 *stack = stacks + (threadIdx.x >> 5) * 4u * TRAVERSAL_STACK;
    const WideNode *nodes = sceneNodes;
    const float4 *tris = sceneTris;
    float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f), d = make_float4(0.0f, 0.0f, 1.0f, 0.0f);
    TraversalState s;
    uint32_t mine = 0xffffffffu;
    const uint32_t t0 = clock256();
    if (CLOSEST && warp < closestWarps) {
        const uint32_t idx = 4u * warp + inWarp;
        const bool have = idx < nClosest;
        if (have) closestRay<BATCH>(pool, pool.s[p], idx, nodes, tris, o, d);
        traverseGroups<false>(s, have, nodes, tris, xyz(o), xyz(d), o.w, d.w, stack, &cnt->errors);
        if (have) {
            float4 hit;
            uint32_t inst;
            const bool ok = closestHit(s, tris, hit, inst);
            if (first) {
                __stcs(&pool.hit[idx], hit);
                __stcs(&pool.hitInst[idx], inst);
            }
            mine = idx << 1 | (ok ? 1u : 0u);
        }
        if ((threadIdx.x & 31u) == 0u) atomicAdd(&clocks[0], clock256() - t0);
    } else if (SHADOW && warp < closestWarps + shadowWarps) {
        const uint32_t idx = 4u * (warp - closestWarps) + inWarp;
        const bool have = idx < nShadow;
        if (have) shadowRay<BATCH>(pool, idx, nodes, tris, o, d);
        traverseGroups<true>(s, have, nodes, tris, xyz(o), xyz(d), SHADOW_EPS, o.w, stack, &cnt->errors);
        if (have && first && s.hitTri < 0) unoccluded<BATCH>(pool, cnt, q, idx, __float_as_uint(d.w));
        if ((threadIdx.x & 31u) == 0u) atomicAdd(&clocks[1], clock256() - t0);
    }
    if (CLOSEST) {  // the block's rays into the shading order with one atomic each for hits and misses
        if (first) found[group] = mine;
        __syncthreads();
        if (threadIdx.x < TRACE_GROUPS) {
            const uint32_t f = found[threadIdx.x];
            if (f != 0xffffffffu) {
                if (f & 1u) pool.order[warpAppend(&cnt->nHit)] = f >> 1;
                else pool.order[pool.capacity - 1u - warpAppend(&cnt->nMiss)] = f >> 1;
            }
        }
    }
}

// CLOSEST: the closest hits of the active paths of parity p.  SHADOW: the
// shadow rays cast by the shading pass of parity q.  Both in one launch trace
// the previous iteration's shadow rays (q = p ^ 1) beside this iteration's
// closest hits: one launch and one drain of its slowest rays less per
// iteration.
//
// Persistent warps (Aila & Laine 2009): a warp takes 32 consecutive queue
// entries with one atomic and traces them to the end.  With so few rays that
// every one gets 8 lanes at once (28 k for 12 blocks on each of 148 SMs) each
// is traced by a group of 8 lanes instead: the launch is then as long as its
// slowest ray, and a group's steps are about four times shorter.
//
// B200, per render: 192 x 108 x 1 spp (20 k paths) traversal 0.33 -> 0.07 ms;
// 1080p x 1 spp of the 852 k-triangle scene 2.71 -> 1.74 ms (closest hits 1.11,
// shadow rays 0.63), most of it in the last iterations; 1080p x 64 spp 83.0 -> 83.4 ms (bound by divergence and
// issue there; 64 spilled bytes in the loop had cost 2.5 %).
template <bool BATCH, bool CLOSEST, bool SHADOW>
__global__ void __launch_bounds__(TRACE_THREADS, 8) k_trace(const WideNode *__restrict__ sceneNodes,
                                                            const float4 *__restrict__ sceneTris,
                                                            const __grid_constant__ PathPool pool, Counters *cnt,
                                                            uint32_t p, uint32_t q) {
    __shared__ uint32_t clocks[2];  // of the block's warps on closest hits and on shadow rays
    waitForPreviousKernel();
    const uint32_t nClosest = CLOSEST ? activeCount(cnt, p) : 0u;
    const uint32_t nShadow = SHADOW ? (CLOSEST ? cnt->nShadowPrev : cnt->nShadow) : 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (SHADOW) cnt->shadowRays += nShadow;
        if (CLOSEST) {
            cnt->nF[p] = 0;  // the film kernel has read it; the shading pass fills it next
            const unsigned long long t = deviceNs();
            cnt->nsFilm += t - cnt->filmStart;
            cnt->traceStart = t;
        }
    }
    if (threadIdx.x < 2u) clocks[threadIdx.x] = 0u;
    __syncthreads();
    if ((nClosest + 3u) / 4u + (nShadow + 3u) / 4u <= gridDim.x * (TRACE_THREADS / 32u)) {
        traceByGroups<BATCH, CLOSEST, SHADOW>(sceneNodes, sceneTris, pool, cnt, p, q, nClosest, nShadow, clocks);
    } else {
        TraversalState s;
        TraversalStack stack;
        const uint32_t lane = threadIdx.x & 31u;
        const uint32_t nChunks = (nClosest + 31u) / 32u;  // closest hits first
        const uint32_t total = nChunks + (nShadow + 31u) / 32u;
        uint32_t *work = CLOSEST ? &cnt->traceWork : &cnt->shadowWork;
        while (true) {
            uint32_t chunk = 0;
            if (lane == 0) chunk = atomicAdd(work, 1u);
            chunk = __shfl_sync(0xffffffffu, chunk, 0);
            if (chunk >= total) break;
            const WideNode *nodes = sceneNodes;
            const float4 *tris = sceneTris;
            float4 o, d;
            const bool closest = CLOSEST && (!SHADOW || chunk < nChunks);
            if (CLOSEST && SHADOW && lane == 0) atomicSub(&clocks[closest ? 0 : 1], clock256());
            if (closest) {
                const uint32_t idx = 32u * chunk + lane;
                if (idx < nClosest) {
                    closestRay<BATCH>(pool, pool.s[p], idx, nodes, tris, o, d);
                    beginTraversal(s, nodes, xyz(o), xyz(d), o.w, d.w);
                    traverse<false>(s, stack, nodes, tris, &cnt->errors);
                    float4 hit;
                    uint32_t inst;
                    const bool ok = closestHit(s, tris, hit, inst);
                    __stcs(&pool.hit[idx], hit);
                    __stcs(&pool.hitInst[idx], inst);
                    if (ok) pool.order[warpAppend(&cnt->nHit)] = idx;
                    else pool.order[pool.capacity - 1u - warpAppend(&cnt->nMiss)] = idx;
                }
            } else if constexpr (SHADOW) {
                const uint32_t idx = 32u * (chunk - nChunks) + lane;
                if (idx < nShadow) {
                    shadowRay<BATCH>(pool, idx, nodes, tris, o, d);
                    beginTraversal(s, nodes, xyz(o), xyz(d), SHADOW_EPS, o.w);
                    traverse<true>(s, stack, nodes, tris, &cnt->errors);
                    if (s.hitTri < 0)
                        unoccluded<BATCH>(pool, cnt, q, idx, __float_as_uint(__ldcg(&pool.shD[idx].w)));
                }
            }
            __syncwarp();
            if (CLOSEST && SHADOW && lane == 0) atomicAdd(&clocks[closest ? 0 : 1], clock256());
        }
    }
    if (CLOSEST) {
        __syncthreads();
        if (SHADOW && threadIdx.x < 2u) atomicAdd(&cnt->traceClocks[threadIdx.x], (unsigned long long)clocks[threadIdx.x]);
        if (threadIdx.x == 0) atomicMax(&cnt->traceEnd, deviceNs());
    }
}

// ------------------------------------------------------------- device-driven loop
// Last node of the body of a CUDA-graph while loop of `itersPerBody`
// wavefront iterations: continue while paths remain, no error was flagged
// and the iteration bound (which every render reaches only on a fault) is
// not passed.  The bound also guarantees that the loop ends.
__global__ void k_loop_condition(Counters *cnt, cudaGraphConditionalHandle handle, uint32_t itersPerBody,
                                 uint32_t maxIterations) {
    const uint32_t it = cnt->loopIterations + itersPerBody;
    cnt->loopIterations = it;
    const bool more = cnt->pathsDone < cnt->numPaths && cnt->errors == 0u && it < maxIterations;
    if (!more && cnt->pathsDone < cnt->numPaths && cnt->errors == 0u) atomicOr(&cnt->errors, ERR_LOOP_BOUND);
    cudaGraphSetConditional(handle, more ? 1u : 0u);
}

// ------------------------------------------------------------- environment map
// kernels/envmap/reduce.metal:3-24 over one level of `cur x cur` quads.
__global__ void k_envmap_reduce(float *mip, int cur) {
    const int tx = blockIdx.x * blockDim.x + threadIdx.x;
    const int ty = blockIdx.y * blockDim.y + threadIdx.y;
    if (tx >= cur || ty >= cur) return;
    const int inputIndex = ty * cur + tx;
    const int gridLength = cur * cur;
    float sum = 0.0f;
    for (int i = 0; i < 4; ++i) sum += mip[gridLength + 4 * inputIndex + i];
    for (int i = 0; i < 4; ++i) mip[gridLength + 4 * inputIndex + i] /= sum;
    const unsigned qx = tx / 2, qy = ty / 2, qw = cur / 2;
    const unsigned outputIndex = cur == 1 ? 0u : 4u * (qy * qw + qx) + (tx & 1) + 2u * (ty & 1);
    mip[outputIndex] = sum;
}
// kernels/envmap/normalize.metal:4-11
__global__ void k_envmap_normalize(const float *sum, float *pdfs, uint32_t gridSize) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= gridSize) return;
    const float scale = (float)gridSize * warp::uniformSquareToSpherePdf() / *sum;
    pdfs[i] *= scale;
}

// Clears *uniform if the map is not uniform: a texel of `pdfs` that differs
// from the first, or a probability of the pyramid (the quads from the second
// level on) other than 1/4.
__global__ void k_envmap_uniform(const float *pdfs, uint32_t numPdfs, const float *quads, uint32_t numQuadFloats,
                                 int *uniform) {
    const float first = pdfs[0];
    bool same = true;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < numPdfs; i += gridDim.x * blockDim.x)
        same = same && pdfs[i] == first;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < numQuadFloats; i += gridDim.x * blockDim.x)
        same = same && quads[i] == 0.25f;
    if (!same) *uniform = 0;
}

// ------------------------------------------------------------- film read-out
// kernels/utils/normalizeImage.metal:11-59
__device__ float3 tonemapHablePartial(float3 x) {
    const float hA = 0.15f, hB = 0.50f, hC = 0.10f, hD = 0.20f, hE = 0.02f, hF = 0.30f;
    return ((x * (hA * x + hC * hB) + hD * hE) / (x * (hA * x + hB) + hD * hF)) - hE / hF;
}
// color = exposure * film; color /= divisor (the frame count, 1 when not
// accumulating), then the tonemap, in the reference's order of operations;
// `channels` 3 (RGB) or 4 (RGB and alpha 1, as normalizeImage writes).
__global__ void k_film_resolve(const float4 *film, const double *film64, int fp64, float *out, uint32_t numPixels,
                               float exposure, float divisor, uint32_t tonemapping, uint32_t channels) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= numPixels) return;
    float3 c;
    if (fp64) c = make_float3((float)film64[3 * (size_t)i], (float)film64[3 * (size_t)i + 1], (float)film64[3 * (size_t)i + 2]);
    else c = xyz(film[i]);
    c = exposure * c;
    if (divisor != 1.0f) c = make_float3(__fdiv_rn(c.x, divisor), __fdiv_rn(c.y, divisor), __fdiv_rn(c.z, divisor));
    if (tonemapping == 1u) {
        const float3 curr = tonemapHablePartial(c * 2.0f);
        const float3 whiteScale = 1.0f / tonemapHablePartial(f3(11.2f));
        c = curr * whiteScale;
    } else if (tonemapping == 2u) {
        const float tA = 2.51f, tB = 0.03f, tC = 2.43f, tD = 0.59f, tE = 0.14f;
        c = saturate((c * (tA * c + tB)) / (c * (tC * c + tD) + tE));
    }
    float *o = out + (size_t)channels * i;
    o[0] = c.x;
    o[1] = c.y;
    o[2] = c.z;
    if (channels == 4) o[3] = 1.0f;
}

// ------------------------------------------------------------- sky texture
// SKY_nishita_skymodel_precompute_texture (host/sky/sky_nishita.cpp:295-341)
// on the device: texel (x, y) of the left half and its mirror image.
__global__ void k_sky_texture(float4 *texels, int width, int height, float sunElevation, float altitude, float air,
                              float dust, float ozone) {
    const int half = width / 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= half * height) return;
    const int y = i / half, x = i - y * half;
    const rmdsky::V3 c = rmdsky::skyTexel(x, y, width, height, sunElevation, altitude, air, dust, ozone);
    const float4 v = make_float4(c.x, c.y, c.z, 1.0f);
    texels[(size_t)y * width + x] = v;
    texels[(size_t)y * width + (width - x - 1)] = v;
}

// ------------------------------------------------------------- test hooks
__global__ void k_debug_prng(uint32_t mode, uint64_t a, uint64_t b, int n, float *out) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    PrngState p = mode == RNG_TEA ? PrngState::tea((uint32_t)a, (uint32_t)b) : PrngState::pcg(a, b);
    for (int i = 0; i < n; i++) out[i] = p.sample();
}
__global__ void k_debug_trace(const WideNode *nodes, const float4 *tris, const float *rays, int n, int any, float *out,
                              uint32_t *inst, uint32_t *errors) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *r = rays + 8 * (size_t)i;
    const float3 o = make_float3(r[0], r[1], r[2]), d = make_float3(r[4], r[5], r[6]);
    float4 h = make_float4(-1.0f, 0.0f, 0.0f, 0.0f);
    uint32_t id = 0;
    if (any) {
        h.x = traceAny(nodes, tris, o, d, r[3], r[7], errors) ? 1.0f : -1.0f;
    } else {
        traceClosest(nodes, tris, o, d, r[3], r[7], h, id, errors);
    }
    out[4 * (size_t)i + 0] = h.x;
    out[4 * (size_t)i + 1] = h.y;
    out[4 * (size_t)i + 2] = h.z;
    out[4 * (size_t)i + 3] = h.w;
    inst[i] = id;
}

// The traversal kernels' triangle layout from the builders' (v0, v1, v2 per
// triangle, float4 each): three copies per triangle, copy k with the
// coordinates rotated so that axis k comes last (device/traverse.cuh).
__global__ void k_rotate_triangles(const float4 *__restrict__ in, float4 *__restrict__ out, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const float4 v = in[3 * (size_t)i + j];
            out[TRI_FLOAT4 * (size_t)i + 0 + j] = make_float4(v.y, v.z, v.x, v.w);
            out[TRI_FLOAT4 * (size_t)i + 3 + j] = make_float4(v.z, v.x, v.y, v.w);
            out[TRI_FLOAT4 * (size_t)i + 6 + j] = v;
        }
    }
}

// ------------------------------------------------------------- scene building
// The meshes' packed arrays as the shading kernels read them: positions and
// normals on 16 bytes, faces with their material.
__global__ void k_pack_mesh(const float *__restrict__ pos, const float *__restrict__ nrm, size_t numVertices,
                            const uint32_t *__restrict__ idx, const uint16_t *__restrict__ mat, size_t numFaces,
                            float4 *__restrict__ vertices, float4 *__restrict__ normals, uint4 *__restrict__ faces) {
    const size_t n = max(numVertices, numFaces), step = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const size_t k = 3 * i;
        if (i < numVertices) {
            vertices[i] = make_float4(pos[k], pos[k + 1], pos[k + 2], 0.0f);
            normals[i] = make_float4(nrm[k], nrm[k + 1], nrm[k + 2], 0.0f);
        }
        if (i < numFaces) faces[i] = make_uint4(idx[k], idx[k + 1], idx[k + 2], mat[i]);
    }
}

__device__ __forceinline__ uint32_t orderedBits(float f) {  // unsigned order = float order
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// The world-space triangles of all instances for the device BVH builder, in
// the host's order and arithmetic (transformPoint: products and sums rounded
// one by one), and their bounds (3 minima, 3 maxima, as orderedBits).
__global__ void k_flatten(const float4 *__restrict__ vertices, const uint4 *__restrict__ faces,
                          const PerInstanceData *__restrict__ instances, uint32_t numInstances, uint32_t n,
                          float *__restrict__ v0, float *__restrict__ v1, float *__restrict__ v2,
                          uint32_t *__restrict__ inst, uint32_t *__restrict__ prim, uint32_t *bounds) {
    float lo[3] = {inf_f(), inf_f(), inf_f()}, hi[3] = {-inf_f(), -inf_f(), -inf_f()};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t a = 0, b = numInstances;  // the last instance that starts at or before i
        while (b - a > 1u) {
            const uint32_t m = (a + b) >> 1;
            if (instances[m].triOffset <= i) a = m;
            else b = m;
        }
        const PerInstanceData &in = instances[a];
        const uint4 f = faces[in.faceOffset + (i - in.triOffset)];
        const uint32_t vi[3] = {f.x, f.y, f.z};
        float *const out[3] = {v0, v1, v2};
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const float4 p = vertices[in.vertexOffset + vi[j]];
            const float4 *M = in.pointTransform;
            float w[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float x = __fmul_rn(comp(xyz(M[0]), k), p.x), y = __fmul_rn(comp(xyz(M[1]), k), p.y);
                const float z = __fmul_rn(comp(xyz(M[2]), k), p.z);
                w[k] = __fadd_rn(__fadd_rn(__fadd_rn(x, y), z), comp(xyz(M[3]), k));
                lo[k] = fminf(lo[k], w[k]);
                hi[k] = fmaxf(hi[k], w[k]);
                out[j][3 * (size_t)i + k] = w[k];
            }
        }
        inst[i] = a;
        prim[i] = i - in.triOffset;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, orderedBits(lo[k])), h = __reduce_max_sync(0xffffffffu, orderedBits(hi[k]));
        if ((threadIdx.x & 31u) == 0u) {
            atomicMin(&bounds[k], l);
            atomicMax(&bounds[3 + k], h);
        }
    }
}

}  // namespace rmd

// ------------------------------------------------------------- launch wrappers
using namespace rmd;

cudaError_t rmdLaunchLoopCondition(Counters *cnt, cudaGraphConditionalHandle handle, uint32_t itersPerBody,
                                   uint32_t maxIterations, cudaStream_t s) {
    k_loop_condition<<<1, 1, 0, s>>>(cnt, handle, itersPerBody, maxIterations);
    return cudaGetLastError();
}

cudaError_t rmdLaunchFrameInit(const PathPool &pool, Counters *cnt, uint64_t firstPath, uint64_t endPath,
                               cudaStream_t s) {
    k_frame_init<<<1, 1, 0, s>>>(cnt, pool.capacity, firstPath, endPath);
    return cudaGetLastError();
}
cudaError_t rmdLaunchFilmRegen(const Context &ctx, const PathPool &pool, const FrameParams &fp, Counters *cnt,
                               uint32_t cur, uint32_t fin, int blocks, cudaStream_t s) {
    if (pool.views) return rmdhost::launchOverlapped(k_film_regen<true>, blocks, 256, s, ctx, pool, fp, cnt, cur, fin);
    return rmdhost::launchOverlapped(k_film_regen<false>, blocks, 256, s, ctx, pool, fp, cnt, cur, fin);
}
cudaError_t rmdLaunchTrace(const WideNode *nodes, const float4 *tris, const PathPool &pool, Counters *cnt, uint32_t cur,
                           int blocks, cudaStream_t s) {
    if (pool.views) return rmdhost::launchOverlapped(k_trace<true, true, true>, blocks, TRACE_THREADS, s, nodes, tris, pool, cnt, cur, cur ^ 1u);
    return rmdhost::launchOverlapped(k_trace<false, true, true>, blocks, TRACE_THREADS, s, nodes, tris, pool, cnt, cur, cur ^ 1u);
}
cudaError_t rmdLaunchTraceClosest(const WideNode *nodes, const float4 *tris, const PathPool &pool, Counters *cnt,
                                  uint32_t cur, int blocks, cudaStream_t s) {
    if (pool.views) return rmdhost::launchOverlapped(k_trace<true, true, false>, blocks, TRACE_THREADS, s, nodes, tris, pool, cnt, cur, 0u);
    return rmdhost::launchOverlapped(k_trace<false, true, false>, blocks, TRACE_THREADS, s, nodes, tris, pool, cnt, cur, 0u);
}
cudaError_t rmdLaunchTraceShadow(const WideNode *nodes, const float4 *tris, const PathPool &pool, Counters *cnt,
                                 uint32_t cur, int blocks, cudaStream_t s) {
    if (pool.views) return rmdhost::launchOverlapped(k_trace<true, false, true>, blocks, TRACE_THREADS, s, nodes, tris, pool, cnt, cur, cur);
    return rmdhost::launchOverlapped(k_trace<false, false, true>, blocks, TRACE_THREADS, s, nodes, tris, pool, cnt, cur, cur);
}
cudaError_t rmdLaunchEnvmapReduce(float *mip, int cur, cudaStream_t s) {
    dim3 b(8, 8), g((cur + 7) / 8, (cur + 7) / 8);
    k_envmap_reduce<<<g, b, 0, s>>>(mip, cur);
    return cudaGetLastError();
}
cudaError_t rmdLaunchEnvmapNormalize(const float *sum, float *pdfs, uint32_t gridSize, cudaStream_t s) {
    k_envmap_normalize<<<(gridSize + 255) / 256, 256, 0, s>>>(sum, pdfs, gridSize);
    return cudaGetLastError();
}
cudaError_t rmdLaunchEnvmapUniform(const float *pdfs, uint32_t numPdfs, const float *quads, uint32_t numQuadFloats,
                                   int *uniform, cudaStream_t s) {
    const uint32_t n = std::max(numPdfs, numQuadFloats);
    k_envmap_uniform<<<std::min<uint32_t>((n + 255) / 256, 148u * 8u), 256, 0, s>>>(pdfs, numPdfs, quads, numQuadFloats,
                                                                                  uniform);
    return cudaGetLastError();
}
cudaError_t rmdLaunchFilmResolve(const float4 *film, const double *film64, int fp64, float *out, uint32_t numPixels,
                                 float exposure, float divisor, uint32_t tonemapping, uint32_t channels, cudaStream_t s) {
    k_film_resolve<<<(numPixels + 255) / 256, 256, 0, s>>>(film, film64, fp64, out, numPixels, exposure, divisor,
                                                            tonemapping, channels);
    return cudaGetLastError();
}
cudaError_t rmdLaunchDebugPrng(uint32_t mode, uint64_t a, uint64_t b, int n, float *out, cudaStream_t s) {
    k_debug_prng<<<1, 1, 0, s>>>(mode, a, b, n, out);
    return cudaGetLastError();
}
cudaError_t rmdLaunchPackMesh(const float *pos, const float *nrm, size_t numVertices, const uint32_t *idx,
                              const uint16_t *mat, size_t numFaces, float4 *vertices, float4 *normals, uint4 *faces,
                              cudaStream_t s) {
    const size_t n = std::max(numVertices, numFaces);
    if (n == 0) return cudaSuccess;
    k_pack_mesh<<<(unsigned)std::min<size_t>((n + 255) / 256, 148u * 16u), 256, 0, s>>>(pos, nrm, numVertices, idx, mat, numFaces,
                                                                             vertices, normals, faces);
    return cudaGetLastError();
}
cudaError_t rmdLaunchFlatten(const float4 *vertices, const uint4 *faces, const PerInstanceData *instances,
                             uint32_t numInstances, uint32_t n, float *v0, float *v1, float *v2, uint32_t *inst,
                             uint32_t *prim, uint32_t *boundsScratch, float *bounds, cudaStream_t s) {
    uint32_t b[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    cudaError_t e = cudaMemcpyAsync(boundsScratch, b, sizeof(b), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
    k_flatten<<<std::min<uint32_t>((n + 255) / 256, 148u * 16u), 256, 0, s>>>(vertices, faces, instances, numInstances, n,
                                                                           v0, v1, v2, inst, prim, boundsScratch);
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(b, boundsScratch, sizeof(b), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return e;
    for (int k = 0; k < 6; k++) {
        const uint32_t u = (b[k] & 0x80000000u) ? (b[k] & 0x7fffffffu) : ~b[k];
        memcpy(&bounds[k], &u, sizeof(float));
    }
    return cudaSuccess;
}
cudaError_t rmdLaunchRotateTriangles(const float4 *in, float4 *out, uint32_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_rotate_triangles<<<std::min<uint32_t>((n + 255) / 256, 148u * 16u), 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}
cudaError_t rmdLaunchDebugTrace(const WideNode *nodes, const float4 *tris, const float *rays, int n, int any, float *out,
                                uint32_t *inst, uint32_t *errors, cudaStream_t s) {
    k_debug_trace<<<(n + 127) / 128, 128, 0, s>>>(nodes, tris, rays, n, any, out, inst, errors);
    return cudaGetLastError();
}
cudaError_t rmdLaunchSkyTexture(float4 *texels, uint32_t width, uint32_t height, float sunElevation, float altitude,
                                float air, float dust, float ozone, cudaStream_t s) {
    const uint32_t n = width / 2 * height;
    if (n == 0) return cudaSuccess;
    k_sky_texture<<<(n + 127) / 128, 128, 0, s>>>(texels, (int)width, (int)height, sunElevation, altitude, air, dust,
                                                  ozone);
    return cudaGetLastError();
}
