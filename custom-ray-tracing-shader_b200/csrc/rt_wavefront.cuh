// Path state of the wavefront integrators (single scene and batch) between
// their stages, device only. A bounce moves what it needs and no more:
// shading is bound by this traffic (it read and wrote 208 bytes per path and
// bounce; now 48 + 16 in and 48 out for a path that goes on, 64 in and
// nothing or 16 out for one that ends).
//   - before the first bounce only the ray is stored; throughput 1, radiance
//     and first-hit values 0 are known, and so is the queue (every path);
//   - origin, direction and throughput are written for paths that go on;
//   - radiance is written when the bounce changed it (always after the first);
//   - albedo, normal and first-hit distance are written once.
#pragma once
#include "rt_render.cuh"

namespace rt {

// Counters of bounce b, zeroed by the generate kernel of a wave: live paths
// and shadow rays queued for it, and the two traversals' fetch positions.
enum { kLive = 0, kExtendFetch = 1, kShadowRays = 2, kShadowFetch = 3, kCountStride = 4 };
constexpr int kWaveCounts = kCountStride * (32 + 1);  // maxBounces is at most 32

#ifdef __CUDACC__
__device__ __forceinline__ int* bounceCounts(const WavefrontBuffers& B, int bounce) { return B.counts + kCountStride * bounce; }
__device__ __forceinline__ void initCounts(const WavefrontBuffers& B, int paths) {
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < kWaveCounts; i += blockDim.x) B.counts[i] = i == kLive ? paths : 0;
}
// The path in place k of the bounce's queue (every path at the first bounce).
__device__ __forceinline__ const int* bounceQueue(const WavefrontBuffers& B, int bounce) {
    return bounce ? B.queue[bounce & 1] : nullptr;
}

// Appends to a queue with one atomic per warp.
__device__ __forceinline__ int warpAppend(int* counter, bool want) {
    unsigned mask = __ballot_sync(0xFFFFFFFFu, want);
    if (!mask) return -1;
    int lane = threadIdx.x & 31;
    int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    return want ? base + __popc(mask & ((1u << lane) - 1u)) : -1;
}

// Path p's ray (rayWord: what the caller keeps beside the direction) before
// its first bounce.
__device__ __forceinline__ void storeStart(const WavefrontBuffers& B, int p, const PathState& st, float rayWord) {
    B.pathA[p] = make_float4(st.origin.x, st.origin.y, st.origin.z, 0.0f);
    B.pathB[p] = make_float4(st.dir.x, st.dir.y, st.dir.z, rayWord);
}
__device__ __forceinline__ PathState loadPath(const WavefrontBuffers& B, int p, bool first, float4 a, float4 b) {
    PathState st;
    st.origin = v3(a.x, a.y, a.z); st.prevPdf = a.w;
    st.dir = v3(b.x, b.y, b.z);
    float4 c = make_float4(1.0f, 1.0f, 1.0f, 0.0f), rad = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!first) { c = B.pathC[p]; rad = B.radiance[p]; }
    st.throughput = v3(c.x, c.y, c.z);
    st.radiance = v3(rad.x, rad.y, rad.z); st.covered = __float_as_uint(rad.w);
    st.albedo = v3(0, 0, 0); st.normal = v3(0, 0, 0);
    st.depth = 0.0f;
    return st;
}
// After the bounce; before: the radiance that loadPath gave.
__device__ __forceinline__ void storePath(const WavefrontBuffers& B, int p, bool first, const PathState& st, float3 before,
                                          bool goesOn, float rayWord) {
    if (goesOn) {
        B.pathA[p] = make_float4(st.origin.x, st.origin.y, st.origin.z, st.prevPdf);
        B.pathB[p] = make_float4(st.dir.x, st.dir.y, st.dir.z, rayWord);
        B.pathC[p] = make_float4(st.throughput.x, st.throughput.y, st.throughput.z, 0.0f);
    }
    const bool changed = __float_as_uint(st.radiance.x) != __float_as_uint(before.x) ||
                         __float_as_uint(st.radiance.y) != __float_as_uint(before.y) ||
                         __float_as_uint(st.radiance.z) != __float_as_uint(before.z);
    if (first || changed)
        B.radiance[p] = make_float4(st.radiance.x, st.radiance.y, st.radiance.z, __uint_as_float(st.covered));
    if (first) {
        B.albedo[p] = make_float4(st.albedo.x, st.albedo.y, st.albedo.z, st.depth);
        B.normal[p] = make_float4(st.normal.x, st.normal.y, st.normal.z, 0.0f);
    }
}
__device__ __forceinline__ void storeShadow(const WavefrontBuffers& B, int slot, const ShadowRequest& req, int p,
                                            float contribWord) {
    B.shadowRay[slot] = make_float4(req.origin.x, req.origin.y, req.origin.z, req.limit);
    B.shadowDir[slot] = make_float4(req.dir.x, req.dir.y, req.dir.z, __int_as_float(p));
    B.shadowContrib[slot] = make_float4(req.contribution.x, req.contribution.y, req.contribution.z, contribWord);
}
// Adds finished path p to a pixel's running sums.
__device__ __forceinline__ void addStored(const WavefrontBuffers& B, int p, Accum& total, float& depthTotal) {
    const float4 rad = B.radiance[p], al = B.albedo[p], no = B.normal[p];
    PathState st;
    st.radiance = v3(rad.x, rad.y, rad.z); st.covered = __float_as_uint(rad.w);
    st.albedo = v3(al.x, al.y, al.z); st.normal = v3(no.x, no.y, no.z);
    addPath(total, st);
    depthTotal = depthTotal + al.w;
}
#endif

}  // namespace rt
