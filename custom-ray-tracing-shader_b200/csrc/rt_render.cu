// Render, query, sampler and denoise kernels for sm_100a.
//
// Two integrators produce bit-identical accumulations:
//  - wavefront (default): per wave of paths (a slice of the pass's, which may
//    span sample rows) a generate kernel writes camera rays, then for every
//    bounce an extend kernel (closest hit) runs over the compacted queue of
//    live paths, a shade kernel applies the bounce and compacts survivors and
//    light-sample rays into queues with warp-aggregated atomics, and a shadow
//    kernel (any hit) resolves the light samples; an accumulate kernel adds
//    the wave's paths to the running sums in row order. A pass of one wave
//    traces a bounce's shadow rays with the next bounce's closest hits. Traversal
//    kernels only hold a ray and its stack, so they run at high occupancy.
//  - one kernel per pixel (megakernel), the reference's launch shape with the
//    same traversal and shading code.
// Traversal stacks start in shared memory, one column per thread (rt_trace.cuh).
#include <algorithm>
#include <vector>

#include "rt_render.cuh"
#include "rt_trace.cuh"
#include "rt_wavefront.cuh"

namespace rt {
namespace {

constexpr int kTileX = 16, kTileY = 8, kMegaBlock = kTileX * kTileY;
// Resident blocks per SM the traversal kernels are compiled for: 8 caps them
// at 64 registers (16-40 bytes of spills) for 32 resident warps. Measured on
// the 1M-triangle workload with waves of 2^24 paths: 6 blocks (77-79
// registers) 2,841 Mrays/s, 7 (72) 2,972, 8 (64) 3,003.
constexpr int kTraceMinBlocks = 8;

// Programmatic dependent launch of a pass's stages (launchStage): a stage lets
// the next one's blocks start as its own leave the SMs and waits for the
// previous stage before it touches memory.
__device__ __forceinline__ void stageBegin() {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// Sampler tables of the pass; zeroes its ray counters and error flag (status:
// kStatusWords words).
__global__ void sobolTablesKernel(const unsigned* dirs, unsigned sample0, int rpp, unsigned seed, unsigned* passXor,
                                  unsigned* seedHash, unsigned long long* status) {
    stageBegin();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kStatusWords) status[i] = 0ull;
    int passEntries = rpp * kSobolDims;
    if (i < passEntries) {
        int r = i / kSobolDims, d = i % kSobolDims;
        passXor[i] = sobolXor(dirs, sample0 + (unsigned)r, (unsigned)d);
    } else if (i < passEntries + kSobolDims) {
        int d = i - passEntries;
        seedHash[d] = sobolHash(seed + (unsigned)d * 0x9e3779b9u);
    }
}

__device__ __forceinline__ void flushCounters(unsigned long long* counters, unsigned a, unsigned b, unsigned c) {
    unsigned sa = __reduce_add_sync(0xFFFFFFFFu, a), sb = __reduce_add_sync(0xFFFFFFFFu, b),
             sc = __reduce_add_sync(0xFFFFFFFFu, c);
    if ((threadIdx.x & 31) == 0) {
        if (sa) atomicAdd(&counters[0], (unsigned long long)sa);
        if (sb) atomicAdd(&counters[1], (unsigned long long)sb);
        if (sc) atomicAdd(&counters[2], (unsigned long long)sc);
    }
}

__global__ void __launch_bounds__(kMegaBlock) megakernel(RenderLaunch L) {
    extern __shared__ uint2 smemStack[];
    uint2* stack = smemStack + threadIdx.x;
    const int stride = kMegaBlock;
    int x = blockIdx.x * kTileX + (threadIdx.x % kTileX);
    int y = blockIdx.y * kTileY + (threadIdx.x / kTileX);
    unsigned nPrimary = 0, nSecondary = 0, nShadow = 0;
    int overflow = 0;
    if (x < L.w && y < L.h)
        renderPixel(L.scene, L.cam, L.set, x, y, L.w, L.h, L.sample0, L.passXor, L.seedHash, L.sums, L.depthSums,
                    L.pixels, stack, stride, &overflow, nPrimary, nSecondary, nShadow);
    flushCounters(L.counters, nPrimary, nSecondary, nShadow);
    if (overflow) atomicExch(L.errorFlag, 1);
}

// ---- wavefront stages ----
// A wave is the paths [start, start + n) of a pass, path k being sample row
// k / (w * h) of pixel k % (w * h); a wave may span several sample rows.
struct WaveArgs {
    RenderLaunch L;
    int start, n;
};
__device__ __forceinline__ int waveRow(const WaveArgs& A, int p) { return (A.start + p) / (A.L.w * A.L.h); }
__device__ __forceinline__ int wavePixel(const WaveArgs& A, int p) { return (A.start + p) % (A.L.w * A.L.h); }

__global__ void generateKernel(WaveArgs A, WavefrontBuffers B) {
    stageBegin();
    initCounts(B, A.n);
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= A.n) return;
    int pix = wavePixel(A, p);
    int x = pix % A.L.w, y = pix / A.L.w;
    Sampler rng{A.L.passXor + waveRow(A, p) * kSobolDims, A.L.seedHash, (unsigned)pix, 0u};
    PathState st = startPath(A.L.cam, A.L.set, x, y, A.L.w, A.L.h, rng);
    storeStart(B, p, st, 0.0f);
}

// Closest hit for every queued path (persistent, dynamic fetch).
struct ExtendIO {
    const int* queue;  // null: every path
    const float4 *pathA, *pathB;
    float4* hits;
    __device__ int path(int k) const { return queue ? queue[k] : k; }
    __device__ void load(int k, float3& o, float3& d, float& limit, unsigned&) const {
        int p = path(k);
        float4 a = pathA[p], b = pathB[p];
        o = v3(a.x, a.y, a.z); d = v3(b.x, b.y, b.z); limit = 1e30f;
    }
    __device__ void store(int k, const Hit& h) const {
        hits[path(k)] = make_float4(h.distance, h.u, h.v, __int_as_float(h.index));
    }
};
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) extendKernel(const uint4* wide, const float4* packed, WavefrontBuffers B,
                                                            int bounce, unsigned long long* counter, int* errorFlag,
                                                            int stackLimit, int refill) {
    stageBegin();
    ExtendIO io{bounceQueue(B, bounce), B.pathA, B.pathB, B.hits};
    int* c = bounceCounts(B, bounce);
    persistentTrace<false>(io, c[kLive], wide, packed, &c[kExtendFetch], counter, errorFlag, stackLimit, refill);
}

// Shading blocks: 6 of 128 threads per SM (80 registers; left alone the kernel
// takes 92 and 2 blocks of 256 fit). On the 1M-triangle pass 33.9 ms at 2 x
// 256, 33.4 at 5 x 128, 33.1 at 6 x 128, 33.3 at 8 x 128.
constexpr int kShadeBlock = 128, kShadePerSm = 6;
__global__ void __launch_bounds__(kShadeBlock, kShadePerSm) shadeKernel(WaveArgs A, WavefrontBuffers B, int bounce) {
    stageBegin();
    int* c = bounceCounts(B, bounce);
    const int count = c[kLive];
    const bool first = bounce == 0;
    const int* queue = bounceQueue(B, bounce);
    int* next = B.queue[(bounce + 1) & 1];
    int stride = gridDim.x * blockDim.x;
    int limit = ((count + 31) / 32) * 32;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < limit; k += stride) {
        bool valid = k < count;
        bool cont = false, shadow = false;
        int p = 0;
        ShadowRequest req;
        if (valid) {
            p = queue ? queue[k] : k;
            float4 hv = B.hits[p];
            PathState st = loadPath(B, p, first, B.pathA[p], B.pathB[p]);
            const float3 before = st.radiance;
            Hit h{__float_as_int(hv.w), hv.x, hv.y, hv.z};
            Sampler rng{A.L.passXor + waveRow(A, p) * kSobolDims, A.L.seedHash, (unsigned)wavePixel(A, p),
                        4u + 8u * (unsigned)bounce};
            unsigned f = shadeBounce(A.L.scene, A.L.set, bounce, st, h, rng, req);
            cont = (f & kContinue) != 0;
            shadow = (f & kShadow) != 0;
            storePath(B, p, first, st, before, cont, 0.0f);
        }
        int slot = warpAppend(&c[kCountStride + kLive], cont);
        if (slot >= 0) next[slot] = p;
        int sslot = warpAppend(&c[kShadowRays], shadow);
        if (sslot >= 0) storeShadow(B, sslot, req, p, 0.0f);
    }
}

// Light-sample visibility for every queued shadow ray (persistent, dynamic
// fetch); unoccluded samples add their contribution to the path's radiance.
struct ShadowIO {
    const float4 *ray, *dir, *contrib;
    float4* radiance;
    __device__ void load(int k, float3& o, float3& d, float& limit, unsigned&) const {
        float4 a = ray[k], b = dir[k];
        o = v3(a.x, a.y, a.z); d = v3(b.x, b.y, b.z); limit = a.w;
    }
    __device__ void store(int k, const Hit& h) const {
        if (h.index >= 0) return;
        int p = __float_as_int(dir[k].w);
        float4 c = contrib[k], rad = radiance[p];
        radiance[p] = make_float4(rad.x + c.x, rad.y + c.y, rad.z + c.z, rad.w);
    }
};
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) shadowKernel(const uint4* wide, const float4* packed, WavefrontBuffers B,
                                                            int bounce, unsigned long long* counter, int* errorFlag,
                                                            int stackLimit, int refill) {
    stageBegin();
    ShadowIO io{B.shadowRay, B.shadowDir, B.shadowContrib, B.radiance};
    int* c = bounceCounts(B, bounce);
    persistentTrace<true>(io, c[kShadowRays], wide, packed, &c[kShadowFetch], counter, errorFlag, stackLimit, refill);
}

// The light samples of a bounce and the closest hits of the next in one
// launch (they are independent: one adds to the paths' radiance, the other
// reads their rays and writes hits): the warps that finish the closest hits
// early go on with the shadow rays instead of idling through the launch's
// drain, and a bounce is two launches instead of three.
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) shadowExtendKernel(const uint4* wide, const float4* packed,
                                                                  WavefrontBuffers B, int bounce,
                                                                  unsigned long long* shadowCounter,
                                                                  unsigned long long* counter, int* errorFlag,
                                                                  int stackLimit, int refill) {
    stageBegin();
    {
        ExtendIO io{bounceQueue(B, bounce + 1), B.pathA, B.pathB, B.hits};
        int* c = bounceCounts(B, bounce + 1);
        persistentTrace<false>(io, c[kLive], wide, packed, &c[kExtendFetch], counter, errorFlag, stackLimit, refill);
    }
    ShadowIO io{B.shadowRay, B.shadowDir, B.shadowContrib, B.radiance};
    int* c = bounceCounts(B, bounce);
    persistentTrace<true>(io, c[kShadowRays], wide, packed, &c[kShadowFetch], shadowCounter, errorFlag, stackLimit, refill);
}

// Adds the wave's paths to their pixels' sums. A thread owns the pixel of
// path j < pixels and adds its paths j, j + pixels, ... in order, so each
// pixel's samples are added in sample order and its sums are read and written
// once per wave (88 bytes, not once per sample row).
__global__ void accumulateKernel(WaveArgs A, WavefrontBuffers B) {
    stageBegin();
    const int pixels = A.L.w * A.L.h;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= min(A.n, pixels)) return;
    const size_t i = (size_t)wavePixel(A, j);
    const int row0 = waveRow(A, j);
    const bool first = row0 == 0 && A.L.sample0 == 0;
    Accum total = first ? Accum{v3(0, 0, 0), v3(0, 0, 0), v3(0, 0, 0), 0u} : A.L.sums[i];
    float depthTotal = first ? 0.0f : A.L.depthSums[i];
    int row = row0 - 1;
    for (long long p = j; p < A.n; p += pixels, row++) addStored(B, (int)p, total, depthTotal);
    A.L.sums[i] = total;
    A.L.depthSums[i] = depthTotal;
    if (row == A.L.set.raysPerPixel - 1)
        A.L.pixels[i] = displayPixel(total, A.L.sample0 + (unsigned)A.L.set.raysPerPixel, A.L.set.exposure);
}

// ---- per-ray queries, sampler values ----
// Rays in the caller's records (RtxQuery: origin, direction, limit, 28 bytes)
// and hits in RtxHit's layout, so neither side of a call is repacked.
struct QueryIO {
    const float* q;
    float4* out;
    __device__ void load(int k, float3& o, float3& d, float& limit, unsigned&) const {
        const float* r = q + 7 * (size_t)k;
        o = v3(__ldg(r), __ldg(r + 1), __ldg(r + 2));
        d = v3(__ldg(r + 3), __ldg(r + 4), __ldg(r + 5));
        limit = __ldg(r + 6);
    }
    __device__ void store(int k, const Hit& h) const {
        out[k] = make_float4(__int_as_float(h.index), h.distance, h.u, h.v);
    }
};
template <bool ANY>
__global__ void __launch_bounds__(kTraceBlock) queryKernel(const uint4* wide, const float4* packed, const float* q,
                                                           int count, float4* out, int* fetch, int* errorFlag,
                                                           int stackLimit, int refill) {
    QueryIO io{q, out};
    persistentTrace<ANY>(io, count, wide, packed, fetch, nullptr, errorFlag, stackLimit, refill);
}

__global__ void sobolSamplesKernel(const unsigned* dirs, const unsigned* pixel, const unsigned* sample,
                                   const unsigned* seed, int count, int ndim, float* out) {
    long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (long long)count * ndim) return;
    int i = (int)(k / ndim), d = (int)(k % ndim);
    out[k] = sobolDirect(dirs, pixel[i], sample[i], seed[i], (unsigned)d);
}

// ---- denoise: guides, edge-avoiding a-trous wavelet filter, present ----
__global__ void denoisePrepareKernel(const Accum* sums, unsigned samples, int count, float4* color, float4* albedo,
                                     float4* normal) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    Accum s = sums[i];
    float inv = 1.0f / (float)samples;
    float3 c = scale(s.radiance, inv), a = scale(s.albedo, inv), n = normalize(s.normal);
    color[i] = make_float4(c.x, c.y, c.z, s.covered ? 1.0f : 0.0f);
    albedo[i] = make_float4(a.x, a.y, a.z, 0.0f);
    normal[i] = make_float4(n.x, n.y, n.z, 0.0f);
}
// x / 0.02f, correctly rounded like the division it replaces: a quotient
// estimate and one residual correction (Markstein 1990), exact against the
// division for every float in [2^-100, 2^100] (checked over all of them) and
// for 0 up to the sign; the rest take the division.
__device__ __forceinline__ float over002(float x) {
    const float magnitude = fabsf(x);
    if (magnitude == 0.0f || (magnitude >= 7.88861e-31f && magnitude <= 1.26765e30f)) {
        const float q = x * 50.0f, rest = __fmaf_rn(-q, 0.02f, x);
        return __fmaf_rn(rest, 50.0f, q);
    }
    return x / 0.02f;
}
// Weight of a tap without its kernel factors' product order changed:
// ((k * wc) * wa) * wn. invPhi is a power of two, so the product with it is
// the quotient by colorPhi.
__device__ __forceinline__ float tapWeight(float k, float4 c0, float4 a0, float4 n0, float4 c, float4 a, float4 n,
                                           float invPhi) {
    const float3 dc = v3(c.x - c0.x, c.y - c0.y, c.z - c0.z);
    const float3 da = v3(a.x - a0.x, a.y - a0.y, a.z - a0.z);
    const float wc = expf(-dot(dc, dc) * invPhi);
    const float wa = expf(over002(-dot(da, da)));
    const float wn = powf(fmaxf(0.0f, n.x * n0.x + n.y * n0.y + n.z * n0.z), 64.0f);
    return k * wc * wa * wn;
}
// One pass of the a-trous filter: 25 taps `step` pixels apart. The pixels of
// one residue (x mod step, y mod step) form a dense lattice on which the taps
// are the neighbours within two, so a block takes a 32 x 16 tile of one
// lattice with its two-point border into shared memory. A tap's weight is the
// same seen from both ends (squares and products of the same pairs), so each
// pair's two exponentials and its power are computed once, by the end that
// comes first, and the 25 weighted sums read them: 14.4 evaluations per
// pixel instead of 25. Bound by those evaluations (about 150 instructions
// each). 1283 x 717, five passes: 695 us with one thread per pixel evaluating
// every tap, 496 us now (85 at step 1, 117 at step 16, whose lattices of 81 x 45
// points fill 96 x 48).
constexpr int kAtX = 32, kAtY = 16, kAtW = kAtX + 4, kAtH = kAtY + 4, kAtOwners = kAtW * (kAtY + 2), kAtThreads = 256;
constexpr size_t kAtrousSmem = sizeof(float4) * 3 * kAtW * kAtH + sizeof(float) * 12 * kAtOwners;
// Index of forward offset (dx, dy): dy = 0 and dx = 1, 2; dy = 1, 2 and dx = -2 .. 2.
__host__ __device__ constexpr int atOffset(int dx, int dy) { return dy == 0 ? dx - 1 : 2 + 5 * (dy - 1) + dx + 2; }
__global__ void __launch_bounds__(kAtThreads) atrousKernel(const float4* in, const float4* albedo, const float4* normal,
                                                           float4* out, int w, int h, int step, float invPhi) {
    extern __shared__ float4 atSmem[];
    float4 *sc = atSmem, *sa = sc + kAtW * kAtH, *sn = sa + kAtW * kAtH;
    float* sw = reinterpret_cast<float*>(sn + kAtW * kAtH);  // [12][kAtOwners]; below 0: no such tap
    const int rx = blockIdx.x % step, ry = blockIdx.y % step;
    const int gx0 = (int)(blockIdx.x / step) * kAtX - 2, gy0 = (int)(blockIdx.y / step) * kAtY - 2;
    for (int i = threadIdx.x; i < kAtW * kAtH; i += kAtThreads) {
        const int gx = gx0 + i % kAtW, gy = gy0 + i / kAtW;
        const int x = gx * step + rx, y = gy * step + ry;
        float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f), a = c, n = c;
        if (gx >= 0 && gy >= 0 && x < w && y < h) {
            const int j = y * w + x;
            c = in[j]; a = albedo[j]; n = normal[j];
        }
        sc[i] = c; sa[i] = a; sn[i] = n;
    }
    __syncthreads();
    constexpr float kernel[3] = {3.0f / 8.0f, 1.0f / 4.0f, 1.0f / 16.0f};
    // Pair weights, by the pixels (owners) whose forward taps they are; a pair
    // with neither end in the tile is not needed.
    for (int i = threadIdx.x; i < kAtOwners; i += kAtThreads) {
        const int lx = i % kAtW, ly = i / kAtW;
        const bool mine = lx >= 2 && lx < kAtX + 2 && ly >= 2;
        const float4 c0 = sc[i], a0 = sa[i], n0 = sn[i];
#pragma unroll
        for (int dy = 0; dy <= 2; dy++)
#pragma unroll
            for (int dx = -2; dx <= 2; dx++) {
                if (dy == 0 && dx <= 0) continue;
                const int px = lx + dx, py = ly + dy;
                if (!mine && !(px >= 2 && px < kAtX + 2 && py >= 2 && py < kAtY + 2)) continue;
                const int j = py * kAtW + px;
                const float4 c = sc[j];
                float weight = -1.0f;
                if (c0.w != 0.0f && c.w != 0.0f)
                    weight = tapWeight(kernel[dx < 0 ? -dx : dx] * kernel[dy], c0, a0, n0, c, sa[j], sn[j], invPhi);
                sw[atOffset(dx, dy) * kAtOwners + i] = weight;
            }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kAtX * kAtY; i += kAtThreads) {
        const int lx = i % kAtX + 2, ly = i / kAtX + 2, at = ly * kAtW + lx;
        const int x = (gx0 + lx) * step + rx, y = (gy0 + ly) * step + ry;
        if (x >= w || y >= h) continue;
        const float4 c0 = sc[at];
        if (c0.w == 0.0f) { out[y * w + x] = c0; continue; }
        float3 sum = v3(0, 0, 0);
        float wsum = 0.0f;
#pragma unroll
        for (int dy = -2; dy <= 2; dy++)
#pragma unroll
            for (int dx = -2; dx <= 2; dx++) {
                const bool forward = dy > 0 || (dy == 0 && dx > 0);
                const float4 c = sc[at + dy * kAtW + dx];
                float wk;
                if (dx == 0 && dy == 0) wk = tapWeight(kernel[0] * kernel[0], c0, sa[at], sn[at], c0, sa[at], sn[at], invPhi);
                else if (forward) wk = sw[atOffset(forward ? dx : 1, forward ? dy : 0) * kAtOwners + at];
                else wk = sw[atOffset(forward ? 1 : -dx, forward ? 0 : -dy) * kAtOwners + at + dy * kAtW + dx];
                if (wk < 0.0f) continue;
                sum = add(sum, scale(v3(c.x, c.y, c.z), wk));
                wsum += wk;
            }
        float3 r = wsum > 0 ? scale(sum, 1.0f / wsum) : v3(c0.x, c0.y, c0.z);
        out[y * w + x] = make_float4(r.x, r.y, r.z, c0.w);
    }
}
__global__ void denoisePresentKernel(const Accum* sums, const float4* color, int count, float exposure, uchar4* pixels) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float4 c4 = color[i];
    float3 c = sums[i].covered ? v3(c4.x, c4.y, c4.z) : v3(0, 0, 0);
    pixels[i] = make_uchar4(tonemap(c.x, exposure), tonemap(c.y, exposure), tonemap(c.z, exposure), 255);
}

__global__ void aovKernel(const Accum* sums, const float* depthSums, unsigned samples, int count, float* aov) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    Accum s = sums[i];
    float inv = 1.0f / (float)samples;
    float3 c = scale(s.radiance, inv), a = scale(s.albedo, inv), n = normalize(s.normal);
    float* o = aov + (size_t)i * 10;
    o[0] = c.x; o[1] = c.y; o[2] = c.z;
    o[3] = a.x; o[4] = a.y; o[5] = a.z;
    o[6] = n.x; o[7] = n.y; o[8] = n.z;
    o[9] = depthSums[i] * inv;
}
// Coverage as bytes from the network's input kernel: the 40-byte sums' flag cost
// their 83 MB again at 1080p (26 us, now 14).
__global__ void presentRadianceKernel(const unsigned char* coverage, const float* radiance, int count, float exposure,
                                      uchar4* pixels) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float* r = radiance + (size_t)i * 3;
    float3 c = coverage[i] ? v3(r[0], r[1], r[2]) : v3(0, 0, 0);
    pixels[i] = make_uchar4(tonemap(c.x, exposure), tonemap(c.y, exposure), tonemap(c.z, exposure), 255);
}

inline int blocks(long long n, int b) { return (int)((n + b - 1) / b); }

int smCount() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    return sms;
}
// Resident blocks of a traversal kernel, for a grid of exactly one wave.
template <class K>
int traceBlocks(K kernel, size_t smem) {
    int perSm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, kTraceBlock, smem) != cudaSuccess || perSm <= 0)
        perSm = 1;
    return smCount() * perSm;
}
constexpr size_t kTraceSmem = traceSharedBytes(kTraceBlock);

// Launches a stage; dependent: with programmatic stream serialization (see
// stageBegin).
template <class... P, class... A>
void launchStage(bool dependent, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace

cudaError_t allocWavefront(WavefrontBuffers& b, int capacity) {
    freeWavefront(b);
    size_t n = (size_t)capacity;
    cudaError_t e;
#define RT_ALLOC(p, count) if ((e = rt::deviceAlloc(reinterpret_cast<void**>(&(p)), sizeof(*(p)) * (count))) != cudaSuccess) { freeWavefront(b); return e; }
    RT_ALLOC(b.pathA, n); RT_ALLOC(b.pathB, n); RT_ALLOC(b.pathC, n);
    RT_ALLOC(b.radiance, n); RT_ALLOC(b.albedo, n); RT_ALLOC(b.normal, n); RT_ALLOC(b.hits, n);
    RT_ALLOC(b.queue[0], n); RT_ALLOC(b.queue[1], n);
    RT_ALLOC(b.shadowRay, n); RT_ALLOC(b.shadowDir, n); RT_ALLOC(b.shadowContrib, n);
    RT_ALLOC(b.counts, kWaveCounts);
#undef RT_ALLOC
    b.capacity = capacity;
    return cudaSuccess;
}
void freeWavefront(WavefrontBuffers& b) {
    void* owned[] = {b.pathA, b.pathB, b.pathC, b.radiance, b.albedo, b.normal, b.hits, b.queue[0], b.queue[1],
                     b.shadowRay, b.shadowDir, b.shadowContrib, b.counts};
    for (void* p : owned)
        if (p) rt::deviceFree(p);
    b = WavefrontBuffers{};
}

cudaError_t buildSobolTables(const unsigned* dirs, unsigned sample0, int rpp, unsigned seed, unsigned* passXor,
                             unsigned* seedHash, unsigned long long* status, cudaStream_t stream) {
    int total = (rpp + 1) * kSobolDims;
    sobolTablesKernel<<<blocks(total, 256), 256, 0, stream>>>(dirs, sample0, rpp, seed, passXor, seedHash, status);
    return cudaGetLastError();
}

cudaError_t launchMegakernel(const RenderLaunch& L, cudaStream_t stream, int* launches) {
    size_t smem = sizeof(uint2) * kStackCapacity * kMegaBlock;
    static bool configured = false;
    if (!configured) {
        cudaFuncSetAttribute(megakernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        configured = true;
    }
    dim3 grid((L.w + kTileX - 1) / kTileX, (L.h + kTileY - 1) / kTileY);
    megakernel<<<grid, kMegaBlock, smem, stream>>>(L);
    if (launches) *launches = 1;
    return cudaGetLastError();
}

cudaError_t launchWavefront(const RenderLaunch& L, WavefrontBuffers& B, const TraceTuning& tuning, cudaStream_t stream,
                            int* launches, float* extendMs, float* shadowMs, bool timing, float* primaryMs,
                            const WaveOverlap* overlap) {
    static int extendBlocks = 0, shadowBlocks = 0, bothBlocks = 0;
    if (!extendBlocks) {
        bothBlocks = traceBlocks(shadowExtendKernel, kTraceSmem);
        shadowBlocks = traceBlocks(shadowKernel, kTraceSmem);
        extendBlocks = traceBlocks(extendKernel, kTraceSmem);
    }
    const size_t smem = kTraceSmem;
    const int stackLimit = tuning.stackLimit;
    const int refill = tuning.refill;
    const int shadeBlocks = smCount() * kShadePerSm;
    int pixels = L.w * L.h;
    int n = 0;
    static thread_local std::vector<cudaEvent_t> pool;
    struct Mark { cudaEvent_t a, b; int kind; };  // 0 primary closest-hit, 1 secondary, 2 shadow
    std::vector<Mark> marks;
    auto event = [&](size_t k) -> cudaEvent_t {
        while (pool.size() <= k) { cudaEvent_t e; cudaEventCreate(&e); pool.push_back(e); }
        return pool[k];
    };
    size_t ev = 0;
    const int total = pixels * L.set.raysPerPixel;  // paths of the pass (at most 4096^2 * 16 < 2^31)
    // A pass of one wave has nothing on another lane to overlap with: its
    // stages overlap with one another instead (dependent launches, shadow rays
    // traced with the next bounce's closest hits), unless they are timed apart.
    const bool single = total <= B.capacity, chained = single && !timing;
    if (single) overlap = nullptr;
    int nLanes = overlap ? std::max(1, std::min(overlap->lanes, kMaxLanes)) : 1;
    for (int k = 1; k < nLanes; k++)
        if (!overlap->buffers[k - 1] || !overlap->streams[k - 1] || overlap->buffers[k - 1]->capacity != B.capacity)
            nLanes = 1;
    const bool two = nLanes > 1;
    WavefrontBuffers* lanes[kMaxLanes] = {&B};
    cudaStream_t laneStream[kMaxLanes] = {stream};
    for (int k = 1; k < nLanes; k++) {
        lanes[k] = overlap->buffers[k - 1];
        laneStream[k] = overlap->streams[k - 1];
    }
    if (two) {
        cudaEventRecord(overlap->fork, stream);  // the other lanes start after the work queued so far
        for (int k = 1; k < nLanes; k++) cudaStreamWaitEvent(laneStream[k], overlap->fork, 0);
    }
    int wave = 0;
    {
        for (int start = 0; start < total; start += B.capacity, wave++) {
            WavefrontBuffers& W = *lanes[wave % nLanes];
            cudaStream_t ws = laneStream[wave % nLanes];
            WaveArgs A{L, start, total - start < B.capacity ? total - start : B.capacity};
            launchStage(chained, generateKernel, blocks(A.n, 256), 256, 0, ws, A, W);
            n++;
            if (chained) {
                const uint4* wide = L.scene.wide;
                const float4* packed = L.scene.packed;
                unsigned long long* rays = L.counters;
                launchStage(true, extendKernel, extendBlocks, kTraceBlock, smem, ws, wide, packed, W, 0, &rays[0], L.errorFlag,
                            stackLimit, refill);
                for (int bounce = 0; bounce < L.set.maxBounces; bounce++) {
                    launchStage(true, shadeKernel, shadeBlocks, kShadeBlock, 0, ws, A, W, bounce);
                    if (bounce + 1 < L.set.maxBounces)
                        launchStage(true, shadowExtendKernel, bothBlocks, kTraceBlock, smem, ws, wide, packed, W, bounce, &rays[2],
                                    &rays[1], L.errorFlag, stackLimit, refill);
                    else
                        launchStage(true, shadowKernel, shadowBlocks, kTraceBlock, smem, ws, wide, packed, W, bounce, &rays[2],
                                    L.errorFlag, stackLimit, refill);
                }
                launchStage(true, accumulateKernel, blocks(std::min(A.n, pixels), 256), 256, 0, ws, A, W);
                n += 2 + 2 * L.set.maxBounces;
                break;
            }
            for (int bounce = 0; bounce < L.set.maxBounces; bounce++) {
                Mark m{nullptr, nullptr, bounce == 0 ? 0 : 1};
                if (timing) { m.a = event(ev++); m.b = event(ev++); cudaEventRecord(m.a, ws); }
                extendKernel<<<extendBlocks, kTraceBlock, smem, ws>>>(L.scene.wide, L.scene.packed, W, bounce,
                                                                      &L.counters[bounce == 0 ? 0 : 1], L.errorFlag,
                                                                      stackLimit, refill);
                if (timing) { cudaEventRecord(m.b, ws); marks.push_back(m); }
                shadeKernel<<<shadeBlocks, kShadeBlock, 0, ws>>>(A, W, bounce);
                Mark s{nullptr, nullptr, 2};
                if (timing) { s.a = event(ev++); s.b = event(ev++); cudaEventRecord(s.a, ws); }
                shadowKernel<<<shadowBlocks, kTraceBlock, smem, ws>>>(L.scene.wide, L.scene.packed, W, bounce,
                                                                      &L.counters[2], L.errorFlag, stackLimit, refill);
                if (timing) { cudaEventRecord(s.b, ws); marks.push_back(s); }
                n += 3;
            }
            // Samples of a pixel are added in sample order: after the
            // previous wave's accumulation, whichever lane ran it.
            if (two && wave > 0) cudaStreamWaitEvent(ws, overlap->accumulated, 0);
            accumulateKernel<<<blocks(std::min(A.n, pixels), 256), 256, 0, ws>>>(A, W);
            n++;
            if (two) cudaEventRecord(overlap->accumulated, ws);
        }
    }
    for (int k = 1; k < nLanes; k++) {
        cudaEventRecord(overlap->joins[k - 1], laneStream[k]);
        cudaStreamWaitEvent(stream, overlap->joins[k - 1], 0);
    }
    cudaError_t e = cudaGetLastError();
    if (launches) *launches = n;
    if (timing && e == cudaSuccess) {
        e = cudaStreamSynchronize(stream);
        float kindMs[3] = {0, 0, 0};
        for (const Mark& m : marks) {
            float ms = 0;
            cudaEventElapsedTime(&ms, m.a, m.b);
            kindMs[m.kind] += ms;
        }
        if (extendMs) *extendMs = kindMs[0] + kindMs[1];
        if (shadowMs) *shadowMs = kindMs[2];
        if (primaryMs) *primaryMs = kindMs[0];
    }
    return e;
}

cudaError_t launchQueries(const uint4* wide, const float4* packed, const float* queries, int count, int any,
                          float4* hits, int* status, const TraceTuning& tuning, cudaStream_t stream) {
    const int stackLimit = tuning.stackLimit;
    const int refill = tuning.refill;
    int *errorFlag = status, *fetch = status + 1;
    cudaError_t e = cudaMemsetAsync(status, 0, 2 * sizeof(int), stream);
    if (e != cudaSuccess) return e;
    // Up to four warps' worth of rays per SM run as blocks of one warp, spread
    // over the SMs (4,096 rays: 128 SMs of one warp instead of 32 of four);
    // more rays in blocks of 128, one wave of resident blocks at most.
    const int block = count <= smCount() * kTraceBlock ? 32 : kTraceBlock;
    const size_t smem = traceSharedBytes(block);
    static int mostAny = traceBlocks(queryKernel<true>, kTraceSmem), most = traceBlocks(queryKernel<false>, kTraceSmem);
    const int want = blocks(count, block), grid = block == 32 ? want : std::min(any ? mostAny : most, want);
    (any ? queryKernel<true> : queryKernel<false>)<<<grid, block, smem, stream>>>(wide, packed, queries, count, hits, fetch,
                                                                                 errorFlag, stackLimit, refill);
    return cudaGetLastError();
}

cudaError_t launchSobolSamples(const unsigned* dirs, const unsigned* pixel, const unsigned* sample, const unsigned* seed,
                               int count, int ndim, float* out, cudaStream_t stream) {
    long long total = (long long)count * ndim;
    sobolSamplesKernel<<<blocks(total, 256), 256, 0, stream>>>(dirs, pixel, sample, seed, count, ndim, out);
    return cudaGetLastError();
}

// Denoised linear radiance as 3 floats per pixel (uncovered pixels 0, as the
// display shows them): src holds srcStride floats per pixel.
__global__ void denoisedRgbKernel(const Accum* sums, const float* src, int srcStride, int count, float* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float* r = src + (size_t)i * srcStride;
    const bool covered = sums[i].covered != 0u;
    out[3 * (size_t)i] = covered ? r[0] : 0.0f;
    out[3 * (size_t)i + 1] = covered ? r[1] : 0.0f;
    out[3 * (size_t)i + 2] = covered ? r[2] : 0.0f;
}

cudaError_t launchDenoisedRgb(const Accum* sums, const float* src, int srcStride, int count, float* out,
                              cudaStream_t stream) {
    denoisedRgbKernel<<<blocks(count, 256), 256, 0, stream>>>(sums, src, srcStride, count, out);
    return cudaGetLastError();
}

cudaError_t launchDenoise(const Accum* sums, unsigned samples, int w, int h, float exposure, float4* work,
                          uchar4* pixels, cudaStream_t stream) {
    int count = w * h;
    float4 *color = work, *albedo = work + count, *normal = work + 2 * (size_t)count, *tmp = work + 3 * (size_t)count;
    denoisePrepareKernel<<<blocks(count, 256), 256, 0, stream>>>(sums, samples, count, color, albedo, normal);
    cudaError_t e = cudaFuncSetAttribute(atrousKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAtrousSmem);
    if (e != cudaSuccess) return e;
    float4 *src = color, *dst = tmp;
    float invPhi = 2.0f;  // colour bandwidth 0.5, halved every pass
    for (int it = 0; it < kAtrousPasses; it++) {
        const int step = 1 << it;
        auto tiles = [&](int size, int tile) { return step * (((size + step - 1) / step + tile - 1) / tile); };
        atrousKernel<<<dim3(tiles(w, kAtX), tiles(h, kAtY)), kAtThreads, kAtrousSmem, stream>>>(src, albedo, normal, dst, w, h,
                                                                                              step, invPhi);
        float4* t = src; src = dst; dst = t;
        invPhi *= 2.0f;
    }
    denoisePresentKernel<<<blocks(count, 256), 256, 0, stream>>>(sums, src, count, exposure, pixels);
    return cudaGetLastError();
}

cudaError_t launchAovs(const Accum* sums, const float* depthSums, unsigned samples, int count, float* aov,
                       cudaStream_t stream) {
    aovKernel<<<blocks(count, 256), 256, 0, stream>>>(sums, depthSums, samples, count, aov);
    return cudaGetLastError();
}
cudaError_t launchPresentRadiance(const unsigned char* coverage, const float* radiance, int count, float exposure, uchar4* pixels,
                                  cudaStream_t stream) {
    presentRadianceKernel<<<blocks(count, 256), 256, 0, stream>>>(coverage, radiance, count, exposure, pixels);
    return cudaGetLastError();
}

}  // namespace rt
