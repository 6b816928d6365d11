// GPU BVH construction.
//
// Stage 1, binned SAH (level-synchronous, all nodes of one depth per pass).
// The split rules are the reference's (Native/bvh.cuh:35-105), evaluated with
// the same floating-point expressions so every decision matches:
//   - primitive box padded by 1e-5 + 1e-6 * max|coord| per axis, centroid
//     (a + b + c) / 3 of the unpadded corners (bvh.cuh:38-48);
//   - leaf when count <= 4 or depth == 32 (bvh.cuh:64);
//   - 12 centroid bins per axis, axes with centroid extent <= 1e-12 skipped,
//     bin = min(11, max(0, int((c - min) * (12 / extent)))) (bvh.cuh:53-76);
//   - split cost A(node) + A(L) nL + A(R) nR against leaf cost A(node) n,
//     strict "<" so the first minimum in (axis, bin) order wins (bvh.cuh:66-91);
//   - partition by bin <= best (bvh.cuh:94-98).
// Binning and box unions are min/max/counts, which are order independent, so
// the tree (node boxes, ranges, counts, depth) equals the reference's. The
// partition here is stable (prefix sums) where the reference uses
// std::partition, so only the order of triangles inside a leaf can differ.
// A final pass renumbers nodes into the reference's depth-first numbering
// (children allocated in pairs when their parent splits), so the node array
// is the reference's node array.
//
// Stage 2, collapse into 8-wide compressed nodes: each wide node greedily
// opens its largest-area interior descendant while the children still fit in
// eight slots; leaves become groups of up to three triangles. Children are
// assigned to slots by ray octant and quantised outward to 8 bits per plane.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "rt_build.cuh"
#include "rt_collapse.cuh"

namespace rt {
namespace {

constexpr int kBins = 12;          // bvh.cuh:29
constexpr int kLeafSize = 4;       // bvh.cuh:64
constexpr int kScanBlock = 1024;   // elements per scan block
constexpr int kBinBlock = 256;
constexpr int kBinPer = 8;         // most positions per thread in the binning pass
// Tasks of at most kSmallTask primitives are binned by one
// block (binKernel); larger ones by position blocks (binLarge).
constexpr int kSmallTask = 2048;
// Tasks of at most kSearchTask are searched by splitKernel straight from their
// primitives and need no bins (1.3M primitives in tasks of 128-500: 110-190 us
// of binning a level against about 25 for the search).
constexpr int kSearchTask = 512;
// Tasks of at most this many primitives are finished by one warp each, down to
// their leaves (subtreeKernel).
constexpr int kSubtree = 32;
// Levels (binned SAH, or wide collapse) queued per host read of the counts:
// a first batch of 8, then 4 at a time. A level without tasks costs its
// launches only.
constexpr int kLevelBatch = 8, kNextLevels = 4;

struct Task {
    int node, first, count, depth;
    float lo[3], hi[3], clo[3], chi[3];
};
struct BinAcc { unsigned count; float lo[3], hi[3], clo[3], chi[3]; };
struct Split { int axis, bin, leftCount, childTask[2]; };
// A finished subtree: its root's raw node, and its other nodes at [base, base +
// 2 * interior) in the reference's depth-first order.
struct Subtree { int root, base, interior; };
// counters: [0] raw nodes, [1] (unused), [2] maximum depth, [3] error, [4]
// subtree tasks, [5] finished blocks of a scan. Errors: 1 nodes, 2 tasks, 3
// wide nodes or triangles, 4 jobs past their capacity; 5 a position, 6 and 7 a
// node outside its range (nothing is written there).
constexpr int kCounters = 8;

__device__ __forceinline__ void atomicMinFloat(float* a, float v) {
    if (v >= 0.0f) atomicMin(reinterpret_cast<int*>(a), __float_as_int(v));
    else atomicMax(reinterpret_cast<unsigned*>(a), __float_as_uint(v));
}
__device__ __forceinline__ void atomicMaxFloat(float* a, float v) {
    if (v >= 0.0f) atomicMax(reinterpret_cast<int*>(a), __float_as_int(v));
    else atomicMin(reinterpret_cast<unsigned*>(a), __float_as_uint(v));
}
RT_HD int binOf(float c, float lo, float s) {
    int b = (int)((c - lo) * s);
    return b < 0 ? 0 : (b > kBins - 1 ? kBins - 1 : b);
}
// Half surface area with the reference's expression (bvh.cuh:20-23).
RT_HD float halfArea(const float lo[3], const float hi[3]) {
    float x = fmaxf(0.0f, hi[0] - lo[0]), y = fmaxf(0.0f, hi[1] - lo[1]), z = fmaxf(0.0f, hi[2] - lo[2]);
    return x * y + x * z + y * z;
}
__device__ __forceinline__ void growBox(float lo[3], float hi[3], const float olo[3], const float ohi[3]) {
    for (int a = 0; a < 3; a++) { lo[a] = fminf(lo[a], olo[a]); hi[a] = fmaxf(hi[a], ohi[a]); }
}

// ---- primitive boxes and root bounds ----
// Grows the root's box and centroid box by a block's values (v: low, high,
// centroid low and high of this thread's primitive): one set of atomics per
// block of 256 threads (per warp they serialised on the root's addresses, 484
// us for 1.3M primitives).
__device__ __forceinline__ void growRoot(float (&v)[12], Task* root) {
    __shared__ float part[8][12];
    for (int off = 16; off > 0; off >>= 1)
        for (int k = 0; k < 12; k++) {
            float o = __shfl_xor_sync(0xFFFFFFFFu, v[k], off);
            v[k] = ((k / 3) & 1) ? fmaxf(v[k], o) : fminf(v[k], o);
        }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 12; k++) part[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 12) {
        const int k = threadIdx.x;
        float x = part[0][k];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) x = ((k / 3) & 1) ? fmaxf(x, part[w][k]) : fminf(x, part[w][k]);
        float* at = k < 3 ? &root->lo[k] : k < 6 ? &root->hi[k - 3] : k < 9 ? &root->clo[k - 6] : &root->chi[k - 9];
        if ((k / 3) & 1) atomicMaxFloat(at, x);
        else atomicMinFloat(at, x);
    }
}
__global__ void primBoxesKernel(const SceneTri* tris, int n, float4* plo, float4* phi, float4* cent, Task* root) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    float v[12];
    for (int k = 0; k < 3; k++) { v[k] = FLT_MAX; v[3 + k] = -FLT_MAX; v[6 + k] = FLT_MAX; v[9 + k] = -FLT_MAX; }
    if (i < n) {
        const SceneTri& t = tris[i];
        float3 o = t.origin;
        float3 b = v3(o.x + t.edge1.x, o.y + t.edge1.y, o.z + t.edge1.z);
        float3 c = v3(o.x + t.edge2.x, o.y + t.edge2.y, o.z + t.edge2.z);
        float lo[3], hi[3], ce[3];
        for (int a = 0; a < 3; a++) {
            float oa = comp(o, a), ba = comp(b, a), ca = comp(c, a);
            lo[a] = fminf(fminf(fminf(FLT_MAX, oa), ba), ca);
            hi[a] = fmaxf(fmaxf(fmaxf(-FLT_MAX, oa), ba), ca);
            ce[a] = (oa + ba + ca) / 3.0f;
            float pad = 1e-5f + 1e-6f * fmaxf(fabsf(lo[a]), fabsf(hi[a]));
            lo[a] -= pad; hi[a] += pad;
        }
        plo[i] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        phi[i] = make_float4(hi[0], hi[1], hi[2], 0.0f);
        cent[i] = make_float4(ce[0], ce[1], ce[2], 0.0f);
        for (int k = 0; k < 3; k++) { v[k] = lo[k]; v[3 + k] = hi[k]; v[6 + k] = ce[k]; v[9 + k] = ce[k]; }
    }
    growRoot(v, root);
}

// Traversal-tree primitives: each triangle cut into `pieces` slabs along the
// longest axis of its box; a piece's box bounds the part of the triangle in
// its slab (vertices inside it and the edges' crossings of its planes), padded
// like the reference pads triangle boxes (bvh.cuh:46-47). The padding exceeds
// the rounding of the clipping, so every point of the triangle lies in the
// padded box of a piece containing it, and the union of the pieces' boxes
// covers the triangle's padded box's content that traversal can reach.
// Pieces of one triangle: the half area of its box over its own area tells
// how much empty space the box holds. Well-shaped triangles (ratio below 12;
// all but a fraction of a percent of ordinary meshes' triangles) stay whole;
// slivers get floor(ratio / 6) pieces, at most maxPieces.
__device__ int piecesOf(const SceneTri& t, int maxPieces) {
    const float3 e1 = t.edge1, e2 = t.edge2;
    const float ex = fmaxf(fmaxf(0.0f, e1.x), e2.x) - fminf(fminf(0.0f, e1.x), e2.x);
    const float ey = fmaxf(fmaxf(0.0f, e1.y), e2.y) - fminf(fminf(0.0f, e1.y), e2.y);
    const float ez = fmaxf(fmaxf(0.0f, e1.z), e2.z) - fminf(fminf(0.0f, e1.z), e2.z);
    const float boxArea = ex * ey + ey * ez + ex * ez;
    const float3 c = cross(e1, e2);
    const float triArea = 0.5f * sqrtf(dot(c, c));
    if (!(triArea > 0.0f) || !(boxArea < FLT_MAX)) return 1;
    const float k = boxArea / triArea / 6.0f;
    return k >= (float)maxPieces ? maxPieces : (k >= 2.0f ? (int)k : 1);
}
__global__ void pieceCountKernel(const SceneTri* tris, int n, int maxPieces, unsigned* counts) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) counts[i] = (unsigned)piecesOf(tris[i], maxPieces);
}
// primTri[first piece of i + s] = i, from the exclusive scan of the counts
// (block-local prefix plus the block's total).
__global__ void pieceFillKernel(const unsigned* counts, const unsigned* prefix, const unsigned* blockSums, int n,
                                int* primTri, int* total) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned first = prefix[i] + blockSums[i / kScanBlock];
    if (primTri)
        for (unsigned s = 0; s < counts[i]; s++) primTri[first + s] = i;
    if (i == n - 1) *total = (int)(first + counts[i]);
}

__global__ void splitBoxesKernel(const SceneTri* tris, const int* primTri, int nPrims, int maxPieces, float4* plo,
                                 float4* phi, float4* cent, Task* root) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    float v[12];
    for (int k = 0; k < 3; k++) { v[k] = FLT_MAX; v[3 + k] = -FLT_MAX; v[6 + k] = FLT_MAX; v[9 + k] = -FLT_MAX; }
    if (r < nPrims) {
        const int i = primTri[r];
        const SceneTri& t = tris[i];
        const int pieces = piecesOf(t, maxPieces);
        int s = 0;  // which piece: primitives of a triangle are consecutive
        while (s < r && s < pieces - 1 && primTri[r - s - 1] == i) s++;
        float3 P[3] = {t.origin, v3(t.origin.x + t.edge1.x, t.origin.y + t.edge1.y, t.origin.z + t.edge1.z),
                       v3(t.origin.x + t.edge2.x, t.origin.y + t.edge2.y, t.origin.z + t.edge2.z)};
        float tlo[3], thi[3];
        for (int a = 0; a < 3; a++) {
            tlo[a] = fminf(fminf(comp(P[0], a), comp(P[1], a)), comp(P[2], a));
            thi[a] = fmaxf(fmaxf(comp(P[0], a), comp(P[1], a)), comp(P[2], a));
        }
        int ax = 0;
        for (int a = 1; a < 3; a++) if (thi[a] - tlo[a] > thi[ax] - tlo[ax]) ax = a;
        const float ext = thi[ax] - tlo[ax];
        const float t0 = s == 0 ? tlo[ax] : tlo[ax] + ext * ((float)s / (float)pieces);
        const float t1 = s == pieces - 1 ? thi[ax] : tlo[ax] + ext * ((float)(s + 1) / (float)pieces);
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        auto grow = [&](float3 q) {
            for (int a = 0; a < 3; a++) { lo[a] = fminf(lo[a], comp(q, a)); hi[a] = fmaxf(hi[a], comp(q, a)); }
        };
        for (int e = 0; e < 3; e++) {
            const float3 p = P[e], q = P[(e + 1) % 3];
            const float pa = comp(p, ax), qa = comp(q, ax);
            if (pa >= t0 && pa <= t1) grow(p);
            for (int side = 0; side < 2; side++) {
                const float plane = side ? t1 : t0;
                if ((pa < plane && qa > plane) || (pa > plane && qa < plane)) {
                    const float u = (plane - pa) / (qa - pa);
                    float3 x = v3(p.x + u * (q.x - p.x), p.y + u * (q.y - p.y), p.z + u * (q.z - p.z));
                    if (ax == 0) x.x = plane; else if (ax == 1) x.y = plane; else x.z = plane;
                    grow(x);
                }
            }
        }
        float ce[3];
        for (int a = 0; a < 3; a++) {
            if (!(lo[a] <= hi[a])) { lo[a] = tlo[a]; hi[a] = thi[a]; }  // nothing collected: whole box
            float pad = 1e-5f + 1e-6f * fmaxf(fabsf(tlo[a]), fabsf(thi[a]));
            lo[a] -= pad; hi[a] += pad;
            ce[a] = 0.5f * (lo[a] + hi[a]);
        }
        plo[r] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        phi[r] = make_float4(hi[0], hi[1], hi[2], 0.0f);
        cent[r] = make_float4(ce[0], ce[1], ce[2], 0.0f);
        for (int k = 0; k < 3; k++) { v[k] = lo[k]; v[3 + k] = hi[k]; v[6 + k] = ce[k]; v[9 + k] = ce[k]; }
    }
    growRoot(v, root);
}

__global__ void iotaKernel(int* a, int n, int value0, int* b, int bValue) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { a[i] = i + value0; if (b) b[i] = bValue; }
}

// Level counts (taskCount[0] open tasks, taskCount[1] of them larger than
// kSmallTask) live on the device, so levels are queued without the host
// reading them: per-task kernels loop over the device count.
__device__ __forceinline__ void clearBins(BinAcc* bins, const int* taskCount, const Task* tasks) {
    if (!taskCount[1]) return;
    const int count = taskCount[0] * 3 * kBins;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        if (tasks[i / (3 * kBins)].count <= kSmallTask) continue;
        BinAcc& b = bins[i];
        b.count = 0;
        for (int a = 0; a < 3; a++) { b.lo[a] = FLT_MAX; b.hi[a] = -FLT_MAX; b.clo[a] = FLT_MAX; b.chi[a] = -FLT_MAX; }
    }
}
__global__ void clearBinsKernel(BinAcc* bins, const int* taskCount, const Task* tasks) { clearBins(bins, taskCount, tasks); }

// Floats as integers of the same order (-0 below +0, as the atomics above
// order them), so warp reductions can use the integer min/max instructions.
__device__ __forceinline__ int orderedKey(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float keyFloat(int k) { return __int_as_float(k >= 0 ? k : k ^ 0x7FFFFFFF); }

// A bin in shared memory, its values as ordered keys. A value that does not
// improve the bin costs a read and a comparison: after the first few
// primitives nearly all of them, where adding each with atomics (13 per
// primitive and axis, the lanes of one bin one after another) bound binning
// (110-200 us a level for 1.3M primitives, 2.5 of the 6.1 ms build). Counts
// and minima/maxima do not depend on the order of accumulation, and a stale
// read only makes an atomic that changes nothing.
struct BinKeys { unsigned count; int lo[3], hi[3], clo[3], chi[3]; };
struct PrimKeys { int lo[3], hi[3], c[3]; };
__device__ __forceinline__ PrimKeys primKeys(float4 lo, float4 hi, float4 c) {
    return PrimKeys{{orderedKey(lo.x), orderedKey(lo.y), orderedKey(lo.z)},
                    {orderedKey(hi.x), orderedKey(hi.y), orderedKey(hi.z)},
                    {orderedKey(c.x), orderedKey(c.y), orderedKey(c.z)}};
}
__device__ __forceinline__ void clearKeys(BinKeys& b) {
    b.count = 0;
    for (int a = 0; a < 3; a++) {
        b.lo[a] = b.clo[a] = orderedKey(FLT_MAX);
        b.hi[a] = b.chi[a] = orderedKey(-FLT_MAX);
    }
}
__device__ __forceinline__ void lower(int* at, int v) {
    if (v < *reinterpret_cast<volatile int*>(at)) atomicMin(at, v);
}
__device__ __forceinline__ void raise(int* at, int v) {
    if (v > *reinterpret_cast<volatile int*>(at)) atomicMax(at, v);
}
__device__ __forceinline__ void addToBin(BinKeys& b, const PrimKeys& p) {
    atomicAdd(&b.count, 1u);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        lower(&b.lo[a], p.lo[a]);
        raise(&b.hi[a], p.hi[a]);
        lower(&b.clo[a], p.c[a]);
        raise(&b.chi[a], p.c[a]);
    }
}
__device__ __forceinline__ BinAcc toBin(const BinKeys& k) {
    BinAcc b;
    b.count = k.count;
    for (int a = 0; a < 3; a++) {
        b.lo[a] = keyFloat(k.lo[a]); b.hi[a] = keyFloat(k.hi[a]);
        b.clo[a] = keyFloat(k.clo[a]); b.chi[a] = keyFloat(k.chi[a]);
    }
    return b;
}

// Bins every primitive of the open tasks above kSmallTask. A block takes a
// chunk of at most kSmallTask positions, which therefore meets at most two of
// them, at its ends: their bins are two sets of shared ones (sb, 2 x 3 kBins),
// added to the global bins at the end.
__device__ void binLarge(const int* order, const int* posTask, const float4* cent, const float4* plo, const float4* phi,
                         const Task* tasks, int nPos, BinAcc* bins, const int* taskCount, BinKeys* sb, int perThread) {
    __shared__ int ends[2];
    if (!taskCount[1]) return;  // no task above kSmallTask at this level
    const int base = blockIdx.x * kBinBlock * perThread, end = min(base + kBinBlock * perThread, nPos);
    if (threadIdx.x < 2) {
        const int t = posTask[threadIdx.x ? end - 1 : base];
        ends[threadIdx.x] = t >= 0 && tasks[t].count > kSmallTask ? t : -1;
    }
    for (int i = threadIdx.x; i < 2 * 3 * kBins; i += kBinBlock) clearKeys(sb[i]);
    __syncthreads();
    for (int k = 0; k < perThread; k++) {
        const int j = base + k * kBinBlock + threadIdx.x;
        if (j >= end) break;
        const int t = posTask[j];
        if (t < 0 || (t != ends[0] && t != ends[1])) continue;
        BinKeys* set = sb + (t == ends[0] ? 0 : 3 * kBins);
        const Task& T = tasks[t];
        const int prim = order[j];
        const float4 c = cent[prim];
        const PrimKeys keys = primKeys(plo[prim], phi[prim], c);
        for (int a = 0; a < 3; a++) {
            const float extent = T.chi[a] - T.clo[a];
            if (extent <= 1e-12f) continue;
            const float ca = a == 0 ? c.x : (a == 1 ? c.y : c.z);
            addToBin(set[a * kBins + binOf(ca, T.clo[a], kBins / extent)], keys);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * 3 * kBins; i += kBinBlock) {
        const int s = i / (3 * kBins), t = ends[s];
        if (t < 0 || !sb[i].count) continue;
        const BinAcc b = toBin(sb[i]);
        BinAcc* d = &bins[(size_t)t * 3 * kBins + i % (3 * kBins)];
        atomicAdd(&d->count, b.count);
        for (int a = 0; a < 3; a++) {
            atomicMinFloat(&d->lo[a], b.lo[a]); atomicMaxFloat(&d->hi[a], b.hi[a]);
            atomicMinFloat(&d->clo[a], b.clo[a]); atomicMaxFloat(&d->chi[a], b.chi[a]);
        }
    }
}

// Adds primitives first + lane, first + lane + step, ... of task T to a warp's
// own bins.
__device__ __forceinline__ void binRange(const int* order, const float4* cent, const float4* plo, const float4* phi,
                                         const Task& T, int first, int step, BinKeys* my, int lane) {
    for (int i = lane; i < 3 * kBins; i += 32) clearKeys(my[i]);
    __syncwarp();
    float scale[3];
    for (int a = 0; a < 3; a++) {
        float extent = T.chi[a] - T.clo[a];
        scale[a] = extent <= 1e-12f ? 0.0f : kBins / extent;
    }
    for (int j = T.first + first + lane; j < T.first + T.count; j += step) {
        const int prim = order[j];
        const float4 c = cent[prim];
        const PrimKeys keys = primKeys(plo[prim], phi[prim], c);
        for (int a = 0; a < 3; a++) {
            if (scale[a] == 0.0f) continue;
            const float ca = a == 0 ? c.x : (a == 1 ? c.y : c.z);
            addToBin(my[a * kBins + binOf(ca, T.clo[a], scale[a])], keys);
        }
    }
    __syncwarp();
}

// The bins of a level's tasks in one launch. Blocks below largeBlocks: position
// chunks of the large tasks. The others go over the tasks of kSearchTask to
// kSmallTask primitives, a block each with warp-private bins in shared
// memory, written out with plain stores, so these bins need no clearing and no global atomics. Bins hold a count and
// minima/maxima, so the order of accumulation does not change them.
__global__ void __launch_bounds__(kBinBlock) binKernel(const int* order, const int* posTask, const float4* cent,
                                                       const float4* plo, const float4* phi, const Task* tasks,
                                                       int nPos, BinAcc* bins, const int* taskCount, int largeBlocks,
                                                       int perThread) {
    __shared__ BinKeys sb[8][3 * kBins];
    if ((int)blockIdx.x < largeBlocks) {
        binLarge(order, posTask, cent, plo, phi, tasks, nPos, bins, taskCount, sb[0], perThread);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nTasks = taskCount[0], first = (int)blockIdx.x - largeBlocks, stride = (int)gridDim.x - largeBlocks;
    for (int t = first; t < nTasks; t += stride) {
        const int n = tasks[t].count;
        if (n <= kSearchTask || n > kSmallTask) continue;
        const Task T = tasks[t];
        binRange(order, cent, plo, phi, T, warp * 32, 256, sb[warp], lane);
        __syncthreads();
        for (int i = threadIdx.x; i < 3 * kBins; i += kBinBlock) {
            BinKeys b = sb[0][i];
            for (int w = 1; w < 8; w++) {
                const BinKeys& o = sb[w][i];
                b.count += o.count;
                for (int a = 0; a < 3; a++) {
                    b.lo[a] = min(b.lo[a], o.lo[a]); b.hi[a] = max(b.hi[a], o.hi[a]);
                    b.clo[a] = min(b.clo[a], o.clo[a]); b.chi[a] = max(b.chi[a], o.chi[a]);
                }
            }
            bins[(size_t)t * 3 * kBins + i] = toBin(b);
        }
        __syncthreads();
    }
}

// Raises the maximum depth; most calls find it there and leave the address alone.
__device__ __forceinline__ void deepen(int* counters, int depth) {
    if (*reinterpret_cast<volatile int*>(&counters[2]) < depth) atomicMax(&counters[2], depth);
}

// A level's splits, one warp per open task: the reference's SAH sweep, then
// node records and the children's tasks. Candidate j = (axis, cut) sits on
// lane j, which unites the boxes on both sides: of its axis's 12 bins, or for
// tasks of at most kSearchTask of the primitives themselves (the same minima
// and maxima), staged 32 at a time in shared memory. The 33rd candidate (the
// z axis's last cut) is a uniform second step or a reduction over the lanes.
// The first minimum in (axis, cut) order wins, as in the reference's loop.
// (One thread per task walked the 36 bins in about 11 us whatever the level
// held.)
// Node and task numbers within a level come in atomic order; nodes are
// renumbered to the reference's order after the build, and tasks carry their
// own ranges. nextCount: the next level's open tasks and those above
// kSmallTask; counters as listed at kCounters.
__global__ void __launch_bounds__(128) splitKernel(const int* order, const float4* cent, const float4* plo, const float4* phi,
                                                   const Task* tasks, const int* taskCount, const BinAcc* bins, Split* splits,
                                                   BinNode* nodes, int* counters, int* nextCount, Task* nextTasks,
                                                   Task* subtrees, int nodeCapacity, int taskCapacity, int subtreeCapacity,
                                                   int leafSize) {
    __shared__ __align__(16) BinAcc sb[4][3 * kBins];
    const unsigned full = 0xFFFFFFFFu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nTasks = taskCount[0], warps = (int)gridDim.x * 4;
    BinAcc* B = sb[warp];
    for (int t = (int)blockIdx.x * 4 + warp; t < nTasks; t += warps) {
        const Task T = tasks[t];
        const float nodeArea = halfArea(T.lo, T.hi), unsplit = nodeArea * T.count;
        bool valid[3];
        for (int a = 0; a < 3; a++) valid[a] = !(T.chi[a] - T.clo[a] <= 1e-12f);
        // Boxes (low, high) and counts on both sides of this lane's candidate,
        // and of the last one.
        const int axis = lane / 11, cut = lane % 11;
        float box[2][6], lastBox[2][6];
        int count[2], lastCount[2];
        auto reset = [](float (&b)[2][6], int (&n)[2]) {
            for (int s = 0; s < 2; s++) {
                for (int k = 0; k < 3; k++) { b[s][k] = FLT_MAX; b[s][3 + k] = -FLT_MAX; }
                n[s] = 0;
            }
        };
        auto reduceMin = [&](float v) { return keyFloat(__reduce_min_sync(full, orderedKey(v))); };
        auto reduceMax = [&](float v) { return keyFloat(__reduce_max_sync(full, orderedKey(v))); };
        const bool search = T.count <= kSearchTask;
        float scale[3];
        for (int a = 0; a < 3; a++) scale[a] = valid[a] ? kBins / (T.chi[a] - T.clo[a]) : 0.0f;
        auto axisOf = [](float x, float y, float z, int a) { return a == 0 ? x : (a == 1 ? y : z); };
        auto binAt = [&](float4 c, int a) { return valid[a] ? binOf(axisOf(c.x, c.y, c.z, a), T.clo[a], scale[a]) : 0; };
        __syncwarp();
        reset(box, count);
        reset(lastBox, lastCount);
        if (search) {
            float4* stage = reinterpret_cast<float4*>(B);  // 32 low corners (w: the three bins), 32 high
            for (int base = 0; base < T.count; base += 32) {
                const int n = min(32, T.count - base);
                __syncwarp();
                if (lane < n) {
                    const int prim = order[T.first + base + lane];
                    const float4 c = cent[prim];
                    float4 lo = plo[prim], hi = phi[prim];
                    const int b2 = binAt(c, 2);
                    lo.w = __int_as_float(binAt(c, 0) | binAt(c, 1) << 4 | b2 << 8);
                    stage[lane] = lo;
                    stage[32 + lane] = hi;
                    const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
                    if (b2 <= kBins - 2) { growBox(lastBox[0], lastBox[0] + 3, l, h); lastCount[0]++; }
                    else { growBox(lastBox[1], lastBox[1] + 3, l, h); lastCount[1]++; }
                }
                __syncwarp();
                for (int i = 0; i < n; i++) {
                    const float4 lo = stage[i], hi = stage[32 + i];
                    const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
                    if (((__float_as_int(lo.w) >> (4 * axis)) & 15) <= cut) { growBox(box[0], box[0] + 3, l, h); count[0]++; }
                    else { growBox(box[1], box[1] + 3, l, h); count[1]++; }
                }
            }
            for (int s = 0; s < 2; s++) {
                for (int k = 0; k < 3; k++) {
                    lastBox[s][k] = reduceMin(lastBox[s][k]);
                    lastBox[s][3 + k] = reduceMax(lastBox[s][3 + k]);
                }
                lastCount[s] = __reduce_add_sync(full, lastCount[s]);
            }
        } else {
            constexpr int kWords = 3 * kBins * (int)(sizeof(BinAcc) / 4);
            for (int i = lane; i < kWords; i += 32)
                reinterpret_cast<unsigned*>(B)[i] = reinterpret_cast<const unsigned*>(bins + (size_t)t * 3 * kBins)[i];
            __syncwarp();
            auto sweep = [&](float (&to)[2][6], int (&n)[2], int a, int c) {
                for (int b = 0; b < kBins; b++) {
                    const BinAcc& o = B[a * kBins + b];
                    if (!o.count) continue;
                    if (b <= c) { growBox(to[0], to[0] + 3, o.lo, o.hi); n[0] += (int)o.count; }
                    else { growBox(to[1], to[1] + 3, o.lo, o.hi); n[1] += (int)o.count; }
                }
            };
            sweep(box, count, axis, cut);
            sweep(lastBox, lastCount, 2, kBins - 2);
        }
        // Costs are sums of areas, not negative: their bits order like them. A
        // candidate that is out (no extent, an empty side, not below the leaf's
        // cost) is above every cost, infinite ones among them.
        auto candidateBits = [&](const float (&b)[2][6], const int (&n)[2], bool axisValid) {
            if (!axisValid || !n[0] || !n[1]) return full;
            const float cost = nodeArea + halfArea(b[0], b[0] + 3) * n[0] + halfArea(b[1], b[1] + 3) * n[1];
            return cost < unsplit ? __float_as_uint(cost) : full;
        };
        const unsigned last = candidateBits(lastBox, lastCount, valid[2]);
        const unsigned bits = candidateBits(box, count, axis == 0 ? valid[0] : axis == 1 ? valid[1] : valid[2]);
        const unsigned best = __reduce_min_sync(full, bits);
        int bestAxis = -1, bestBin = -1, winner = -1;
        if (best != full) {
            winner = __ffs(__ballot_sync(full, bits == best)) - 1;
            bestAxis = winner / 11;
            bestBin = winner % 11;
        }
        if (last < best) { bestAxis = 2; bestBin = kBins - 2; winner = -1; }
        if (bestAxis < 0) {
            if (lane == 0) {
                nodes[T.node] = BinNode{v3(T.lo[0], T.lo[1], T.lo[2]), T.first, v3(T.hi[0], T.hi[1], T.hi[2]), T.count};
                splits[t] = Split{-1, -1, 0, {-1, -1}};
                deepen(counters, T.depth);
            }
            continue;
        }
        // Lane s < 2 makes child s: the winning candidate's box and count, and
        // its centroid box over its bins or primitives.
        int child = 0, leftCount = 0;
        Task C;
        C.count = 0;
        bool open = false, small = false;
        for (int s = 0; s < 2; s++) {
            float w[6];
            for (int k = 0; k < 6; k++) w[k] = winner < 0 ? lastBox[s][k] : __shfl_sync(full, box[s][k], winner);
            const int n = winner < 0 ? lastCount[s] : __shfl_sync(full, count[s], winner);
            if (lane == s) {
                for (int k = 0; k < 3; k++) { C.lo[k] = w[k]; C.hi[k] = w[3 + k]; }
                C.count = n;
            }
        }
        float cen[2][6];
        {
            int unused[2];
            reset(cen, unused);
        }
        if (search) {
            for (int i = lane; i < T.count; i += 32) {
                const float4 c = cent[order[T.first + i]];
                const float p[3] = {c.x, c.y, c.z};
                if (binAt(c, bestAxis) <= bestBin) growBox(cen[0], cen[0] + 3, p, p);
                else growBox(cen[1], cen[1] + 3, p, p);
            }
            for (int s = 0; s < 2; s++)
                for (int k = 0; k < 3; k++) {
                    cen[s][k] = reduceMin(cen[s][k]);
                    cen[s][3 + k] = reduceMax(cen[s][3 + k]);
                }
        } else {
            for (int b = 0; b < kBins; b++) {
                const BinAcc& o = B[bestAxis * kBins + b];
                if (!o.count) continue;
                if (b <= bestBin) growBox(cen[0], cen[0] + 3, o.clo, o.chi);
                else growBox(cen[1], cen[1] + 3, o.clo, o.chi);
            }
        }
        if (lane < 2) {
            for (int k = 0; k < 3; k++) { C.clo[k] = lane ? cen[1][k] : cen[0][k]; C.chi[k] = lane ? cen[1][3 + k] : cen[0][3 + k]; }
            C.depth = T.depth + 1;
            open = !(C.count <= leafSize || C.depth == kBinaryMaxDepth);
            small = open && C.count <= kSubtree;
            open = open && !small;
        }
        if (lane == 0) {
            child = atomicAdd(&counters[0], 2);
            deepen(counters, T.depth + 1);
        }
        child = __shfl_sync(full, child, 0);
        leftCount = __shfl_sync(full, C.count, 0);
        if (child + 2 > nodeCapacity) {
            if (lane == 0) { atomicExch(&counters[3], 1); splits[t] = Split{-1, -1, 0, {-1, -1}}; }
            continue;
        }
        int taskIndex = -1;
        if (lane < 2) {
            C.node = child + lane;
            C.first = T.first + (lane ? leftCount : 0);
            if (small) {
                const int m = atomicAdd(&counters[4], 1);
                if (m >= subtreeCapacity) atomicExch(&counters[3], 2);
                else subtrees[m] = C;
            } else if (open) {
                const int k = atomicAdd(&nextCount[0], 1);
                if (C.count > kSmallTask) atomicAdd(&nextCount[1], 1);
                if (k >= taskCapacity) atomicExch(&counters[3], 2);
                else { nextTasks[k] = C; taskIndex = k; }
            } else {
                nodes[C.node] = BinNode{v3(C.lo[0], C.lo[1], C.lo[2]), C.first, v3(C.hi[0], C.hi[1], C.hi[2]), C.count};
            }
        }
        const int rightTask = __shfl_sync(full, taskIndex, 1);
        if (lane == 0) {
            nodes[T.node] = BinNode{v3(T.lo[0], T.lo[1], T.lo[2]), child, v3(T.hi[0], T.hi[1], T.hi[2]), 0};
            splits[t] = Split{bestAxis, bestBin, leftCount, {taskIndex, rightTask}};
        }
    }
}

// 1 when position j's primitive goes to its task's left child.
__device__ __forceinline__ unsigned leftFlag(int j, const int* order, const int* posTask, const float4* cent,
                                             const Task* tasks, const Split* splits) {
    const int t = posTask[j];
    if (t < 0) return 0u;
    const Split S = splits[t];
    if (S.axis < 0) return 0u;
    const Task& T = tasks[t];
    float lo = T.clo[S.axis];
    float s = kBins / (T.chi[S.axis] - lo);
    float4 c = cent[order[j]];
    float ca = S.axis == 0 ? c.x : (S.axis == 1 ? c.y : c.z);
    return binOf(ca, lo, s) <= S.bin ? 1u : 0u;
}

// Exclusive scan of 4 consecutive values per thread over a block of 256, block
// total to *sum (thread 7's store); returns the thread's prefix.
__device__ __forceinline__ unsigned scanBlock(const unsigned (&v)[4], unsigned* warpSums, unsigned* sum) {
    const unsigned local = v[0] + v[1] + v[2] + v[3];
    unsigned incl = local;
    for (int off = 1; off < 32; off <<= 1) {
        unsigned o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if ((threadIdx.x & 31) >= off) incl += o;
    }
    if ((threadIdx.x & 31) == 31) warpSums[threadIdx.x >> 5] = incl;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned w = threadIdx.x < 8 ? warpSums[threadIdx.x] : 0u, wi = w;
        for (int off = 1; off < 8; off <<= 1) {
            unsigned o = __shfl_up_sync(0xFFFFFFFFu, wi, off);
            if (threadIdx.x >= off) wi += o;
        }
        if (threadIdx.x < 8) warpSums[threadIdx.x] = wi - w;
        if (threadIdx.x == 7) *sum = wi;
    }
    __syncthreads();
    return warpSums[threadIdx.x >> 5] + incl - local;
}
// Exclusive scan of the block totals, in place, by one block of 256 threads.
__device__ void scanTotals(unsigned* sums, int count) {
    __shared__ unsigned carry;
    __shared__ unsigned warpSums[8];
    __shared__ unsigned total;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < count; base += 1024) {
        unsigned v[4];
        const int j = base + threadIdx.x * 4;
        for (int k = 0; k < 4; k++) v[k] = j + k < count ? __ldcg(sums + j + k) : 0u;
        unsigned run = carry + scanBlock(v, warpSums, &total);
        for (int k = 0; k < 4; k++) {
            if (j + k < count) sums[j + k] = run;
            run += v[k];
        }
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
}
// The block that finishes last scans the totals (done: zero before the launch
// and after it). Every block of the grid calls this once its total is stored.
__device__ void scanTotalsLast(unsigned* sums, int count, int* done) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(done, 1) == count - 1 ? 1 : 0;
        if (last) *done = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    scanTotals(sums, count);
}
__global__ void __launch_bounds__(256) scanBlocksKernel(const unsigned* in, unsigned* data, int n, unsigned* blockSums,
                                                        int* done) {
    __shared__ unsigned warpSums[8];
    const int j = blockIdx.x * kScanBlock + threadIdx.x * 4;
    unsigned v[4];
    for (int k = 0; k < 4; k++) v[k] = j + k < n ? in[j + k] : 0u;
    unsigned run = scanBlock(v, warpSums, &blockSums[blockIdx.x]);
    for (int k = 0; k < 4; k++) {
        if (j + k < n) data[j + k] = run;
        run += v[k];
    }
    scanTotalsLast(blockSums, (int)gridDim.x, done);
}
// A level's partition, first half: every position's side and the scan of the
// sides. Also records the node count after the level's splits (the first node
// of the next depth) and clears the bins of the next level's large tasks.
__global__ void __launch_bounds__(256) partitionKernel(const int* order, const int* posTask, const float4* cent,
                                                       const Task* tasks, const Split* splits, int n, unsigned* flags,
                                                       unsigned* prefix, unsigned* blockSums, int* counters, int* levelStart,
                                                       const int* taskCount, const int* nextCount, const Task* nextTasks,
                                                       BinAcc* bins) {
    __shared__ unsigned warpSums[8];
    if (blockIdx.x == 0 && threadIdx.x == 0) *levelStart = counters[0];
    if (!taskCount[0]) return;  // a level past the last: nothing moves
    clearBins(bins, nextCount, nextTasks);
    const int j = blockIdx.x * kScanBlock + threadIdx.x * 4;
    unsigned v[4];
    for (int k = 0; k < 4; k++) {
        v[k] = j + k < n ? leftFlag(j + k, order, posTask, cent, tasks, splits) : 0u;
        if (j + k < n) flags[j + k] = v[k];
    }
    unsigned run = scanBlock(v, warpSums, &blockSums[blockIdx.x]);
    for (int k = 0; k < 4; k++) {
        if (j + k < n) prefix[j + k] = run;
        run += v[k];
    }
    scanTotalsLast(blockSums, (int)gridDim.x, &counters[5]);
}
// The consumer adds both levels: prefix(j) = data[j] + sums[j / kScanBlock].

__global__ void scatterKernel(const int* order, const int* posTask, const Task* tasks, const Split* splits,
                              const unsigned* flags, const unsigned* prefix, const unsigned* blockSums, int nPos,
                              int* orderNext, int* posTaskNext, const int* taskCount, int* error) {
    if (!taskCount[0]) return;
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nPos) return;
    int t = posTask[j];
    int prim = order[j];
    if (t < 0 || splits[t].axis < 0) { orderNext[j] = prim; posTaskNext[j] = -1; return; }
    const Task& T = tasks[t];
    Split S = splits[t];
    unsigned pj = prefix[j] + blockSums[j / kScanBlock];
    unsigned p0 = prefix[T.first] + blockSums[T.first / kScanBlock];
    int leftRank = (int)(pj - p0);
    bool left = flags[j] != 0u;
    int dst = left ? T.first + leftRank : T.first + S.leftCount + ((j - T.first) - leftRank);
    if (dst < T.first || dst >= T.first + T.count) { atomicExch(error, 5); return; }
    orderNext[dst] = prim;
    posTaskNext[dst] = S.childTask[left ? 0 : 1];
}

// ---- subtrees of at most kSubtree primitives ----
constexpr int kSubtreeWarps = 4;
struct SubtreeEntry { unsigned mask; int first, depth, slot; float lo[3], hi[3], clo[3], chi[3]; };
struct SubtreeShared {
    float4 lo[kSubtree], hi[kSubtree];    // primitive boxes; lo.w: the bins of the three axes, 4 bits each
    BinNode nodes[2 * (kSubtree - 1)];    // all nodes but the root, in depth-first order (children in pairs)
    SubtreeEntry stack[kSubtree];         // right siblings not yet visited
};

// One warp builds the whole subtree of a small task; lane l holds primitive l
// of the task's range and a node is a mask of lanes. The partition is stable,
// so a node's primitives are its lanes in order and nothing moves until the
// leaves write the range. The split search is the reference's over its 33
// candidates (3 axes x 11 bins): candidate j on lane j, which unites the
// boxes on both sides over the node's primitives (minima and maxima, the
// same values as uniting bins), the 33rd by warp reductions; the first
// minimum wins as in splitTask. Nodes are visited depth first, left before
// right, so a split's rank among the subtree's splits is the reference's
// numbering of its children.
// This replaces about 12 levels of global binning, splitting and partitioning
// (3.0 of the 9.2 ms of the 1.3M-piece tree, 0.9 of 1.4 ms at 8,000 triangles).
// Bound by instructions, about 300 per split and 20 more per primitive.
__global__ void __launch_bounds__(32 * kSubtreeWarps) subtreeKernel(int* order, const float4* cent, const float4* plo,
                                                                    const float4* phi, const Task* tasks, int* counters,
                                                                    BinNode* nodes, int nodeCapacity, int leafSize,
                                                                    int* interiorOf, Subtree* done) {
    __shared__ SubtreeShared shared[kSubtreeWarps];
    const unsigned full = 0xFFFFFFFFu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    SubtreeShared& S = shared[warp];
    const int count = counters[4];
    const int axis = lane / 11, cut = lane % 11;  // this lane's candidate
    auto axisOf = [](float x, float y, float z, int a) { return a == 0 ? x : (a == 1 ? y : z); };
    for (int t = blockIdx.x * kSubtreeWarps + warp; t < count; t += gridDim.x * kSubtreeWarps) {
        const Task T = tasks[t];
        const bool have = lane < T.count;
        int prim = 0;
        float4 lo = make_float4(0, 0, 0, 0), hi = lo, c = lo;
        if (have) {
            prim = order[T.first + lane];
            lo = plo[prim]; hi = phi[prim]; c = cent[prim];
        }
        __syncwarp();
        S.lo[lane] = lo;
        S.hi[lane] = hi;
        SubtreeEntry N;
        N.mask = __ballot_sync(full, have);
        N.first = T.first; N.depth = T.depth; N.slot = -1;
        for (int a = 0; a < 3; a++) { N.lo[a] = T.lo[a]; N.hi[a] = T.hi[a]; N.clo[a] = T.clo[a]; N.chi[a] = T.chi[a]; }
        BinNode root;
        int interior = 0, top = 0, depth = T.depth;
        // Writes a node's record (children by their place in S.nodes).
        auto record = [&](int slot, const float* l, const float* h, int first, int n) {
            const BinNode r{v3(l[0], l[1], l[2]), first, v3(h[0], h[1], h[2]), n};
            if (slot < 0) root = r;
            else if (lane == 0) S.nodes[slot] = r;
        };
        auto leaf = [&](unsigned mask, int first) {
            if ((mask >> lane) & 1u) order[first + __popc(mask & below)] = prim;
        };
        auto reduceMin = [&](float v, bool in) { return keyFloat(__reduce_min_sync(full, in ? orderedKey(v) : 0x7FFFFFFF)); };
        auto reduceMax = [&](float v, bool in) { return keyFloat(__reduce_max_sync(full, in ? orderedKey(v) : (int)0x80000000)); };
        for (;;) {
            const int n = __popc(N.mask);
            const bool mine = (N.mask >> lane) & 1u;
            int bestAxis = -1, bestCut = 0;
            float side[2][6];  // the winning candidate's boxes: low, high
            if (n > leafSize && N.depth != kBinaryMaxDepth) {
                const float nodeArea = halfArea(N.lo, N.hi), unsplit = nodeArea * n;
                int bin[3] = {0, 0, 0};
                bool valid[3];
                for (int a = 0; a < 3; a++) {
                    const float extent = N.chi[a] - N.clo[a];
                    valid[a] = !(extent <= 1e-12f);
                    if (valid[a]) bin[a] = binOf(axisOf(c.x, c.y, c.z, a), N.clo[a], kBins / extent);
                }
                __syncwarp();
                reinterpret_cast<int*>(&S.lo[lane])[3] = bin[0] | bin[1] << 4 | bin[2] << 8;
                __syncwarp();
                float L[6], R[6];
                for (int k = 0; k < 3; k++) { L[k] = R[k] = FLT_MAX; L[3 + k] = R[3 + k] = -FLT_MAX; }
                int nl = 0;
                for (unsigned m = N.mask; m; m &= m - 1u) {
                    const int i = __ffs(m) - 1;
                    const float4 pl = S.lo[i], ph = S.hi[i];
                    if (((__float_as_int(pl.w) >> (4 * axis)) & 15) <= cut) {
                        L[0] = fminf(L[0], pl.x); L[1] = fminf(L[1], pl.y); L[2] = fminf(L[2], pl.z);
                        L[3] = fmaxf(L[3], ph.x); L[4] = fmaxf(L[4], ph.y); L[5] = fmaxf(L[5], ph.z);
                        nl++;
                    } else {
                        R[0] = fminf(R[0], pl.x); R[1] = fminf(R[1], pl.y); R[2] = fminf(R[2], pl.z);
                        R[3] = fmaxf(R[3], ph.x); R[4] = fmaxf(R[4], ph.y); R[5] = fmaxf(R[5], ph.z);
                    }
                }
                const int nr = n - nl;
                const bool usable = (axis == 0 ? valid[0] : axis == 1 ? valid[1] : valid[2]) && nl && nr;
                const float cost = nodeArea + halfArea(L, L + 3) * nl + halfArea(R, R + 3) * nr;
                // Costs are sums of areas, not negative: their bits order like them.
                const unsigned bits = usable && cost < unsplit ? __float_as_uint(cost) : full;
                unsigned best = __reduce_min_sync(full, bits);
                if (best != full) {
                    const int winner = __ffs(__ballot_sync(full, bits == best)) - 1;
                    bestAxis = winner / 11;
                    bestCut = winner % 11;
                    for (int k = 0; k < 6; k++) {
                        side[0][k] = __shfl_sync(full, L[k], winner);
                        side[1][k] = __shfl_sync(full, R[k], winner);
                    }
                }
                // Candidate 32: the last cut of the z axis.
                const unsigned low = __ballot_sync(full, mine && bin[2] <= kBins - 2), high = N.mask & ~low;
                if (valid[2] && low && high) {
                    float l[6], r[6];
                    const bool inLow = (low >> lane) & 1u, inHigh = (high >> lane) & 1u;
                    l[0] = reduceMin(lo.x, inLow); l[1] = reduceMin(lo.y, inLow); l[2] = reduceMin(lo.z, inLow);
                    l[3] = reduceMax(hi.x, inLow); l[4] = reduceMax(hi.y, inLow); l[5] = reduceMax(hi.z, inLow);
                    r[0] = reduceMin(lo.x, inHigh); r[1] = reduceMin(lo.y, inHigh); r[2] = reduceMin(lo.z, inHigh);
                    r[3] = reduceMax(hi.x, inHigh); r[4] = reduceMax(hi.y, inHigh); r[5] = reduceMax(hi.z, inHigh);
                    const float last = nodeArea + halfArea(l, l + 3) * __popc(low) + halfArea(r, r + 3) * __popc(high);
                    if (last < unsplit && __float_as_uint(last) < best) {
                        bestAxis = 2;
                        bestCut = kBins - 2;
                        for (int k = 0; k < 6; k++) { side[0][k] = l[k]; side[1][k] = r[k]; }
                    }
                }
                if (bestAxis >= 0) {
                    const int b = bestAxis == 0 ? bin[0] : bestAxis == 1 ? bin[1] : bin[2];
                    const unsigned left = __ballot_sync(full, mine && b <= bestCut);
                    const int pair = 2 * interior++;
                    record(N.slot, N.lo, N.hi, pair, 0);
                    const int childDepth = N.depth + 1;
                    depth = max(depth, childDepth);
                    const unsigned masks[2] = {left, N.mask & ~left};
                    const int firsts[2] = {N.first, N.first + __popc(left)};
                    bool go = false;
                    SubtreeEntry next;
                    for (int s = 1; s >= 0; s--) {
                        const int k = __popc(masks[s]);
                        if (k <= leafSize || childDepth == kBinaryMaxDepth) {
                            record(pair + s, side[s], side[s] + 3, firsts[s], k);
                            leaf(masks[s], firsts[s]);
                            continue;
                        }
                        SubtreeEntry E;
                        const bool in = (masks[s] >> lane) & 1u;
                        E.mask = masks[s]; E.first = firsts[s]; E.depth = childDepth; E.slot = pair + s;
                        for (int a = 0; a < 3; a++) { E.lo[a] = side[s][a]; E.hi[a] = side[s][3 + a]; }
                        E.clo[0] = reduceMin(c.x, in); E.clo[1] = reduceMin(c.y, in); E.clo[2] = reduceMin(c.z, in);
                        E.chi[0] = reduceMax(c.x, in); E.chi[1] = reduceMax(c.y, in); E.chi[2] = reduceMax(c.z, in);
                        if (s == 1) {
                            if (lane == 0) S.stack[top] = E;
                            top++;
                        } else {
                            next = E;
                            go = true;
                        }
                    }
                    if (go) { N = next; continue; }
                }
            }
            if (bestAxis < 0) {
                record(N.slot, N.lo, N.hi, N.first, n);
                leaf(N.mask, N.first);
            }
            if (!top) break;
            top--;
            __syncwarp();
            N = S.stack[top];
            __syncwarp();
        }
        int base = 0;
        if (lane == 0) {
            if (interior) base = atomicAdd(&counters[0], 2 * interior);
            deepen(counters, depth);
        }
        base = __shfl_sync(full, base, 0);
        __syncwarp();
        if (base + 2 * interior > nodeCapacity) {
            if (lane == 0) atomicExch(&counters[3], 1);
            continue;
        }
        if (lane == 0) {
            if (root.count == 0) root.first += base;
            nodes[T.node] = root;
            if (interiorOf) interiorOf[T.node] = interior;
            if (done) done[t] = Subtree{T.node, base, interior};
        }
        for (int i = lane; i < 2 * interior; i += 32) {
            BinNode r = S.nodes[i];
            if (r.count == 0) r.first += base;
            nodes[base + i] = r;
        }
    }
}

// ---- renumbering into the reference's depth-first numbering ----
// Nodes below topNodes were made level by level; an interior one whose
// children lie above is the root of a finished subtree, whose interior count
// subtreeKernel has set and whose other nodes keep their order.
__global__ void subtreeInteriorKernel(const BinNode* nodes, int begin, int end, int topNodes, int* interior) {
    int i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    const BinNode& n = nodes[i];
    if (n.count > 0) interior[i] = 0;
    else if (n.first < topNodes) interior[i] = 1 + interior[n.first] + interior[n.first + 1];
}
__global__ void preorderKernel(const BinNode* nodes, int begin, int end, int topNodes, int count, const int* interior,
                               int* rank, int* newIndex, int* error) {
    int i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    const BinNode& n = nodes[i];
    if (n.count > 0 || n.first >= topNodes) return;
    int c = n.first, r = rank[i];
    if (c < 1 || c + 1 >= topNodes || r < 0 || 2 + 2 * r >= count) { atomicExch(error, 6); return; }
    newIndex[c] = 1 + 2 * r;
    newIndex[c + 1] = 2 + 2 * r;
    rank[c] = r + 1;
    rank[c + 1] = r + 1 + interior[c];
}
__global__ void renumberKernel(const BinNode* nodes, int topNodes, int count, const int* newIndex, const int* rank,
                               BinNode* out, int* error) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= topNodes) return;
    BinNode n = nodes[i];
    if (n.count == 0) n.first = n.first < topNodes ? newIndex[n.first] : 1 + 2 * rank[i];
    int dst = newIndex[i];
    if (dst < 0 || dst >= count || (n.count == 0 && (n.first < 1 || n.first + 1 >= count))) { atomicExch(error, 7); return; }
    out[dst] = n;
}
// The nodes of the finished subtrees, a warp each: those of a root of rank r
// follow from 1 + 2 r.
__global__ void placeSubtreesKernel(const BinNode* nodes, const Subtree* done, const int* counters, const int* rank, int count,
                                    BinNode* out, int* error) {
    const int warps = (int)(gridDim.x * blockDim.x) >> 5, lane = threadIdx.x & 31;
    for (int t = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < counters[4]; t += warps) {
        const Subtree S = done[t];
        const int to = 1 + 2 * rank[S.root];
        if (to < 1 || to + 2 * S.interior > count) {
            if (lane == 0 && S.interior) atomicExch(error, 7);
            continue;
        }
        for (int i = lane; i < 2 * S.interior; i += 32) {
            BinNode n = nodes[S.base + i];
            if (n.count == 0) n.first += to - S.base;
            out[to + i] = n;
        }
    }
}

// ---- collapse into wide nodes (logic in rt_collapse.cuh) ----
// planCollapse and emitCollapse with eight lanes per job (four jobs a warp):
// a lane holds one candidate while the node's children are opened, then one
// kid: its box, triangles, slot and quantised planes. One thread per job
// walked some hundred dependent loads one after another (65 us a level even
// for a few jobs). The choices, their order and the arithmetic are
// planCollapse's; within a level storage comes in job order per warp.
// jobCount: this wide level's jobs; nextCount receives the next level's.
struct CollapseShared { WideNode node[4]; };
__global__ void __launch_bounds__(64) collapseKernel(const BinNode* bn, const int* order, const float4* plo, const float4* phi,
                               const SceneTri* tris, const Job* jobs, const int* jobCount, Job* nextJobs,
                               int* nextCount, WideNode* wide, float4* packed, int* counters, int wideCapacity,
                               int jobCapacity, int triCapacity, int group, int width, const int* primTri) {
    __shared__ CollapseShared shared[2];
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7, slotOfJob = lane >> 3;
    const int nJobs = *jobCount;
    auto get = [&](auto v, int from) { return __shfl_sync(full, v, from, 8); };
    auto sumAll = [&](int v) { for (int o = 4; o; o >>= 1) v += __shfl_xor_sync(full, v, o, 8); return v; };
    auto orAll = [&](unsigned v) { for (int o = 4; o; o >>= 1) v |= __shfl_xor_sync(full, v, o, 8); return v; };
    auto minAll = [&](float v) { for (int o = 4; o; o >>= 1) v = fminf(v, __shfl_xor_sync(full, v, o, 8)); return v; };
    auto maxAll = [&](float v) { for (int o = 4; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(full, v, o, 8)); return v; };
    // The lane of the best key (the larger where MAX, the lower lane of
    // equals), or -1 when no lane takes part.
    auto pick = [&](float key, bool in, bool largest) {
        int at = in ? sub : -1;
        for (int o = 4; o; o >>= 1) {
            const float k = __shfl_xor_sync(full, key, o, 8);
            const int l = __shfl_xor_sync(full, at, o, 8);
            const bool better = l >= 0 && (at < 0 || (largest ? k > key : k < key) || (k == key && l < at));
            if (better) { key = k; at = l; }
        }
        return at;
    };
    for (int base = ((int)blockIdx.x * 2 + warp) * 4; base < nJobs; base += (int)gridDim.x * 8) {
        const int j = base + slotOfJob;
        const bool have = j < nJobs;
        Job J = have ? jobs[j] : Job{1, 0, 0, 0, 0};
        if (have && J.kind == 0 && bn[J.node].count > 0) { J.kind = 1; J.first = bn[J.node].first; J.count = bn[J.node].count; }
        const bool inner = have && J.kind == 0;
        // Candidates: lane i holds the i-th.
        BinNode cand{};
        int node = -1, slots = 0, opened = 0, nc = inner ? 2 : 0;
        float area = -1.0f;
        auto place = [&](int n) {
            node = n;
            cand = bn[n];
            slots = slotsOf(cand, group, width);
            area = -1.0f;
            opened = 0;
            if (cand.count == 0) {
                const float lo[3] = {cand.low.x, cand.low.y, cand.low.z}, hi[3] = {cand.high.x, cand.high.y, cand.high.z};
                area = collapseHalfArea(lo, hi);
                opened = slotsOf(bn[cand.first], group, width) + slotsOf(bn[cand.first + 1], group, width);
            }
        };
        if (inner && sub < 2) place(bn[J.node].first + sub);
        for (bool more = inner;;) {
            const int total = sumAll(slots);
            const bool can = more && node >= 0 && area > -1.0f && nc < width && total - 1 + opened <= width;
            const int best = pick(area, can, true);
            more = more && best >= 0;
            if (!__any_sync(full, more)) break;
            const int first = get(cand.first, best < 0 ? 0 : best);
            if (more) {
                if (sub == best) place(first);
                else if (sub == nc) place(first + 1);
                nc++;
            }
        }
        // Leaves that do not fit inline become wide children of their own,
        // the largest first (the first of equals).
        bool asNode = false;
        for (bool more = inner;;) {
            const int total = sumAll(asNode ? 1 : slots);
            const bool over = more && total > width;
            const int at = pick((float)cand.count, over && node >= 0 && !asNode && cand.count > group, true);
            more = over && at >= 0;
            if (!__any_sync(full, more)) break;
            if (more && sub == at) asNode = true;
        }
        // Kids: lane k takes the k-th.
        int kind = -1, kidNode = -1, first = 0, count = 0;
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        {
            const bool range = node >= 0 && cand.count > 0 && (asNode || cand.count > width * group);
            const int mine = node < 0 ? 0 : cand.count == 0 || range ? 1 : (cand.count + group - 1) / group;
            int before = 0;
            for (int i = 0; i < 8; i++) {
                const int n = get(mine, i), r = get(range ? 1 : 0, i), cn = get(node, i), cf = get(cand.first, i), cc = get(cand.count, i);
                const float l[3] = {get(cand.low.x, i), get(cand.low.y, i), get(cand.low.z, i)};
                const float h[3] = {get(cand.high.x, i), get(cand.high.y, i), get(cand.high.z, i)};
                if (sub >= before && sub < before + n && sub < width) {
                    if (cc == 0 || r) {
                        kind = cc == 0 ? 0 : 1;
                        kidNode = cc == 0 ? cn : -1;
                        first = cc == 0 ? 0 : cf;
                        count = cc;
                        if (kind == 0)
                            for (int a = 0; a < 3; a++) { lo[a] = l[a]; hi[a] = h[a]; }
                    } else {
                        kind = 2;
                        first = cf + (sub - before) * group;
                        count = imin(group, cc - (sub - before) * group);
                    }
                }
                before += n;
            }
        }
        if (have && !inner) {
            const int chunk = J.count <= width * group ? group : (J.count + width - 1) / width;
            const int g = sub * chunk;
            if (g < J.count && sub < width) {
                first = J.first + g;
                count = imin(chunk, J.count - g);
                kind = chunk == group || count <= group ? 2 : 1;
            }
        }
        // Boxes of primitive ranges, and each triangle group's triangles once.
        int tri[3] = {-1, -1, -1}, nTri = 0;
        if (kind > 0) {
            for (int i = 0; i < count; i++) {
                const int p = order[first + i];
                const float4 a = plo[p], b = phi[p];
                lo[0] = fminf(lo[0], a.x); lo[1] = fminf(lo[1], a.y); lo[2] = fminf(lo[2], a.z);
                hi[0] = fmaxf(hi[0], b.x); hi[1] = fmaxf(hi[1], b.y); hi[2] = fmaxf(hi[2], b.z);
                if (kind == 2) {
                    const int t = primTri ? primTri[p] : p;
                    if (t != tri[0] && t != tri[1] && t != tri[2]) {
                        if (nTri == 0) tri[0] = t;
                        else if (nTri == 1) tri[1] = t;
                        else tri[2] = t;
                        nTri++;
                    }
                }
            }
        }
        float nlo[3], nhi[3];
        for (int a = 0; a < 3; a++) { nlo[a] = minAll(lo[a]); nhi[a] = maxAll(hi[a]); }
        // Slots: greedily the cheapest (kid, slot) pair.
        float ck[3];
        for (int a = 0; a < 3; a++) ck[a] = 0.5f * (lo[a] + hi[a]) - 0.5f * (nlo[a] + nhi[a]);
        int slot = -1;
        {
            unsigned freeSlots = 0xFFu;
            const int nk = __popc((__ballot_sync(full, kind >= 0) >> (slotOfJob * 8)) & 0xFFu);
            const int rounds = __reduce_max_sync(full, nk);
            float cost = FLT_MAX;
            int at = -1;
            auto cheapest = [&]() {
                cost = FLT_MAX;
                at = -1;
                for (int s = 0; s < 8; s++) {
                    if (!((freeSlots >> s) & 1u)) continue;
                    const float c = slotCost(ck, s);
                    if (c < cost) { cost = c; at = s; }
                }
            };
            if (kind >= 0) cheapest();
            for (int round = 0; round < rounds; round++) {
                const bool waiting = kind >= 0 && slot < 0;
                int winner = pick(cost, waiting && at >= 0, false);
                const int next = pick(0.0f, waiting, false);
                int taken = get(at, winner < 0 ? 0 : winner);
                if (winner < 0) {  // non-finite costs: the first waiting kid into the first free slot
                    winner = next;
                    taken = __ffs(freeSlots) - 1;
                }
                if (winner >= 0) {
                    if (sub == winner) slot = taken;
                    freeSlots &= ~(1u << taken);
                    if (waiting && sub != winner && at == taken) cheapest();
                }
            }
        }
        // Storage: the warp's jobs in order.
        const unsigned innerSlots = orAll(kind == 0 || kind == 1 ? 1u << slot : 0u);
        const unsigned triCounts = orAll(kind == 2 ? (unsigned)nTri << (2 * slot) : 0u);  // 2 bits per slot
        const int ni = __popc(innerSlots), nt = __popc(triCounts & 0x5555u) + 2 * __popc(triCounts & 0xAAAAu);
        int si = 0, st = 0, ti = 0, tt = 0;
        for (int g = 0; g < 4; g++) {
            const int a = __shfl_sync(full, ni, g * 8), b = __shfl_sync(full, nt, g * 8);
            if (g < slotOfJob) { si += a; st += b; }
            ti += a;
            tt += b;
        }
        int childBase = 0, triBase = 0, jobBase = 0;
        if (lane == 0) {
            if (ti) { childBase = atomicAdd(&counters[0], ti); jobBase = atomicAdd(nextCount, ti); }
            if (tt) triBase = atomicAdd(&counters[1], tt);
        }
        childBase = __shfl_sync(full, childBase, 0) + si;
        jobBase = __shfl_sync(full, jobBase, 0) + si;
        triBase = __shfl_sync(full, triBase, 0) + st;
        const bool fits = childBase + ni <= wideCapacity && triBase + nt <= triCapacity;
        if (have && !fits && sub == 0) atomicExch(&counters[3], 3);
        // The node record in shared memory: lane 0 the header, then each kid
        // its slot's bytes.
        WideNode& W = shared[warp].node[slotOfJob];
        unsigned char ebits[3];
        for (int a = 0; a < 3; a++) ebits[a] = gridExponent(nhi[a] - nlo[a]);
        __syncwarp();
        if (sub < 5) reinterpret_cast<uint4*>(&W)[sub] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
        if (sub == 0) {
            W.px = nlo[0]; W.py = nlo[1]; W.pz = nlo[2];
            W.ex = ebits[0]; W.ey = ebits[1]; W.ez = ebits[2];
            W.imask = (unsigned char)innerSlots;
            W.childBase = (unsigned)childBase;
            W.triBase = (unsigned)triBase;
        }
        if (kind >= 0 && fits) {
            for (int a = 0; a < 3; a++) quantise(lo[a], hi[a], nlo[a], gridStep(ebits[a]), W.qlo[a][slot], W.qhi[a][slot]);
            const unsigned lower = (1u << slot) - 1u, lower2 = (1u << (2 * slot)) - 1u;
            if (kind == 2) {
                const unsigned below = triCounts & lower2;
                const int offset = __popc(below & 0x5555u) + 2 * __popc(below & 0xAAAAu);
                W.meta[slot] = groupMeta(nTri, offset);
                for (int i = 0; i < nTri; i++) {
                    const int p = i == 0 ? tri[0] : i == 1 ? tri[1] : tri[2];
                    packTriangle(tris[p], p, packed + (size_t)(triBase + offset + i) * 3);
                }
            } else {
                W.meta[slot] = innerMeta(slot);
                const int rank = __popc(innerSlots & lower), q = jobBase + rank;
                if (q >= jobCapacity) atomicExch(&counters[3], 4);
                else nextJobs[q] = Job{kind, kidNode, first, count, childBase + rank};
            }
        }
        __syncwarp();
        if (have && fits && sub < 5) reinterpret_cast<uint4*>(wide + J.wide)[sub] = reinterpret_cast<const uint4*>(&W)[sub];
        __syncwarp();
    }
}

inline int blocksFor(long long n, int block) { return (int)((n + block - 1) / block); }

// What an error of the kernels (counters[3]) means to the caller.
cudaError_t buildError(int code, const char** failure) {
    if (!code) return cudaSuccess;
    *failure = code <= 2 ? "BVH build ran out of node or task capacity"
             : code <= 4 ? "wide BVH collapse ran out of capacity" : "BVH build met an index out of its range";
    return code <= 4 ? cudaErrorMemoryAllocation : cudaErrorUnknown;
}

template <class T>
cudaError_t alloc(T*& p, size_t count) { return rt::deviceAlloc(reinterpret_cast<void**>(&p), sizeof(T) * (count ? count : 1)); }

}  // namespace

void freeBvh(BuiltBvh& b) {
    void* owned[] = {b.binNodes, b.order, b.wideNodes, b.packedTris, b.primLo, b.primHi};
    for (void* p : owned)
        if (p) rt::deviceFree(p);
    b = BuiltBvh{};
}

cudaError_t pieceMap(const SceneTri* tris, int triCount, int maxPieces, cudaStream_t stream, int** primTri, int* total,
                     float* ms) {
    unsigned *counts = nullptr, *pfx = nullptr, *sums = nullptr;
    int* dTotal = nullptr;
    int* map = nullptr;
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    const int nb = blocksFor(triCount, kScanBlock);
    int hostTotal = 0;
    if (primTri) *primTri = nullptr;
    if (ms) *ms = 0.0f;
    // Every allocation before the first kernel, so the timed span is the kernels'.
    cudaError_t err = alloc(counts, triCount);
    if (err == cudaSuccess) err = alloc(pfx, triCount);
    if (err == cudaSuccess) err = alloc(sums, nb);
    if (err == cudaSuccess) err = alloc(dTotal, 2);  // the total, and the scan's count of finished blocks
    if (err == cudaSuccess && primTri) err = alloc(map, (size_t)triCount * maxPieces);
    if (err == cudaSuccess) err = cudaEventCreate(&t0);
    if (err == cudaSuccess) err = cudaEventCreate(&t1);
    if (err == cudaSuccess) err = cudaMemsetAsync(dTotal, 0, 2 * sizeof(int), stream);
    if (err == cudaSuccess) err = cudaEventRecord(t0, stream);
    if (err == cudaSuccess) {
        pieceCountKernel<<<blocksFor(triCount, 256), 256, 0, stream>>>(tris, triCount, maxPieces, counts);
        scanBlocksKernel<<<nb, 256, 0, stream>>>(counts, pfx, triCount, sums, dTotal + 1);
        pieceFillKernel<<<blocksFor(triCount, 256), 256, 0, stream>>>(counts, pfx, sums, triCount, map, dTotal);
        err = cudaGetLastError();
    }
    if (err == cudaSuccess) err = cudaEventRecord(t1, stream);
    if (err == cudaSuccess) err = cudaMemcpyAsync(&hostTotal, dTotal, sizeof(int), cudaMemcpyDeviceToHost, stream);
    if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
    if (err == cudaSuccess && ms) err = cudaEventElapsedTime(ms, t0, t1);
    if (t0) cudaEventDestroy(t0);
    if (t1) cudaEventDestroy(t1);
    if (err != cudaSuccess) settle(stream);
    rt::deviceFree(counts); rt::deviceFree(pfx); rt::deviceFree(sums); rt::deviceFree(dTotal);
    if (err == cudaSuccess && (hostTotal < triCount || hostTotal > triCount * maxPieces)) err = cudaErrorUnknown;
    if (err != cudaSuccess) { rt::deviceFree(map); return err; }
    if (primTri) *primTri = map;
    *total = hostTotal;
    return cudaSuccess;
}

cudaError_t buildBvh(const SceneTri* tris, int triCount, cudaStream_t stream, BuiltBvh& out, BuildResult& result,
                     const char** failure, int leafGroup, int width, int pieces, int leafSize) {
    if (width != 4 && width != 8) { *failure = "BVH width must be 4 or 8"; return cudaErrorInvalidValue; }
    if (leafSize < 1 || leafSize > 8) { *failure = "BVH leaf size must be 1..8"; return cudaErrorInvalidValue; }
    if (pieces < 1 || pieces > 8 || (long long)triCount * pieces > 0x3FFFFFFFll) {
        *failure = "BVH pieces per triangle must be 1..8";
        return cudaErrorInvalidValue;
    }
    *failure = nullptr;
    cudaError_t err = cudaSuccess;
    // Primitives: the triangles, or for a traversal tree their pieces
    // (piecesOf each, consecutive, primTri[p] = triangle of primitive p).
    int n = triCount;
    int* primTri = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr, e2 = nullptr;
    float pieceMs = 0.0f;
    if ((err = cudaEventCreate(&e0)) != cudaSuccess) return err;
    if (pieces > 1) {
        int total = 0;
        err = pieceMap(tris, triCount, pieces, stream, &primTri, &total, &pieceMs);
        if (err != cudaSuccess) { cudaEventDestroy(e0); *failure = "triangle pieces"; return err; }
        if (total == triCount) {  // no triangle is split: a tree over the triangles themselves
            rt::deviceFree(primTri);
            primTri = nullptr;
        }
        n = total;
    }
    const int nodeCapacity = 2 * n + 2;
    const int taskCapacity = n / (kSubtree + 1) + 2;
    const int subtreeCapacity = n / (leafSize + 1) + 2;
    const int wideCapacity = 2 * n + 8;
    // Temporaries.
    float4* cent = nullptr; int* orderB = nullptr; int* posTask = nullptr; int* posTaskB = nullptr;
    Task* tasks = nullptr; Task* tasksB = nullptr; Task* subtrees = nullptr; Subtree* done = nullptr; BinAcc* bins = nullptr; Split* splits = nullptr;
    unsigned* flags = nullptr; unsigned* prefix = nullptr; unsigned* blockSums = nullptr; int* counters = nullptr;
    BinNode* rawNodes = nullptr; int* interior = nullptr; int* rank = nullptr; int* newIndex = nullptr;
    Job* jobs = nullptr; Job* jobsB = nullptr;
    int* levelCounts = nullptr; int* levelStartDev = nullptr; int* jobCounts = nullptr;
    int hostCounters[kCounters] = {}, hostLevels[2 * (kBinaryMaxDepth + 2 + kLevelBatch)], hostStarts[kBinaryMaxDepth + 4 + kLevelBatch];
    int hostJobs[kStackCapacity + 2 + kLevelBatch];
    std::vector<int> levelStart;
    // A tree over pieces is only traced: its nodes stay as they are numbered.
    const bool renumber = pieces == 1;
    int nScanBlocks = blocksFor(n, kScanBlock);

#define RT_TRY(x) do { err = (x); if (err != cudaSuccess) goto done; } while (0)
    RT_TRY(alloc(out.primLo, n)); RT_TRY(alloc(out.primHi, n)); RT_TRY(alloc(cent, n));
    RT_TRY(alloc(out.order, n)); RT_TRY(alloc(orderB, n)); RT_TRY(alloc(posTask, n)); RT_TRY(alloc(posTaskB, n));
    RT_TRY(alloc(tasks, taskCapacity)); RT_TRY(alloc(tasksB, taskCapacity)); RT_TRY(alloc(subtrees, subtreeCapacity));
    RT_TRY(alloc(bins, (size_t)taskCapacity * 3 * kBins)); RT_TRY(alloc(splits, taskCapacity));
    RT_TRY(alloc(flags, n)); RT_TRY(alloc(prefix, n)); RT_TRY(alloc(blockSums, nScanBlocks));
    RT_TRY(alloc(counters, kCounters)); RT_TRY(alloc(rawNodes, nodeCapacity));
    {
        const int levelSlots = kBinaryMaxDepth + 2 + kLevelBatch, jobSlots = kStackCapacity + 2 + kLevelBatch;
        RT_TRY(alloc(levelCounts, 2 * levelSlots)); RT_TRY(alloc(levelStartDev, levelSlots + 2));
        RT_TRY(alloc(jobCounts, jobSlots));
    }
    // Renumbering and collapse buffers at their upper bounds (node count <=
    // nodeCapacity, wide nodes and jobs <= 2n + 8), so no allocation falls
    // inside the timed spans.
    if (renumber) {
        RT_TRY(alloc(interior, nodeCapacity)); RT_TRY(alloc(rank, nodeCapacity)); RT_TRY(alloc(newIndex, nodeCapacity));
        RT_TRY(alloc(out.binNodes, nodeCapacity)); RT_TRY(alloc(done, subtreeCapacity));
    }
    RT_TRY(alloc(out.wideNodes, (size_t)wideCapacity * 5));
    RT_TRY(alloc(out.packedTris, (size_t)n * 3));
    RT_TRY(alloc(jobs, wideCapacity)); RT_TRY(alloc(jobsB, wideCapacity));
    RT_TRY(cudaEventCreate(&e1)); RT_TRY(cudaEventCreate(&e2));
    RT_TRY(cudaEventRecord(e0, stream));  // build time: the kernels, not the allocations before them
    {
        Task root{};
        root.node = 0; root.first = 0; root.count = n; root.depth = 0;
        for (int a = 0; a < 3; a++) { root.lo[a] = root.clo[a] = FLT_MAX; root.hi[a] = root.chi[a] = -FLT_MAX; }
        RT_TRY(cudaMemcpyAsync(tasks, &root, sizeof(Task), cudaMemcpyHostToDevice, stream));
        // A root of few primitives is a subtree task itself.
        const bool smallRoot = n <= kSubtree;
        int init[kCounters] = {1, 0, 0, 0, smallRoot ? 1 : 0, 0, 0, 0};
        RT_TRY(cudaMemcpyAsync(counters, init, sizeof(init), cudaMemcpyHostToDevice, stream));
        if (!primTri)
            primBoxesKernel<<<blocksFor(n, 256), 256, 0, stream>>>(tris, n, out.primLo, out.primHi, cent, tasks);
        else
            splitBoxesKernel<<<blocksFor(n, 256), 256, 0, stream>>>(tris, primTri, n, pieces, out.primLo, out.primHi,
                                                                    cent, tasks);
        iotaKernel<<<blocksFor(n, 256), 256, 0, stream>>>(out.order, n, 0, posTask, 0);
        RT_TRY(cudaGetLastError());
        // Binned SAH, level by level without the host in the loop: each
        // level's counts (open tasks, tasks above kSmallTask) are written
        // by the previous level's split kernel into levelCounts, and the
        // per-task kernels loop over them, so the host queues a batch of
        // levels and reads the counts once per batch. A level with no task
        // only copies the order through. Depth is at most kBinaryMaxDepth,
        // so at most kBinaryMaxDepth + 1 levels hold tasks.
        const int levelSlots = kBinaryMaxDepth + 2 + kLevelBatch;
        RT_TRY(cudaMemsetAsync(levelCounts, 0, sizeof(int) * 2 * levelSlots, stream));
        RT_TRY(cudaMemsetAsync(levelStartDev, 0, sizeof(int) * (levelSlots + 2), stream));
        {
            int rootCounts[2] = {smallRoot ? 0 : 1, n > kSmallTask ? 1 : 0};
            int starts[2] = {0, 1};  // depth 0 holds node 0
            RT_TRY(cudaMemcpyAsync(levelCounts, rootCounts, sizeof(rootCounts), cudaMemcpyHostToDevice, stream));
            RT_TRY(cudaMemcpyAsync(levelStartDev, starts, sizeof(starts), cudaMemcpyHostToDevice, stream));
        }
        if (smallRoot) RT_TRY(cudaMemcpyAsync(subtrees, tasks, sizeof(Task), cudaMemcpyDeviceToDevice, stream));
        // Enough position blocks for the SMs where there are few positions.
        const int perThread = std::max(1, std::min(kBinPer, n / (148 * kBinBlock)));
        const int largeBlocks = n > kSmallTask ? blocksFor(n, kBinBlock * perThread) : 0;
        const int smallBlocks = std::max(1, std::min(n / kSearchTask, 1184));
        const int splitBlocks = std::max(1, std::min(blocksFor(taskCapacity, 4), 1184));
        const int clearBlocks = std::max(1, std::min(blocksFor((long long)taskCapacity * 3 * kBins, 256), 1184));
        clearBinsKernel<<<clearBlocks, 256, 0, stream>>>(bins, levelCounts, tasks);
        int level = 0, used = 0;  // levels queued, and those that held tasks
        if (!smallRoot)
            for (int batch = kLevelBatch;; batch = kNextLevels) {
                for (int b = 0; b < batch && level < levelSlots - 1; b++, level++) {
                    const int* tc = levelCounts + 2 * level;
                    int* nc = levelCounts + 2 * (level + 1);
                    binKernel<<<largeBlocks + smallBlocks, kBinBlock, 0, stream>>>(out.order, posTask, cent, out.primLo, out.primHi,
                                                                                   tasks, n, bins, tc, largeBlocks, perThread);
                    splitKernel<<<splitBlocks, 128, 0, stream>>>(out.order, cent, out.primLo, out.primHi, tasks, tc, bins, splits, rawNodes, counters, nc, tasksB, subtrees,
                                                                 nodeCapacity, taskCapacity, subtreeCapacity, leafSize);
                    partitionKernel<<<nScanBlocks, 256, 0, stream>>>(out.order, posTask, cent, tasks, splits, n, flags, prefix,
                                                                     blockSums, counters, levelStartDev + level + 2, tc, nc,
                                                                     tasksB, bins);
                    scatterKernel<<<blocksFor(n, 256), 256, 0, stream>>>(out.order, posTask, tasks, splits, flags, prefix,
                                                                         blockSums, n, orderB, posTaskB, tc, counters + 3);
                    std::swap(out.order, orderB); std::swap(posTask, posTaskB); std::swap(tasks, tasksB);
                }
                RT_TRY(cudaGetLastError());
                RT_TRY(cudaMemcpyAsync(hostCounters, counters, sizeof(hostCounters), cudaMemcpyDeviceToHost, stream));
                RT_TRY(cudaMemcpyAsync(hostLevels, levelCounts, sizeof(int) * 2 * levelSlots, cudaMemcpyDeviceToHost, stream));
                RT_TRY(cudaStreamSynchronize(stream));
                if ((err = buildError(hostCounters[3], failure)) != cudaSuccess) goto done;
                if (hostLevels[2 * level] == 0) break;  // the next level has no task
                if (level >= levelSlots - 1) { *failure = "BVH build exceeded the depth limit"; err = cudaErrorUnknown; goto done; }
            }
        while (used < level && hostLevels[2 * used] > 0) used++;
        if ((level - used) & 1) std::swap(out.order, orderB);  // levels past the last moved nothing
        // Subtrees of small tasks. Few are known before the levels end; the
        // kernel loops over the device count.
        const int topNodes = smallRoot ? 1 : hostCounters[0];
        subtreeKernel<<<std::max(1, std::min(blocksFor(subtreeCapacity, kSubtreeWarps), 148 * 8)), 32 * kSubtreeWarps, 0, stream>>>(
            out.order, cent, out.primLo, out.primHi, subtrees, counters, rawNodes, nodeCapacity, leafSize, interior, done);
        RT_TRY(cudaGetLastError());
        RT_TRY(cudaMemcpyAsync(hostCounters, counters, sizeof(hostCounters), cudaMemcpyDeviceToHost, stream));
        RT_TRY(cudaMemcpyAsync(hostStarts, levelStartDev, sizeof(int) * (level + 2), cudaMemcpyDeviceToHost, stream));
        RT_TRY(cudaStreamSynchronize(stream));
        if ((err = buildError(hostCounters[3], failure)) != cudaSuccess) goto done;
        levelStart.assign(hostStarts, hostStarts + level + 2);
        int nodeCount = hostCounters[0];
        result.binaryNodes = nodeCount;
        result.binaryDepth = hostCounters[2];
        if (renumber) {
            // levelStart[d] .. levelStart[d+1] are the nodes of depth d made level by level.
            while (levelStart.size() > 2 && levelStart.back() == levelStart[levelStart.size() - 2]) levelStart.pop_back();
            int depths = (int)levelStart.size() - 1;
            for (int d = depths - 1; d >= 0; d--) {
                int b = levelStart[d], e = levelStart[d + 1];
                subtreeInteriorKernel<<<blocksFor(e - b, 256), 256, 0, stream>>>(rawNodes, b, e, topNodes, interior);
            }
            RT_TRY(cudaMemsetAsync(rank, 0xFF, sizeof(int) * topNodes, stream));
            RT_TRY(cudaMemsetAsync(newIndex, 0xFF, sizeof(int) * topNodes, stream));
            RT_TRY(cudaMemsetAsync(rank, 0, sizeof(int), stream));
            RT_TRY(cudaMemsetAsync(newIndex, 0, sizeof(int), stream));
            for (int d = 0; d < depths; d++) {
                int b = levelStart[d], e = levelStart[d + 1];
                preorderKernel<<<blocksFor(e - b, 256), 256, 0, stream>>>(rawNodes, b, e, topNodes, nodeCount, interior, rank,
                                                                          newIndex, counters + 3);
            }
            renumberKernel<<<blocksFor(topNodes, 256), 256, 0, stream>>>(rawNodes, topNodes, nodeCount, newIndex, rank,
                                                                         out.binNodes, counters + 3);
            placeSubtreesKernel<<<std::max(1, std::min(blocksFor(subtreeCapacity, 8), 1184)), 256, 0, stream>>>(
                rawNodes, done, counters, rank, nodeCount, out.binNodes, counters + 3);
        } else {
            std::swap(out.binNodes, rawNodes);
        }
        RT_TRY(cudaGetLastError());
        RT_TRY(cudaEventRecord(e1, stream));

        // Collapse, one wide level per launch; job counts per level on the
        // device (jobCounts), read once per batch of levels.
        const int jobCapacity = wideCapacity;
        Job rootJob{0, 0, 0, 0, 0};
        RT_TRY(cudaMemcpyAsync(jobs, &rootJob, sizeof(Job), cudaMemcpyHostToDevice, stream));
        int cinit[3] = {1, 0, 0};  // the error stays: the renumbering may have set it
        RT_TRY(cudaMemcpyAsync(counters, cinit, sizeof(cinit), cudaMemcpyHostToDevice, stream));
        const int jobSlots = kStackCapacity + 2 + kLevelBatch;
        RT_TRY(cudaMemsetAsync(jobCounts, 0, sizeof(int) * jobSlots, stream));
        RT_TRY(cudaMemcpyAsync(jobCounts, cinit, sizeof(int), cudaMemcpyHostToDevice, stream));  // one root job
        const int collapseBlocks = std::max(1, std::min(blocksFor(jobCapacity, 8), 2368));
        int wideLevel = 0, wideDepth = 0;
        for (;;) {
            for (int b = 0; b < kLevelBatch && wideLevel < jobSlots - 1; b++, wideLevel++) {
                collapseKernel<<<collapseBlocks, 64, 0, stream>>>(out.binNodes, out.order, out.primLo, out.primHi, tris,
                                                                  jobs, jobCounts + wideLevel, jobsB,
                                                                  jobCounts + wideLevel + 1,
                                                                  reinterpret_cast<WideNode*>(out.wideNodes),
                                                                  out.packedTris, counters, wideCapacity, jobCapacity, n,
                                                                  leafGroup, width, primTri);
                std::swap(jobs, jobsB);
            }
            RT_TRY(cudaGetLastError());
            RT_TRY(cudaMemcpyAsync(hostCounters, counters, 8 * sizeof(int), cudaMemcpyDeviceToHost, stream));
            RT_TRY(cudaMemcpyAsync(hostJobs, jobCounts, sizeof(int) * jobSlots, cudaMemcpyDeviceToHost, stream));
            RT_TRY(cudaStreamSynchronize(stream));
            if ((err = buildError(hostCounters[3], failure)) != cudaSuccess) goto done;
            if (hostJobs[wideLevel] == 0) break;
            if (wideLevel >= jobSlots - 1) break;
        }
        while (wideDepth < jobSlots && hostJobs[wideDepth] > 0) wideDepth++;
        if (wideDepth > kStackCapacity) { *failure = "wide BVH deeper than the traversal stack"; err = cudaErrorUnknown; goto done; }
        RT_TRY(cudaEventRecord(e2, stream));
        RT_TRY(cudaEventSynchronize(e2));
        // Every primitive is packed once, except pieces of a triangle that
        // share a leaf group (packed once for the group).
        if (!primTri ? hostCounters[1] != n : (hostCounters[1] < triCount || hostCounters[1] > n)) {
            *failure = "wide BVH collapse lost triangles";
            err = cudaErrorUnknown;
            goto done;
        }
        result.wideNodes = hostCounters[0];
        result.packedTriangles = hostCounters[1];
        result.wideDepth = wideDepth;
        RT_TRY(cudaEventElapsedTime(&result.buildMs, e0, e1));
        result.buildMs += pieceMs;
        RT_TRY(cudaEventElapsedTime(&result.collapseMs, e1, e2));
    }
done:
#undef RT_TRY
    if (err != cudaSuccess) settle(stream);
    rt::deviceFree(cent); rt::deviceFree(orderB); rt::deviceFree(posTask); rt::deviceFree(posTaskB); rt::deviceFree(tasks); rt::deviceFree(tasksB); rt::deviceFree(subtrees);
    rt::deviceFree(done);
    rt::deviceFree(bins); rt::deviceFree(splits); rt::deviceFree(flags); rt::deviceFree(prefix); rt::deviceFree(blockSums); rt::deviceFree(counters);
    rt::deviceFree(rawNodes); rt::deviceFree(interior); rt::deviceFree(rank); rt::deviceFree(newIndex); rt::deviceFree(jobs); rt::deviceFree(jobsB);
    rt::deviceFree(primTri);
    rt::deviceFree(levelCounts); rt::deviceFree(levelStartDev); rt::deviceFree(jobCounts);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (e2) cudaEventDestroy(e2);
    if (err != cudaSuccess) freeBvh(out);
    return err;
}

}  // namespace rt
