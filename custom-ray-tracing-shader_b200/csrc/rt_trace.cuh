// Persistent ray-query kernels with dynamic ray fetch (device only).
//
// Each warp keeps 32 rays in flight and advances them in rounds of triangle
// tests and node visits (see persistentTrace). When fewer than `refill` lanes
// are busy, the warp fetches new rays for its idle lanes with one atomic per
// warp, so lanes do not idle while the slowest ray of a fixed batch finishes
// (persistent threads with dynamic fetch, Aila and Laine, HPG 2009). The
// traversal stack of each ray keeps its first kSharedStack entries in shared
// memory (one column per thread) and the rest in local memory.
//
// Results are those of rt::traverse (rt_bvh.cuh): the same triangle test, the
// same acceptance rule and tie-break, the same conservative box tests, so the
// closest hit and the any-hit verdict are identical; only the visiting order
// of work differs, which the results do not depend on.
#pragma once
#include "rt_bvh.cuh"

namespace rt {

// Stack entries per ray held in shared memory (deeper entries live in
// local memory, which L1 caches). Fewer entries leave more of the SM's
// L1/shared storage to L1, which serves the node and triangle fetches: on
// the 1M-triangle workload 16 entries gave 3,007 Mrays/s, 12 and 10 3,026,
// 8 3,052-3,059, 6 3,056, 4 2,996-3,003.
constexpr int kSharedStack = 8;
constexpr int kTraceBlock = 128;

// Per-lane traversal state in registers. The ray's origin and direction for
// triangle tests and its best hit live in WarpTriangles, where any lane of
// the warp may test for it; tmax mirrors the best hit's distance.
struct LaneRay {
    RaySetup r;
    float tmax;
    uint2 group, triGroup;
    int top;
};

// Node step, taken when the lane has no pending triangles: pops an entry if
// the current group has no interior children left, then visits one child
// node (its eight child boxes). Returns true when the traversal is complete.
__device__ __forceinline__ bool nodeStep(LaneRay& L, const uint4* nodes, uint2* sstack, int stride, uint2* lstack,
                                         int& overflow, int stackLimit) {
    if (L.group.y <= 0x00FFFFFFu) {
        if (L.top == 0) return true;
        L.top--;  // only groups with interior children are pushed
        L.group = L.top < kSharedStack ? sstack[L.top * stride] : lstack[L.top - kSharedStack];
    }
    int bit = 31 - __clz(L.group.y & 0xFF000000u);
    L.group.y &= ~(1u << bit);
    unsigned slot = ((unsigned)bit - 24u) ^ L.r.octInv;
    unsigned child = L.group.x + __popc(L.group.y & 0xFFu & ((1u << slot) - 1u));
    if (L.group.y > 0x00FFFFFFu) {
        if (L.top >= stackLimit) { overflow = 1; return true; }
        if (L.top < kSharedStack) sstack[L.top * stride] = L.group;
        else lstack[L.top - kSharedStack] = L.group;
        L.top++;
    }
    unsigned childBase, triBase, imask;
    unsigned mask = intersectWideNode(nodes + (size_t)child * 5, L.r, L.tmax, childBase, triBase, imask);
    L.group = make_uint2(childBase, (mask & 0xFF000000u) | imask);
    L.triGroup = make_uint2(triBase, mask & 0x00FFFFFFu);
    return false;
}

// Per-warp shared state of the cooperative triangle phase: the rays in flight
// (written when a lane fetches one) and each round's pending triangles.
// 1,888 bytes per warp: with the stacks a block of 4 warps takes 15,744
// bytes, so that 8 blocks stay within 132 KB of the SM's storage and leave
// the rest to L1.
struct WarpTriangles {
    float4 origin[32];              // each lane's ray origin
    float4 dir[32];                 // each lane's ray direction
    unsigned long long best[32];    // (distance bits << 32 | index) of each lane's best hit
    float2 uv[32];                  // barycentrics of that hit
    uint2 group[32];                // each lane's pending triangle group
    unsigned short start[32];       // exclusive prefix sum of pending triangle counts
    unsigned char owner[32];        // lanes with pending triangles, in lane order
};
constexpr size_t traceSharedBytes(int block) {
    return sizeof(uint2) * kSharedStack * block + sizeof(WarpTriangles) * (block / 32);
}

// Key ordering hits like the reference's acceptance rule (renderer.cu:153):
// smaller distance first, then smaller triangle index. Distances are
// positive, so their bit patterns order like the values. Before any hit the
// best is (limit, index -1) and the rule accepts only distances below the
// limit (i < -1 never holds), so that state is keyed with low word 0: a
// candidate at exactly the limit has a key >= it and is rejected.
__device__ __forceinline__ unsigned long long hitKey(float distance, int index) {
    return ((unsigned long long)__float_as_uint(distance) << 32) | (unsigned)(index < 0 ? 0 : index);
}

// root: index of the ray's root node (0 for a single scene; the scene's
// first node when several scenes share one node array).
__device__ __forceinline__ void laneStart(LaneRay& L, float3 o, float3 d, float limit, unsigned root, WarpTriangles& W,
                                          unsigned lane) {
    L.r = setupRay(o, d);
    L.tmax = limit;
    L.group = make_uint2(root, 0x80000000u);
    L.triGroup = make_uint2(0u, 0u);
    L.top = 0;
    W.origin[lane] = make_float4(o.x, o.y, o.z, 0.0f);
    W.dir[lane] = make_float4(d.x, d.y, d.z, 0.0f);
    W.best[lane] = hitKey(limit, -1);
    W.uv[lane] = make_float2(0.0f, 0.0f);
}

// Cooperative triangle phase: the warp's pending triangles (all lanes' groups)
// are dealt out one per lane per iteration; each candidate hit is merged into
// its ray's best with a shared-memory 64-bit atomicMin on hitKey. The result
// is the minimum over the same candidate set as testing them one by one, so
// it equals the sequential outcome. Returns true for a lane whose best hit
// changed (any-hit: the query is answered).
//
// Dealing: counts are below 32, so their prefix sums come from one ballot per
// bit of the counts; of a round's work items, item w belongs to the last
// owner whose first item is at or before w, found from the mask of first
// items by a population count.
__device__ __forceinline__ bool warpTrianglePhase(LaneRay& L, bool busy, const float4* tris, WarpTriangles& W,
                                                  unsigned lane, unsigned below) {
    const unsigned full = 0xFFFFFFFFu;
    const unsigned count = busy ? __popc(L.triGroup.y) : 0u;
    const unsigned pending = __ballot_sync(full, count != 0u);
    if (pending == 0u) return false;
    const unsigned b0 = __ballot_sync(full, count & 1u), b1 = __ballot_sync(full, count & 2u),
                   b2 = __ballot_sync(full, count & 4u);
    unsigned excl = __popc(b0 & below) + 2u * __popc(b1 & below) + 4u * __popc(b2 & below);
    unsigned total = __popc(b0) + 2u * __popc(b1) + 4u * __popc(b2);
    if (__any_sync(full, count > 7u)) {
        const unsigned b3 = __ballot_sync(full, count & 8u), b4 = __ballot_sync(full, count & 16u);
        excl += 8u * __popc(b3 & below) + 16u * __popc(b4 & below);
        total += 8u * __popc(b3) + 16u * __popc(b4);
    }
    if (count) {
        W.group[lane] = L.triGroup;
        W.start[lane] = (unsigned short)excl;
        W.owner[__popc(pending & below)] = (unsigned char)lane;
    }
    __syncwarp();
    unsigned before = 0u;  // owners whose first item lies before this iteration's items
    for (unsigned base = 0; base < total; base += 32u) {
        const unsigned first = excl - base;
        const unsigned heads = __reduce_or_sync(full, count && first < 32u ? 1u << first : 0u);
        unsigned long long key = ~0ull;
        unsigned owner = 0;
        float u = 0.0f, v = 0.0f;
        if (base + lane < total) {
            owner = W.owner[before + __popc(heads & (below | (1u << lane))) - 1u];
            const uint2 g = W.group[owner];
            unsigned m = g.y;
            for (unsigned skip = base + lane - W.start[owner]; skip; skip--) m &= m - 1u;
            const float4* t = tris + (size_t)(g.x + (unsigned)(__ffs(m) - 1)) * 3;
            float4 a = __ldg(t), b = __ldg(t + 1), c = __ldg(t + 2);
            float4 o4 = W.origin[owner], d4 = W.dir[owner];
            float dist = intersectTriangle(v3(o4.x, o4.y, o4.z), v3(d4.x, d4.y, d4.z), a, b, c, u, v);
            if (dist > 0) {
                unsigned long long k = hitKey(dist, __float_as_int(c.z));
                if (k < W.best[owner]) { atomicMin(&W.best[owner], k); key = k; }
            }
        }
        before += __popc(heads);
        __syncwarp();
        if (key != ~0ull && W.best[owner] == key) W.uv[owner] = make_float2(u, v);
        __syncwarp();
    }
    bool changed = false;
    if (count) {
        // A first hit lies below the limit; a later one at an equal distance
        // (a smaller index) changes nothing here.
        const float distance = __uint_as_float((unsigned)(W.best[lane] >> 32));
        changed = distance < L.tmax;
        L.tmax = distance;
        L.triGroup.y = 0u;
    }
    return changed;
}

// Persistent query loop over `count` rays of an IO object providing
//   __device__ void load(int k, float3& o, float3& d, float& limit, unsigned& root);
//   __device__ void store(int k, const Hit& h);
// `fetch` must be zero at launch. Adds the number of finished queries to
// *done and sets *errorFlag on stack overflow (more than stackLimit <=
// kStackCapacity entries). Dynamic shared memory: traceSharedBytes(blockDim.x).
//
// Each round has a triangle phase, in which the warp tests all pending
// triangles of its lanes cooperatively (warpTrianglePhase), and a node phase,
// in which every busy lane takes one node step. The node step (eight box
// tests) is the costly one, so running it in lockstep for all busy lanes
// keeps the warp's lanes doing useful work.
template <bool ANY, class IO>
__device__ __forceinline__ void persistentTrace(IO& io, int count, const uint4* nodes, const float4* tris, int* fetch,
                                                unsigned long long* done, int* errorFlag, int stackLimit,
                                                int refill) {
    extern __shared__ uint2 smemStack[];
    uint2* sstack = smemStack + threadIdx.x;
    const int stride = blockDim.x;
    WarpTriangles* warps = reinterpret_cast<WarpTriangles*>(smemStack + kSharedStack * blockDim.x);
    WarpTriangles& W = warps[threadIdx.x >> 5];
    uint2 lstack[kStackCapacity - kSharedStack];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    LaneRay L;
    int k = -1, overflow = 0;
    bool drained = false, hit = false;
    // The lane's finished query: its best hit, or none within the limit.
    auto finish = [&]() {
        const unsigned long long b = W.best[lane];
        const float2 uv = W.uv[lane];
        io.store(k, Hit{hit ? (int)(unsigned)(b & 0xFFFFFFFFull) : -1, __uint_as_float((unsigned)(b >> 32)), uv.x, uv.y});
    };
    unsigned finished = 0;
    for (;;) {
        if (!drained) {
            unsigned idle = __ballot_sync(0xFFFFFFFFu, k < 0);
            if (idle) {
                int leader = __ffs(idle) - 1, base = 0;
                if ((int)lane == leader) base = atomicAdd(fetch, __popc(idle));
                base = __shfl_sync(0xFFFFFFFFu, base, leader);
                if (base + __popc(idle) >= count) drained = true;
                if (k < 0) {
                    int mine = base + __popc(idle & below);
                    if (mine < count) {
                        float3 o, d;
                        float limit;
                        unsigned root = 0;
                        io.load(mine, o, d, limit, root);
                        if (limit > 0.0f) {
                            laneStart(L, o, d, limit, root, W, lane);
                            k = mine;
                            hit = false;
                        } else {
                            // No distance can be accepted (limit <= 0 or NaN):
                            // the reference's answer is "no hit" at once.
                            io.store(mine, Hit{-1, limit, 0.0f, 0.0f});
                            finished++;
                        }
                    }
                }
            }
        }
        if (!__any_sync(0xFFFFFFFFu, k >= 0)) break;
        const int threshold = drained ? 1 : refill;
        for (;;) {
            if (warpTrianglePhase(L, k >= 0, tris, W, lane, below)) hit = true;
            if (k >= 0 && ((ANY && hit) || nodeStep(L, nodes, sstack, stride, lstack, overflow, stackLimit))) {
                finish();
                k = -1;
                finished++;
            }
            if (__popc(__ballot_sync(0xFFFFFFFFu, k >= 0)) < threshold) break;
        }
    }
    unsigned s = __reduce_add_sync(0xFFFFFFFFu, finished);
    if (lane == 0 && s && done) atomicAdd(done, (unsigned long long)s);
    if (overflow) atomicExch(errorFlag, 1);
}

}  // namespace rt
