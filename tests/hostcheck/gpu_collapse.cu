// The library's build of one scene and the host form of its collapse over the
// same binary tree, for a test that holds the two against each other (needs a
// GPU). Includes the sources of the build, so that the nodes are the library's.
#include "../../custom-ray-tracing-shader_b200/csrc/rt_memory.cu"
#include "../../custom-ray-tracing-shader_b200/csrc/rt_build.cu"

using namespace rt;

extern "C" {

// result: [0] wide nodes, [1] packed triangles, [2] wide nodes and [3] packed
// triangles of the host form. Arrays of 2 * pieces * n + 8 nodes (80 bytes) and
// pieces * n triangles (48 bytes). Returns 0, or a CUDA error.
int gc_collapse(const SceneTri* hostTris, int n, int width, int pieces, int leafSize, uint4* wide, float4* packed,
                uint4* hostWide, float4* hostPacked, int* result) {
    SceneTri* tris = nullptr;
    BuiltBvh bvh;
    BuildResult built;
    const char* why = nullptr;
    int* primTri = nullptr;
    int prims = n;
    cudaError_t e = cudaMalloc(&tris, sizeof(SceneTri) * n);
    if (e == cudaSuccess) e = cudaMemcpy(tris, hostTris, sizeof(SceneTri) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = buildBvh(tris, n, 0, bvh, built, &why, 3, width, pieces, leafSize);
    if (e == cudaSuccess && pieces > 1) e = pieceMap(tris, n, pieces, 0, &primTri, &prims);
    std::vector<BinNode> bn((size_t)built.binaryNodes);
    std::vector<int> order((size_t)prims), map((size_t)prims);
    std::vector<float4> lo((size_t)prims), hi((size_t)prims);
    auto get = [&](void* to, const void* from, size_t bytes) {
        if (e == cudaSuccess && bytes) e = cudaMemcpy(to, from, bytes, cudaMemcpyDeviceToHost);
    };
    get(bn.data(), bvh.binNodes, sizeof(BinNode) * bn.size());
    get(order.data(), bvh.order, sizeof(int) * prims);
    get(lo.data(), bvh.primLo, sizeof(float4) * prims);
    get(hi.data(), bvh.primHi, sizeof(float4) * prims);
    if (primTri) get(map.data(), primTri, sizeof(int) * prims);
    get(wide, bvh.wideNodes, sizeof(WideNode) * (size_t)built.wideNodes);
    get(packed, bvh.packedTris, sizeof(float4) * 3 * (size_t)built.packedTriangles);
    const bool split = prims > n;
    freeBvh(bvh);
    deviceFree(primTri);
    cudaFree(tris);
    trimDeviceMemory();
    if (e != cudaSuccess) return (int)e;
    std::vector<Job> jobs{Job{0, 0, 0, 0, 0}}, next((size_t)2 * prims + 8);
    int counters[4] = {1, 0, 0, 0};
    while (!jobs.empty() && !counters[3]) {
        counters[2] = 0;
        for (const Job& j : jobs)
            collapseJob(j, bn.data(), order.data(), lo.data(), hi.data(), hostTris, next.data(),
                        reinterpret_cast<WideNode*>(hostWide), hostPacked, counters, 2 * prims + 8, 2 * prims + 8, prims, 3,
                        width, split ? map.data() : nullptr);
        jobs.assign(next.begin(), next.begin() + counters[2]);
    }
    result[0] = built.wideNodes;
    result[1] = built.packedTriangles;
    result[2] = counters[0];
    result[3] = counters[1];
    return counters[3] ? 9999 : 0;
}

}  // extern "C"
