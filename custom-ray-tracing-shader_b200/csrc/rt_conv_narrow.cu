// 3x3 convolutions of the denoiser on narrow or small images (the deep levels
// of training crops and of 1080p frames) and of layers whose weights don't fit
// shared memory, on the fifth-generation tensor cores.
//
// The pipelined kernel's tile is 128 pixels of one image row, so an image 8,
// 16, 32 or 64 pixels wide leaves most of every MMA to padding and makes a
// chain of tiles out of little work. Here a tile is 128 consecutive positions
// of the zero-padded image taken as one line: a strip of R output rows is
// staged with its halo as (R + 2) rows of w + 2 pixels, one TMA box per slab
// of 16, 32 or 64 channels with the 32-, 64- or 128-byte swizzle (the K-major
// operand layout, 8-pixel groups a constant stride apart across the row
// ends), and tap (dy, dx) is the same line shifted by dy (w + 2) + dx pixels.
// The two padding positions of each row (2 / (w + 2) of a tile) compute
// values that are not stored. Wider images are cut into equal column segments
// of up to 64 pixels, each staged with its own halo.
//
// A block owns a slice of the output channels (its weights stay in shared
// memory, three TMA boxes per slab, one per kernel row, each with its own
// barrier) and every grid-stride strip; two stages of input where they fit.
// Roles: warp 0 loads, warp 1 issues the MMAs of a strip's tiles into one of
// up to two sets of accumulators, warps 2-9 drain them (alternate tiles).
// Hand-offs are mbarriers; waits are bounded as in rt_conv_pipe.cu.
//
// Streamed layers (224 -> 96 and its data gradient: 387 KB of weights) fill a
// stage with one slab of a strip and that slab of the weights, up to four in
// flight, and keep the accumulators of a strip over its slabs: the weights are
// read once per strip, and the block computes all or half of the channels.
//
// Measured at 32 images (ncu, cold): 128 -> 128 channels at 8 x 8 36 -> 10 us,
// 224 -> 96 at 16 x 16 122 -> 27 (resident slices of 16 channels), 64 -> 64 at
// 32 x 32 30 -> 13, 48 -> 48 at 64 x 64 32 -> 22; all 28 such convolutions of a
// training step 1.21 -> 0.49 ms. Streamed, 224 -> 96 at 240 x 136: 71 us in the
// single-role kernel on the same concatenated input (73 reading its halves in
// place), 22 here.
// What is left is launch, the weights' first load and one to five strips per block.
//
// The products are accumulated in the order of the kernel that runs the
// layer on wide images, so results are bit-identical to it: taps outer and
// channels inner, or for the streamed layers, whose channels rt_conv_tc.cu
// takes in chunks of 16, chunks outer and taps inner.
#include <algorithm>
#include <cstdint>

#include "rt_tc_ptx.cuh"

namespace rt {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kTile = 128;
constexpr int kEpilogueWarps = 8;
constexpr int kThreads = 64 + 32 * kEpilogueWarps;
constexpr int kMaxTiles = 16;            // tiles per strip
constexpr int kMaxStages = 4;
constexpr uint32_t kHeader = 2048;
constexpr uint32_t kSmemMax = 227u * 1024u;

struct NarrowArgs {
    int n, h, w, pitch, cin;
    int segments, segWidth;           // column segments of the image (pitch = segWidth + 2)
    int coutTotal, cout, slices;      // output channels of the layer, of a block, and slices
    int rows, strips, units;
    int slabs;
    uint32_t slabBytes, stageBytes, weightBytes, weightSpace;  // weightSpace: weightBytes on a 1024-byte boundary
    int stages, sets;                 // input stages, accumulator sets
    uint32_t setCols, tmemCols;
    const float* bias;
    bf16* outB;
    float* outF;
    int relu, accumulate, reverseTaps;
    int* errorFlag;
    unsigned long long waitLimitNs;
};

struct Header {
    static constexpr uint32_t full = 0;         // kMaxStages
    static constexpr uint32_t empty = 8 * kMaxStages;
    static constexpr uint32_t weights = 16 * kMaxStages;  // 3 kernel rows
    static constexpr uint32_t accFull = weights + 32;     // 2 sets x kMaxTiles
    static constexpr uint32_t accEmpty = accFull + 16 * kMaxTiles;  // 2 sets x kMaxTiles
    static constexpr uint32_t drain = accEmpty + 16 * kMaxTiles;
    static constexpr uint32_t tmemSlot = drain + 8;
    static constexpr uint32_t abort = tmemSlot + 4;
    static constexpr uint32_t bias = 1024;      // up to 128 floats
};
static_assert(Header::abort + 4 <= Header::bias && Header::bias + 512 <= kHeader, "header size");

// K-major swizzled descriptor of rows of S channels.
template <int S>
__device__ __forceinline__ uint64_t rowsDescriptor(uint32_t addr) {
    return ummaSmemDesc(addr, 16u, 16u * S) | slabLayout(S);
}

// The 9 x K MMAs of one tile; a: descriptors of the tile's start in the three
// kernel rows' lines (first slab), aSlab and bSlab descriptor units between
// slabs, bTap between taps.
template <int S>
__device__ __forceinline__ void issueStep(uint32_t acc, const uint64_t (&a)[3], uint64_t b, uint32_t aSlab, int bSlab,
                                          int bTap, uint32_t idesc, int t, int k, bool fresh) {
    mma(acc, a[t / 3] + (uint64_t)((t % 3) * (S / 8) + (k % (S / 16)) * 2 + (k / (S / 16)) * aSlab),
        b + (uint64_t)(int64_t)((k % (S / 16)) * 2 + (k / (S / 16)) * bSlab + t * bTap), idesc, fresh ? 0u : 1u);
}
template <int S, int K>
__device__ __forceinline__ void issueTile(uint32_t acc, const uint64_t (&a)[3], uint64_t b, uint32_t aSlab, int bSlab,
                                          int bTap, uint32_t idesc) {
#pragma unroll
    for (int t = 0; t < 9; t++)
#pragma unroll
        for (int k = 0; k < K; k++) issueStep<S>(acc, a, b, aSlab, bSlab, bTap, idesc, t, k, t == 0 && k == 0);
}
// The same for one slab of a streamed layer: chunks of 16 channels outer.
template <int S>
__device__ __forceinline__ void issueSlab(uint32_t acc, const uint64_t (&a)[3], uint64_t b, int bTap, uint32_t idesc,
                                          bool first) {
#pragma unroll
    for (int k = 0; k < S / 16; k++)
#pragma unroll
        for (int t = 0; t < 9; t++) issueStep<S>(acc, a, b, 0u, 0, bTap, idesc, t, k, first && t == 0 && k == 0);
}
// The K steps a slab width occurs with (cin / 16 of the network's layers).
template <int S>
__device__ __forceinline__ void issueTileK(int k, uint32_t acc, const uint64_t (&a)[3], uint64_t b, uint32_t aSlab,
                                           int bSlab, int bTap, uint32_t idesc) {
    if constexpr (S == 16) {
        if (k == 1) issueTile<S, 1>(acc, a, b, aSlab, bSlab, bTap, idesc);
        else if (k == 3) issueTile<S, 3>(acc, a, b, aSlab, bSlab, bTap, idesc);
        else if (k == 5) issueTile<S, 5>(acc, a, b, aSlab, bSlab, bTap, idesc);
        else issueTile<S, 7>(acc, a, b, aSlab, bSlab, bTap, idesc);
    } else if constexpr (S == 32) {
        if (k == 2) issueTile<S, 2>(acc, a, b, aSlab, bSlab, bTap, idesc);
        else if (k == 6) issueTile<S, 6>(acc, a, b, aSlab, bSlab, bTap, idesc);
        else if (k == 10) issueTile<S, 10>(acc, a, b, aSlab, bSlab, bTap, idesc);
        else issueTile<S, 14>(acc, a, b, aSlab, bSlab, bTap, idesc);
    } else {
        if (k == 4) issueTile<S, 4>(acc, a, b, aSlab, bSlab, bTap, idesc);
        else issueTile<S, 8>(acc, a, b, aSlab, bSlab, bTap, idesc);
    }
}
inline bool knownCin(int cin) {
    for (int c : {16, 32, 48, 64, 80, 96, 112, 128, 160, 224})
        if (c == cin) return true;
    return false;
}

// Unit u: image, first column and row and rows of a strip of a segment, and its tiles.
struct Unit { int img, x0, y0, rows, tiles; };
__device__ __forceinline__ Unit unitOf(const NarrowArgs& a, int u) {
    const int column = u / a.strips, img = column / a.segments, x0 = (column - img * a.segments) * a.segWidth;
    const int y0 = (u - column * a.strips) * a.rows, rows = min(a.rows, a.h - y0);
    return Unit{img, x0, y0, rows, (rows * a.pitch + kTile - 1) / kTile};
}

// STREAM: a stage is one slab of a strip and of the block's weights; else all
// slabs of a strip, with the weights resident.
template <int S, bool STREAM>
__global__ void __launch_bounds__(kThreads) convNarrowKernel(const __grid_constant__ CUtensorMap inMap,
                                                            const __grid_constant__ CUtensorMap wMap, NarrowArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = smemAddr(smem);
    volatile int* abortFlag = reinterpret_cast<volatile int*>(smem + Header::abort);
    const uint32_t wAddr = base + kHeader, stage0 = wAddr + a.weightSpace;
    const uint64_t limit = a.waitLimitNs;
    if (base & 1023u) {  // swizzled slabs need an aligned base: report, touch nothing
        if (threadIdx.x == 0) atomicExch(a.errorFlag, 1);
        return;
    }
    const int nBase = (int)(blockIdx.x % (unsigned)a.slices) * a.cout;
    const int firstUnit = (int)(blockIdx.x / (unsigned)a.slices), unitStride = (int)(gridDim.x / (unsigned)a.slices);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; s++) {
            barInit(base + Header::full + 8 * s, 1);
            barInit(base + Header::empty + 8 * s, 1);
        }
        for (int s = 0; s < 3; s++) barInit(base + Header::weights + 8 * s, 1);
        for (int s = 0; s < 2 * kMaxTiles; s++) {
            barInit(base + Header::accFull + 8 * s, 1);
            barInit(base + Header::accEmpty + 8 * s, 4);  // the four warps that drain the tile
        }
        barInit(base + Header::drain, 1);
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        // The weights before the wait for the previous kernel: it does not
        // write them (see rt_conv_pipe.cu). Kernel row r's taps as they are
        // used (the data gradient reads the taps reversed).
        for (int r = 0; r < 3 && !STREAM; r++) {
            const int row = a.reverseTaps ? 2 - r : r;
            barExpectTx(base + Header::weights + 8 * r, a.weightBytes / 3u);
            for (int j = 0; j < a.slabs; j++)
                tmaLoad3(wAddr + (uint32_t)((j * 9 + row * 3) * a.cout) * 2u * S, &wMap, j * S, nBase, row * 3,
                         base + Header::weights + 8 * r);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + Header::tmemSlot),
                     "r"(a.tmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        // The next kernel may start its setup only now: started before this
        // block's allocation, a block of it on the same SM could take the
        // columns first and keep them while it waits for this kernel.
        asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    float* sBias = reinterpret_cast<float*>(smem + Header::bias);
    for (int c = threadIdx.x; c < a.cout; c += kThreads) sBias[c] = a.bias ? a.bias[nBase + c] : 0.0f;
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + Header::tmemSlot);

    if (warp == 0) {
        // ---- producer ----
        // Fill k: a strip (STREAM: a slab of one) in stage k % stages.
        int k = 0;
        bool ok = true;
        const int perFill = STREAM ? 1 : a.slabs;
        for (int u = firstUnit; u < a.units && ok; u += unitStride) {
            const Unit U = unitOf(a, u);
            for (int first = 0; first < a.slabs; first += perFill, k++) {
                const int st = k % a.stages;
                if (!waitPhaseWarp(base + Header::empty + 8 * st, (uint32_t)(((k / a.stages) & 1) ^ 1), abortFlag, limit)) { ok = false; break; }
                if (lane == 0) {
                    const uint32_t fb = base + Header::full + 8 * st, stage = stage0 + (uint32_t)st * a.stageBytes;
                    barExpectTx(fb, (uint32_t)(perFill * (a.rows + 2) * a.pitch) * 2u * S + (STREAM ? a.weightBytes : 0u));
                    for (int j = 0; j < perFill; j++)
                        tmaLoad4(stage + (uint32_t)j * a.slabBytes, &inMap, (first + j) * S, U.x0 - 1, U.y0 - 1, U.img, fb);
                    if (STREAM)
                        for (int r = 0; r < 3; r++)
                            tmaLoad3(stage + a.slabBytes + (uint32_t)(r * 3 * a.cout) * 2u * S, &wMap, first * S, nBase, r * 3, fb);
                }
                __syncwarp();
            }
        }
        if (!ok) *abortFlag = 1;
        // Every issued load lands before the block exits.
        if (lane == 0) {
            for (int r = 0; r < 3 && !STREAM; r++) pollPhase(base + Header::weights + 8 * r, 0u, limit);
            for (int e = k > a.stages ? k - a.stages : 0; e < k; e++)
                pollPhase(base + Header::full + 8 * (e % a.stages), (uint32_t)((e / a.stages) & 1), limit);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer ----
        if (lane == 0) {
            bool ok = true;
            const uint32_t idesc = ummaInstrDescBf16(kTile, a.cout);
            const uint64_t wDesc = rowsDescriptor<S>(wAddr);
            const uint32_t aSlab = a.slabBytes >> 4;
            const int wTap = a.cout * 2 * S / 16, bTap = a.reverseTaps ? -wTap : wTap;
            const uint64_t b = a.reverseTaps ? wDesc + (uint64_t)(8 * wTap) : wDesc;
            int k = 0, strip = 0;  // fills and strips so far
            uint32_t used[2] = {0u, 0u};  // per set, bit i: parity of tile i's uses so far
            for (int u = firstUnit; u < a.units && ok; u += unitStride, strip++) {
                const int set = a.sets == 2 ? strip & 1 : 0;
                const Unit U = unitOf(a, u);
                const uint32_t pitch = (uint32_t)a.pitch * 2u * S;
                for (int j = 0; j < (STREAM ? a.slabs : 1) && ok; j++, k++) {
                    const int st = k % a.stages;
                    ok = waitPhase(base + Header::full + 8 * st, (uint32_t)((k / a.stages) & 1), abortFlag, limit);
                    for (int r = 0; r < 3 && ok && k == 0 && !STREAM; r++)
                        ok = waitPhase(base + Header::weights + 8 * r, 0u, abortFlag, limit);
                    if (!ok) break;
                    uint32_t line = stage0 + (uint32_t)st * a.stageBytes;
                    const uint64_t bSlab = STREAM ? b + (uint64_t)((line + a.slabBytes - wAddr) >> 4) : b;
                    for (int i = 0; i < U.tiles; i++, line += kTile * 2 * S) {
                        if (j == 0) {
                            // The tile's accumulator drained since its last use.
                            ok = waitPhase(base + Header::accEmpty + 8 * (set * kMaxTiles + i),
                                           (((set ? used[1] : used[0]) >> i) & 1u) ^ 1u, abortFlag, limit);
                            if (!ok) break;
                            if (set) used[1] ^= 1u << i;
                            else used[0] ^= 1u << i;
                        }
                        tcFenceAfter();
                        const uint64_t rows[3] = {rowsDescriptor<S>(line), rowsDescriptor<S>(line + pitch),
                                                  rowsDescriptor<S>(line + 2 * pitch)};
                        const uint32_t acc = tmem + (uint32_t)set * a.setCols + (uint32_t)(i * a.cout);
                        if (STREAM) issueSlab<S>(acc, rows, bSlab, bTap, idesc, j == 0);
                        else issueTileK<S>(a.cin / 16, acc, rows, b, aSlab, 9 * wTap, bTap, idesc);
                        if (!STREAM || j == a.slabs - 1) commit(base + Header::accFull + 8 * (set * kMaxTiles + i));
                    }
                    if (!ok) break;
                    commit(base + Header::empty + 8 * st);
                }
            }
            if (ok) {
                // The commits' arrivals land before shared memory goes away.
                for (int e = k > a.stages ? k - a.stages : 0; e < k; e++)
                    pollPhase(base + Header::empty + 8 * (e % a.stages), (uint32_t)((e / a.stages) & 1), limit);
            } else {
                *abortFlag = 1;
                commit(base + Header::drain);
                pollPhase(base + Header::drain, 0u, limit);
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue: warps 2-5 the even tiles, 6-9 the odd ones ----
        const int quarter = warp & 3, parity = (warp - 2) >> 2;
        int k = 0;
        bool ok = true;
        // Per accumulator set, the phase of each tile's barrier: a tile's
        // barrier completes once per strip that has the tile.
        uint32_t phases[2] = {0u, 0u};
        for (int u = firstUnit; u < a.units && ok; u += unitStride, k++) {
            const int set = a.sets == 2 ? k & 1 : 0;
            const Unit U = unitOf(a, u);
            for (int i = parity; i < U.tiles; i += 2) {
                if (!waitPhaseWarp(base + Header::accFull + 8 * (set * kMaxTiles + i), ((set ? phases[1] : phases[0]) >> i) & 1u,
                                   abortFlag, limit)) { ok = false; break; }
                if (set) phases[1] ^= 1u << i;
                else phases[0] ^= 1u << i;
                tcFenceAfter();
                const int m = i * kTile + quarter * 32 + lane, row = m / a.pitch, col = m - row * a.pitch, x = U.x0 + col;
                const bool inside = col < a.segWidth && x < a.w && row < U.rows;
                const size_t pix = ((size_t)U.img * a.h + U.y0 + row) * a.w + x;
                for (int c = 0; c < a.cout; c += 16) {
                    uint32_t r[16];
                    __syncwarp();  // the load needs converged lanes; the stores below diverge
                    tmemLoad16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)set * a.setCols + (uint32_t)(i * a.cout + c), r);
                    if (!inside) continue;
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        v[j] = __uint_as_float(r[j]) + sBias[c + j];
                        v[j] = a.relu ? fmaxf(v[j], 0.0f) : v[j];
                    }
                    if (a.outF) {
                        float4* o = reinterpret_cast<float4*>(a.outF + pix * a.coutTotal + nBase + c);
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            uint32_t words[8];
#pragma unroll
                            for (int j = 0; j < 8; j += 4) {
                                float4 s = make_float4(v[8 * q + j], v[8 * q + j + 1], v[8 * q + j + 2], v[8 * q + j + 3]);
                                if (a.accumulate) {
                                    const float4 old = o[2 * q + j / 4];
                                    s = make_float4(old.x + s.x, old.y + s.y, old.z + s.z, old.w + s.w);
                                }
                                words[j] = __float_as_uint(s.x); words[j + 1] = __float_as_uint(s.y);
                                words[j + 2] = __float_as_uint(s.z); words[j + 3] = __float_as_uint(s.w);
                            }
                            storeWords8(o + 2 * q, words);
                        }
                    } else {
                        uint32_t words[8];
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                            words[j] = *reinterpret_cast<uint32_t*>(&pair);
                        }
                        storeWords8(a.outB + pix * a.coutTotal + nBase + c, words);
                    }
                }
                tcFenceBefore();
                __syncwarp();
                if (lane == 0) barArrive(base + Header::accEmpty + 8 * (set * kMaxTiles + i));
            }
        }
    }
    tcFenceBefore();
    __syncthreads();
    if (threadIdx.x == 0 && *abortFlag) atomicExch(a.errorFlag, 1);
    if (warp == 1) {
        tcFenceAfter();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(a.tmemCols)
                     : "memory");
    }
}

template <int S, bool STREAM>
cudaError_t launch(const CUtensorMap& inMap, const CUtensorMap& wMap, const NarrowArgs& a, int grid, uint32_t smemBytes,
                   cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(convNarrowKernel<S, STREAM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)kThreads);
    cfg.dynamicSmemBytes = smemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, convNarrowKernel<S, STREAM>, inMap, wMap, a);
}
template <int S>
cudaError_t launchC(bool chunked, const CUtensorMap& inMap, const CUtensorMap& wMap, const NarrowArgs& a, int grid,
                    uint32_t smemBytes, cudaStream_t stream) {
    return chunked ? launch<S, true>(inMap, wMap, a, grid, smemBytes, stream)
                   : launch<S, false>(inMap, wMap, a, grid, smemBytes, stream);
}

}  // namespace

cudaError_t convNarrow(const bf16* in, int n, int h, int w, int cin, const bf16* weights, bool reverseTaps,
                       const float* bias, int cout, bf16* outB, float* outF, bool relu, bool accumulate, bool chunked,
                       int* errorFlag, cudaStream_t stream) {
    if (n < 1 || h < 1 || w < 1 || !knownCin(cin) || cout < 16 || cout % 16 || (!outB && !outF) || !errorFlag)
        return cudaErrorNotSupported;
    const int S = slabChannels(cin);
    NarrowArgs a{};
    a.n = n; a.h = h; a.w = w; a.cin = cin; a.coutTotal = cout;
    // Columns in equal segments of up to kNarrowWidth, each with its own halo.
    a.segments = (w + kNarrowWidth - 1) / kNarrowWidth;
    a.segWidth = (w + a.segments - 1) / a.segments;
    a.pitch = a.segWidth + 2;
    a.slabs = cin / S;
    int sms = 0, device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    sms = std::max(1, sms);
    // Slices of the output channels and rows per strip: the pair whose
    // busiest block takes the fewest cycles, counting about 60 per MMA (N up
    // to 64; half a cycle per column above 120), 24 bytes per cycle from L2 for
    // the weights and the first strip, and the larger of the two per strip
    // after that (their sum where only one stage fits).
    double best = -1.0;
    long long bestPer = 0;
    for (int s = 1; s <= cout / 16; s++) {
        const int slice = cout / s;
        if (cout % s || slice % 16 || slice > 128) continue;
        const int held = chunked ? S : cin;  // input channels whose weights are held at a time
        const uint32_t weightBytes = 9u * (uint32_t)held * (uint32_t)slice * 2u, space = (weightBytes + 1023u) & ~1023u;
        const int perSlice = std::max(1, sms / s);
        for (int rows = 1; rows <= std::min(h, 254); rows++) {
            const int tiles = (rows * a.pitch + kTile - 1) / kTile;
            if (tiles > kMaxTiles || tiles * slice > 512) break;
            // The last tile reads up to 2 rows and 2 pixels past its start + 128.
            const int line = std::max((rows + 2) * a.pitch, tiles * kTile + 2 * a.pitch + 2);
            const uint32_t slabBytes = ((uint32_t)line * 2u * (uint32_t)S + 1023u) & ~1023u;
            const uint32_t stage = chunked ? slabBytes + space : (uint32_t)a.slabs * slabBytes;
            const uint32_t fixed = kHeader + (chunked ? 0u : space);
            if (fixed + stage > kSmemMax) break;
            const int strips = (h + rows - 1) / rows;
            const long long units = (long long)n * a.segments * strips;
            if (units * s > 0x7FFFFFFFll) continue;
            const long long per = (units + perSlice - 1) / perSlice, fills = chunked ? per * a.slabs : per;
            const int stages = (int)std::min<long long>({fills, chunked ? kMaxStages : 2, (kSmemMax - fixed) / stage});
            const double mmas = tiles * 9.0 * (held / 16) * std::max(60.0, slice * 0.55), load = stage / 24.0;
            const double cost = 3000.0 + (chunked ? 0.0 : weightBytes / 24.0) + load + mmas + tiles * 150.0 +
                                (double)(fills - 1) * (stages >= 2 ? std::max(mmas, load) + 300.0 : mmas + load + 1000.0);
            if (best >= 0.0 && cost >= best) continue;
            best = cost;
            bestPer = per;
            a.cout = slice; a.slices = s;
            a.rows = rows; a.strips = strips; a.units = (int)units;
            a.slabBytes = slabBytes; a.stageBytes = stage; a.weightBytes = weightBytes; a.weightSpace = chunked ? 0u : space;
            a.stages = stages;
            a.setCols = (uint32_t)(tiles * slice);
            a.sets = per > 1 && 2u * a.setCols <= 512u ? 2 : 1;
        }
    }
    if (best < 0.0) return cudaErrorNotSupported;
    // Wider images whose weights stay resident: only small ones, whose strips
    // load behind the MMAs. One 1080p inference, this kernel against the
    // pipelined one (us): 64 -> 64 at 480 x 272 25 / 33, 48 -> 64 22 / 30,
    // 64 -> 96 at 240 x 136 12 / 19, 128 -> 128 at 120 x 68 11 / 23; but
    // 96 -> 96 at 240 x 136, one stage and two strips per block, 30 / 25, and
    // 48 -> 48 at 960 x 544 61 / 48. Streamed layers at any size: 224 -> 96 at
    // 240 x 136 22 us against 71 in the single-role kernel.
    if (!chunked && w > kNarrowWidth && ((long long)n * h * w > 1024ll * sms || (bestPer > 1 && a.stages < 2)))
        return cudaErrorNotSupported;
    a.tmemCols = 32;
    while (a.tmemCols < a.setCols * (uint32_t)a.sets) a.tmemCols <<= 1;
    a.bias = bias; a.outB = outB; a.outF = outF;
    a.relu = relu ? 1 : 0; a.accumulate = accumulate ? 1 : 0; a.reverseTaps = reverseTaps ? 1 : 0;
    a.errorFlag = errorFlag;
    a.waitLimitNs = 1000000000ull;
    auto fn = encodeTiled();
    if (!fn) return cudaErrorNotSupported;
    CUtensorMap inMap{}, wMap{};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    {
        const cuuint64_t dims[4] = {(cuuint64_t)cin, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
        const cuuint64_t strides[3] = {(cuuint64_t)cin * 2, (cuuint64_t)w * cin * 2, (cuuint64_t)h * w * cin * 2};
        const cuuint32_t box[4] = {(cuuint32_t)S, (cuuint32_t)a.pitch, (cuuint32_t)(a.rows + 2), 1};
        if (fn(&inMap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(in), dims, strides, box, elem,
               CU_TENSOR_MAP_INTERLEAVE_NONE, slabSwizzle(S), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorNotSupported;
    }
    {
        const cuuint64_t dims[3] = {(cuuint64_t)cin, (cuuint64_t)cout, 9};
        const cuuint64_t strides[2] = {(cuuint64_t)cin * 2, (cuuint64_t)cout * cin * 2};
        const cuuint32_t box[3] = {(cuuint32_t)S, (cuuint32_t)a.cout, 3};
        if (fn(&wMap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(weights), dims, strides, box, elem,
               CU_TENSOR_MAP_INTERLEAVE_NONE, slabSwizzle(S), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorNotSupported;
    }
    const int grid = (int)std::min<long long>(a.units, std::max(1, sms / a.slices)) * a.slices;
    const uint32_t smemBytes = kHeader + a.weightSpace + (uint32_t)a.stages * a.stageBytes;
    return S == 64   ? launchC<64>(chunked, inMap, wMap, a, grid, smemBytes, stream)
           : S == 32 ? launchC<32>(chunked, inMap, wMap, a, grid, smemBytes, stream)
                     : launchC<16>(chunked, inMap, wMap, a, grid, smemBytes, stream);
}

}  // namespace rt
