// Weight gradient of the denoiser's 3x3 convolutions on the fifth-generation
// tensor cores: dw[tap][ci][co] += sum over pixels p of
// x[p + off(tap)][ci] * dy[p][co], with x and dy NHWC BF16 and dw FP32.
//
// Per tap this is a GEMM whose K is the pixels. An image row segment of up
// to 128 pixels is staged by TMA as slabs of 16, 32 or 64 channels (the
// widest dividing the channel count) with the 32-, 64- or 128-byte swizzle:
// pixel rows of 2 x width bytes, which is the MN-major swizzled operand
// layout (K groups of 8 pixels 16 x width bytes apart, SBO; channel groups a
// slab apart, LBO). The column tap dx is a shift of x's start address by
// pixel rows.
//
// The three row taps are stacked along M: the slabs of x's rows y - 1, y and
// y + 1 follow each other in shared memory, so M runs over (dy, ci) in blocks
// of 128 rows, N over the output channels, and one pass over a dY row feeds
// all nine taps: ceil(3 cin / 128) blocks x 3 column taps of accumulators in
// tensor memory. (One block per row tap, each padding its cin rows to M =
// 128 and staging x and dY again as planes of 8 channels, took 125 us for
// 32 -> 32 channels at 32 x 128 x 128 pixels; this form 50 us. Its floors:
// 67 MB of operands, 10 us; 98,304 MMAs of N = 32, 14 us.)
// Where the accumulators pass 512 columns, blocks of the grid take slices of
// the M blocks. Rows of the last M block beyond 3 cin read the next staged row
// and are dropped (a row of D depends on its row of A only).
//
// K is split over the blocks: each takes a group of consecutive row segments
// (of 128 pixels) in order and adds its accumulators to dw with 16-byte FP32
// reductions at the end. Which products share an accumulator, and in what
// order, decides the rounding of the gradient (2e-6 to 5e-6 of a layer's between
// two groupings, against 1e-7 from the order of the blocks' additions), and
// Adam from fresh moments turns such differences into whole steps of weights
// whose gradient is near zero. So the grouping is part of the training's result
// and is fixed (see wgradTc): not by what balances best, and with the column
// tap as a shift of x, never of dY, whose products would pair up otherwise.
// Spread over all multiprocessors with dY shifted where its channels are one
// slab (all column taps in one MMA of N = 3 cout) the 18 layers of a step took
// 473 us instead of 659 and the layer above 29; beside the backward pass, on a
// stream of its own, that is 1.69 ms a step instead of 1.84.
//
// Segments are staged as wide as the image rounded up to 16 pixels (at most
// 128), so the narrow deep levels do no work for padding; a stage holds up to
// `rows` dY rows and rows + 2 x rows.
//
// Roles: warp 0 issues the TMA loads into two or more stages, warp 1 issues
// the MMAs and owns the tensor memory, warps 2-5 drain the accumulators at
// the end. Waits are bounded as in rt_conv_pipe.cu.
#include <algorithm>
#include <cstdint>

#include "rt_tc_ptx.cuh"

namespace rt {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kM = 128;                 // rows of an M block, and the most pixels per row segment
constexpr int kThreads = 192;
constexpr int kMaxStages = 4;
constexpr int kMaxRows = 8;             // dY rows per stage
constexpr uint32_t kHeader = 1024;
constexpr uint32_t kSmemMax = 227u * 1024u;

// Bytes of a staged row slab of `s` channels x px pixels, on a boundary of
// the swizzle pattern (8 pixel rows).
__host__ __device__ constexpr uint32_t slabBytes(int px, int s) {
    return ((uint32_t)px * 2u * (uint32_t)s + 16u * (uint32_t)s - 1u) & ~(16u * (uint32_t)s - 1u);
}

struct WgradArgs {
    int h, w, cin, cout;
    int px;                        // pixels of a segment that are staged (K per row): 16..128, a multiple of 16
    int tilesPerRow, segments, perGroup;
    int rows;                      // most dY rows per stage
    int xSlabs, dSlabs;            // slabs per row
    uint32_t xSlab, dSlab;         // bytes of one
    uint32_t xBytes, stageBytes;   // x part of a stage, and the whole stage
    int stages;
    int blocksPerSlice, mBlocks;   // M blocks of 128 rows per grid slice, and in all
    uint32_t tmemCols;
    float* dw;
    int* errorFlag;
    unsigned long long waitLimitNs;
};

struct Header {
    static constexpr uint32_t full = 0;                 // kMaxStages
    static constexpr uint32_t empty = 8 * kMaxStages;   // kMaxStages
    static constexpr uint32_t done = 16 * kMaxStages;
    static constexpr uint32_t drain = 16 * kMaxStages + 8;
    static constexpr uint32_t tmemSlot = 16 * kMaxStages + 16;
    static constexpr uint32_t abort = 16 * kMaxStages + 20;
};

// Instruction descriptor: FP32 accumulator, BF16 A and B, both MN-major
// (bits 15 and 16), N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idescMnMajor(int m, int n) {
    return ummaInstrDescBf16(m, n) | (1u << 15) | (1u << 16);
}
// MN-major swizzled operand descriptor of slabs of S channels, `slab` bytes
// apart.
template <int S>
__device__ __forceinline__ uint64_t slabDescriptor(uint32_t addr, uint32_t slab) {
    return ummaSmemDesc(addr, slab, 16u * S) | slabLayout(S);
}

// The MMAs of one dY row and one M block: KK steps of 16 pixels for each
// column tap, descriptors as compile-time offsets from two bases (one thread
// issues; computing descriptors per MMA is several times slower than the
// tensor pipe).
template <int SX, int SD, int KK>
__device__ __forceinline__ void issueRow(uint32_t acc, uint32_t accStep, uint64_t x, uint64_t d, uint32_t idesc,
                                         uint32_t first) {
#pragma unroll
    for (int dx = 0; dx < 3; dx++)
#pragma unroll
        for (int kk = 0; kk < KK; kk++)
            mma(acc + (uint32_t)dx * accStep, x + (uint64_t)(dx * (SX / 8) + kk * 2 * SX), d + (uint64_t)(kk * 2 * SD),
                idesc, (first || kk > 0) ? 1u : 0u);
}
template <int SX, int SD>
__device__ __forceinline__ void issueRowK(int kk, uint32_t acc, uint32_t accStep, uint64_t x, uint64_t d, uint32_t idesc,
                                          uint32_t first) {
    switch (kk) {
        case 1: issueRow<SX, SD, 1>(acc, accStep, x, d, idesc, first); break;
        case 2: issueRow<SX, SD, 2>(acc, accStep, x, d, idesc, first); break;
        case 3: issueRow<SX, SD, 3>(acc, accStep, x, d, idesc, first); break;
        case 4: issueRow<SX, SD, 4>(acc, accStep, x, d, idesc, first); break;
        case 5: issueRow<SX, SD, 5>(acc, accStep, x, d, idesc, first); break;
        case 6: issueRow<SX, SD, 6>(acc, accStep, x, d, idesc, first); break;
        case 7: issueRow<SX, SD, 7>(acc, accStep, x, d, idesc, first); break;
        default: issueRow<SX, SD, 8>(acc, accStep, x, d, idesc, first); break;
    }
}

// The stage that begins at segment s of a group that ends before `end`: image,
// first pixel and first row, and its dY rows (consecutive segments of one
// image where a row is one segment, else one).
struct Strip { int img, x0, y0, rows; };
__device__ __forceinline__ Strip stripAt(const WgradArgs& a, int s, int end) {
    const int row = s / a.tilesPerRow, xt = s - row * a.tilesPerRow, img = row / a.h, y0 = row - img * a.h;
    return Strip{img, xt * kM, y0, a.tilesPerRow == 1 ? min(min(a.rows, a.h - y0), end - s) : 1};
}

template <int SX, int SD>
__global__ void __launch_bounds__(kThreads) wgradTcKernel(const __grid_constant__ CUtensorMap xMap,
                                                         const __grid_constant__ CUtensorMap dMap, WgradArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = smemAddr(smem);
    volatile int* abortFlag = reinterpret_cast<volatile int*>(smem + Header::abort);
    const uint32_t stage0 = base + kHeader;
    const int S = a.stages;
    const uint64_t limit = a.waitLimitNs;
    if (base & 1023u) {  // swizzled slabs need an aligned base: report, touch nothing
        if (threadIdx.x == 0) atomicExch(a.errorFlag, 1);
        return;
    }
    // This block's M blocks, and the slabs of the stacked rows they cover.
    const int b0 = (int)blockIdx.y * a.blocksPerSlice, b1 = min(a.mBlocks, b0 + a.blocksPerSlice);
    const int slab0 = b0 * (kM / SX), slab1 = min(b1 * (kM / SX), 3 * a.xSlabs);
    const int seg0 = (int)blockIdx.x * a.perGroup, seg1 = min(a.segments, seg0 + a.perGroup);  // its group

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            barInit(base + Header::full + 8 * s, 1);
            barInit(base + Header::empty + 8 * s, 1);
        }
        barInit(base + Header::done, 1);
        barInit(base + Header::drain, 1);
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + Header::tmemSlot),
                     "r"(a.tmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + Header::tmemSlot);

    if (warp == 0) {
        // ---- producer: one stage per strip ----
        int k = 0;
        bool ok = true;
        for (int s = seg0; s < seg1; k++) {
            const int st = k % S;
            if (!waitPhaseWarp(base + Header::empty + 8 * st, (uint32_t)(((k / S) & 1) ^ 1), abortFlag, limit)) { ok = false; break; }
            // The lanes issue the boxes: first dY's, then x's.
            const Strip U = stripAt(a, s, seg1);
            s += U.rows;
            const uint32_t fb = base + Header::full + 8 * st;
            const uint32_t xs = stage0 + (uint32_t)st * a.stageBytes, ds = xs + a.xBytes;
            const int dBoxes = U.rows * a.dSlabs, xBoxes = (U.rows + 2) * a.xSlabs;
            // Staged row j (image row y0 - 1 + j) slab c is slab (j - r) xSlabs
            // + c of dY row r's stack: loaded when some r's M blocks cover it.
            auto needed = [&](int i) {
                if (gridDim.y == 1) return true;
                const int j = i / a.xSlabs, c = i - j * a.xSlabs;
                const int rLo = max(0, j - 2), rHi = min(U.rows - 1, j);
                for (int r = rLo; r <= rHi; r++) {
                    const int q = (j - r) * a.xSlabs + c;
                    if (q >= slab0 && q < slab1) return true;
                }
                return false;
            };
            int mine = 0;
            for (int i = lane; i < xBoxes; i += 32) mine += needed(i) ? 1 : 0;
            const uint32_t boxes = (uint32_t)__reduce_add_sync(0xFFFFFFFFu, mine);
            if (lane == 0)
                barExpectTx(fb, boxes * (uint32_t)(a.px + 2) * 2u * SX + (uint32_t)(dBoxes * a.px) * 2u * SD);
            __syncwarp();
            for (int i = lane; i < dBoxes; i += 32) {
                const int r = i / a.dSlabs, c = i - r * a.dSlabs;
                tmaLoad4(ds + (uint32_t)i * a.dSlab, &dMap, c * SD, U.x0, U.y0 + r, U.img, fb);
            }
            for (int i = lane; i < xBoxes; i += 32) {
                const int j = i / a.xSlabs, c = i - j * a.xSlabs;
                if (needed(i)) tmaLoad4(xs + (uint32_t)i * a.xSlab, &xMap, c * SX, U.x0 - 1, U.y0 - 1 + j, U.img, fb);
            }
            __syncwarp();
        }
        if (!ok) *abortFlag = 1;
        // Every issued load lands before the block exits (latest phase of
        // each of the last S stages).
        if (lane == 0)
            for (int e = k > S ? k - S : 0; e < k; e++)
                pollPhase(base + Header::full + 8 * (e % S), (uint32_t)((e / S) & 1), limit);
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer ----
        if (lane == 0) {
            bool ok = true;
            const uint32_t idesc = idescMnMajor(kM, a.cout);
            const uint32_t cols = (uint32_t)a.cout;
            int k = 0, st = 0;
            uint32_t parity = 0, started = 0;
            for (int s = seg0; s < seg1 && ok; k++) {
                ok = waitPhase(base + Header::full + 8 * st, parity, abortFlag, limit);
                if (!ok) break;
                tcFenceAfter();
                const int rows = stripAt(a, s, seg1).rows;
                s += rows;
                uint32_t xs = stage0 + (uint32_t)st * a.stageBytes, ds = xs + a.xBytes;
                for (int r = 0; r < rows; r++) {
                    const uint64_t dDesc = slabDescriptor<SD>(ds, a.dSlab);
                    for (int b = b0; b < b1; b++)
                        issueRowK<SX, SD>(a.px / 16, tmem + (uint32_t)(b - b0) * 3u * cols, cols,
                                          slabDescriptor<SX>(xs + (uint32_t)(b * (kM / SX)) * a.xSlab, a.xSlab), dDesc, idesc, started);
                    started = 1u;
                    xs += (uint32_t)a.xSlabs * a.xSlab;
                    ds += (uint32_t)a.dSlabs * a.dSlab;
                }
                commit(base + Header::empty + 8 * st);
                if (++st == S) { st = 0; parity ^= 1u; }
            }
            if (ok) {
                commit(base + Header::done);
                // The releases' arrivals land before shared memory goes away.
                for (int e = k > S ? k - S : 0; e < k; e++)
                    pollPhase(base + Header::empty + 8 * (e % S), (uint32_t)((e / S) & 1), limit);
            } else {
                *abortFlag = 1;
                commit(base + Header::drain);
                pollPhase(base + Header::drain, 0u, limit);
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue: add the accumulators to dw ----
        const int quarter = warp & 3;
        const bool ok = waitPhaseWarp(base + Header::done, 0u, abortFlag, limit);
        if (ok && seg0 < seg1) {
            tcFenceAfter();
            for (int b = b0; b < b1; b++) {
                const int q = b * kM + quarter * 32 + lane;  // (dy, ci) of this thread's accumulator row
                const int dy = q / a.cin, ci = q % a.cin;
                for (int dx = 0; dx < 3; dx++) {
                    float* out = a.dw + ((size_t)(dy * 3 + dx) * a.cin + ci) * a.cout;
                    for (int c = 0; c < a.cout; c += 16) {
                        uint32_t v[16];
                        __syncwarp();  // the load needs converged lanes; the additions below may diverge
                        tmemLoad16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(((b - b0) * 3 + dx) * a.cout + c), v);
                        if (dy > 2) continue;
#pragma unroll
                        for (int j = 0; j < 16; j += 4)
                            atomicAdd(reinterpret_cast<float4*>(out + c + j),
                                      make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                  __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3])));
                    }
                }
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

// Boxes of one slab of `slab` channels x boxPixels of one row, swizzled;
// zero fill outside the image.
bool makeActivationMap(CUtensorMap* map, const bf16* ptr, int n, int h, int w, int c, int slab, uint32_t boxPixels) {
    auto fn = encodeTiled();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    const cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)w * c * 2, (cuuint64_t)h * w * c * 2};
    const cuuint32_t box[4] = {(cuuint32_t)slab, boxPixels, 1, 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(ptr), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, slabSwizzle(slab), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int SX, int SD>
cudaError_t launch(const CUtensorMap& xMap, const CUtensorMap& dMap, const WgradArgs& a, dim3 grid, uint32_t smemBytes,
                   cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(wgradTcKernel<SX, SD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    wgradTcKernel<SX, SD><<<grid, kThreads, smemBytes, stream>>>(xMap, dMap, a);
    return cudaGetLastError();
}
template <int SX>
cudaError_t launchD(int sd, const CUtensorMap& xMap, const CUtensorMap& dMap, const WgradArgs& a, dim3 grid,
                    uint32_t smemBytes, cudaStream_t stream) {
    return sd == 64   ? launch<SX, 64>(xMap, dMap, a, grid, smemBytes, stream)
           : sd == 32 ? launch<SX, 32>(xMap, dMap, a, grid, smemBytes, stream)
                      : launch<SX, 16>(xMap, dMap, a, grid, smemBytes, stream);
}

}  // namespace

bool wgradTcSupported(int cin, int cout) {
    return cin % 16 == 0 && cout % 16 == 0 && cin >= 16 && cout >= 16 && cout <= 128 && cin <= 256;
}

cudaError_t wgradTc(const bf16* x, const bf16* dy, int n, int h, int w, int cin, int cout, float* dw, int* errorFlag,
                    cudaStream_t stream) {
    if (!wgradTcSupported(cin, cout) || n < 1 || h < 1 || w < 1 || !errorFlag || (reinterpret_cast<uintptr_t>(dw) & 15))
        return cudaErrorNotSupported;
    const int sx = slabChannels(cin), sd = slabChannels(cout);
    WgradArgs a{};
    a.h = h; a.w = w; a.cin = cin; a.cout = cout;
    a.xSlabs = cin / sx; a.dSlabs = cout / sd;
    a.mBlocks = (3 * cin + kM - 1) / kM;
    // As many M blocks per grid slice as 512 columns of accumulators hold,
    // evenly over the slices.
    const int fit = std::min(a.mBlocks, 512 / (3 * cout));
    if (fit < 1) return cudaErrorNotSupported;
    const int slices = (a.mBlocks + fit - 1) / fit;
    a.blocksPerSlice = (a.mBlocks + slices - 1) / slices;
    a.tmemCols = 32;
    while (a.tmemCols < (uint32_t)(a.blocksPerSlice * 3 * cout)) a.tmemCols <<= 1;
    int sms = 0, device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // The groups of segments that are summed in one accumulator. A weight's
    // gradient is rounded as its group sums are, and the first Adam steps carry
    // such roundings on (an update is close to the gradient's sign), so the
    // groups follow from the layer and the image sizes alone: two for every
    // three multiprocessors, fewer where a row tap's input channels pass 128.
    a.tilesPerRow = (w + kM - 1) / kM;
    const long long segments = (long long)n * h * a.tilesPerRow;
    if (segments > 0x7FFFFFFFll) return cudaErrorNotSupported;
    a.segments = (int)segments;
    const int most = std::max(1, 2 * std::max(1, sms) / (3 * (cin >= cout ? (cin + kM - 1) / kM : 1)));
    const int wanted = std::min(a.segments, most);
    a.perGroup = (a.segments + wanted - 1) / wanted;
    const int groups = (a.segments + a.perGroup - 1) / a.perGroup;
    // Rows per stage, by estimated cycles: two stages have to fit; a strip costs
    // the larger of its MMAs (about 60 cycles each for N up to 64, 0.85 N above)
    // and its loads (20 bytes a cycle) and about 1,200 of latency.
    a.px = std::min(kM, (w + 15) / 16 * 16);
    a.xSlab = slabBytes(a.px + 2, sx);
    a.dSlab = slabBytes(a.px, sd);
    // A stage: rows + 2 rows of x, then the dY rows. The last M block may
    // read past the stacked rows, at most `over` bytes past x's part.
    const uint32_t over = (uint32_t)(a.mBlocks * (kM / sx) - 3 * a.xSlabs) * a.xSlab;
    const double mmaCycles = std::max(60.0, 0.85 * cout);
    double bestCost = -1.0;
    for (int rows = 1; rows <= std::min({kMaxRows, h, a.perGroup, a.tilesPerRow == 1 ? kMaxRows : 1}); rows++) {
        const uint32_t xPart = ((uint32_t)((rows + 2) * a.xSlabs) * a.xSlab + 1023u) & ~1023u;
        const uint32_t stage = (xPart + std::max(over, (uint32_t)(rows * a.dSlabs) * a.dSlab) + 1023u) & ~1023u;
        if (kHeader + 2u * stage > kSmemMax) break;
        const double mmas = (double)rows * a.blocksPerSlice * 3 * (a.px / 16) * mmaCycles;
        const double loads = ((rows + 2.0) * (a.px + 2) * cin / slices + (double)rows * a.px * cout) * 2.0 / 20.0;
        const double cost = ((a.perGroup + rows - 1) / rows) * (std::max(mmas, loads) + 1200.0);
        if (bestCost >= 0.0 && cost >= bestCost) continue;
        bestCost = cost;
        a.rows = rows;
        a.xBytes = xPart; a.stageBytes = stage;
    }
    if (bestCost < 0.0) return cudaErrorNotSupported;
    a.stages = 2;
    while (a.stages < kMaxStages && kHeader + (uint32_t)(a.stages + 1) * a.stageBytes <= kSmemMax) a.stages++;
    a.dw = dw;
    a.errorFlag = errorFlag;
    a.waitLimitNs = 1000000000ull;
    CUtensorMap xMap{}, dMap{};
    if (!makeActivationMap(&xMap, x, n, h, w, cin, sx, (uint32_t)(a.px + 2)) ||
        !makeActivationMap(&dMap, dy, n, h, w, cout, sd, (uint32_t)a.px))
        return cudaErrorNotSupported;
    const dim3 grid((unsigned)groups, (unsigned)slices);
    const uint32_t smemBytes = kHeader + (uint32_t)a.stages * a.stageBytes;
    return sx == 64   ? launchD<64>(sd, xMap, dMap, a, grid, smemBytes, stream)
           : sx == 32 ? launchD<32>(sd, xMap, dMap, a, grid, smemBytes, stream)
                      : launchD<16>(sd, xMap, dMap, a, grid, smemBytes, stream);
}

}  // namespace rt
