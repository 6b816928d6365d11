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
// 32 -> 32 channels at 32 x 128 x 128 pixels; this form 29 us. Its floors:
// 67 MB of operands, 10 us; 32,768 MMAs of N = 96, 10 us.)
//
// Where dY's channels are one slab (32 or 64 output channels), the column taps
// sit side by side along N as well: a shift by one pixel is one pixel row of
// the slab, so with a group stride of one pixel row N covers dY shifted by 0,
// 1 and 2 pixels, and one MMA does all nine taps of a block (N = 96 takes ~80
// cycles, three of N = 32 ~42 each and three issues). Then x is staged without
// and dY with the one-pixel halo, and group g holds tap dx = 2 - g. Else the
// tap shifts x's start address.
// Where the accumulators pass 512 columns, blocks of the grid take slices of
// the M blocks. Split K over the blocks; each adds its accumulators to dw
// with 16-byte FP32 reductions at the end. Rows of the last M block beyond 3 cin
// read the next staged row and are dropped (a row of D depends on its row of
// A only).
//
// Segments are as wide as the image rounded up to 16 pixels (at most 128), so the narrow
// deep levels do no work for padding; a stage holds `rows` dY rows and
// rows + 2 x rows.
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
    int xHalo, dHalo;              // pixels staged on each side of a segment (one of them 1)
    int px;                        // pixels per segment (K per row): 16..128, a multiple of 16
    int tilesPerRow, strips, units, rows;
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

// The MMAs of one dY row and one M block: KK steps of 16 pixels, for all
// column taps at once (WIDE) or for each, descriptors as compile-time offsets
// from two bases (one thread issues; computing descriptors per MMA is several
// times slower than the tensor pipe).
template <int SX, int SD, bool WIDE, int KK>
__device__ __forceinline__ void issueRow(uint32_t acc, uint32_t accStep, uint64_t x, uint64_t d, uint32_t idesc,
                                         uint32_t first) {
#pragma unroll
    for (int dx = 0; dx < (WIDE ? 1 : 3); dx++)
#pragma unroll
        for (int kk = 0; kk < KK; kk++)
            mma(acc + (uint32_t)dx * accStep, x + (uint64_t)(dx * (SX / 8) + kk * 2 * SX), d + (uint64_t)(kk * 2 * SD),
                idesc, (first || kk > 0) ? 1u : 0u);
}
template <int SX, int SD, bool WIDE>
__device__ __forceinline__ void issueRowK(int kk, uint32_t acc, uint32_t accStep, uint64_t x, uint64_t d, uint32_t idesc,
                                          uint32_t first) {
    switch (kk) {
        case 1: issueRow<SX, SD, WIDE, 1>(acc, accStep, x, d, idesc, first); break;
        case 2: issueRow<SX, SD, WIDE, 2>(acc, accStep, x, d, idesc, first); break;
        case 3: issueRow<SX, SD, WIDE, 3>(acc, accStep, x, d, idesc, first); break;
        case 4: issueRow<SX, SD, WIDE, 4>(acc, accStep, x, d, idesc, first); break;
        case 5: issueRow<SX, SD, WIDE, 5>(acc, accStep, x, d, idesc, first); break;
        case 6: issueRow<SX, SD, WIDE, 6>(acc, accStep, x, d, idesc, first); break;
        case 7: issueRow<SX, SD, WIDE, 7>(acc, accStep, x, d, idesc, first); break;
        default: issueRow<SX, SD, WIDE, 8>(acc, accStep, x, d, idesc, first); break;
    }
}

// Unit u: image, first pixel and first row, and its dY rows.
struct Unit { int img, x0, y0, rows; };
__device__ __forceinline__ Unit unitOf(const WgradArgs& a, int u) {
    const int strip = u % a.strips, xt = (u / a.strips) % a.tilesPerRow, img = u / (a.strips * a.tilesPerRow);
    const int y0 = strip * a.rows;
    return Unit{img, xt * a.px, y0, min(a.rows, a.h - y0)};
}

template <int SX, int SD, bool WIDE>
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
        // ---- producer: one stage per unit ----
        int k = 0;
        bool ok = true;
        for (int u = (int)blockIdx.x; u < a.units; u += (int)gridDim.x, k++) {
            const int st = k % S;
            if (!waitPhaseWarp(base + Header::empty + 8 * st, (uint32_t)(((k / S) & 1) ^ 1), abortFlag, limit)) { ok = false; break; }
            // The lanes issue the boxes: first dY's, then x's.
            const Unit U = unitOf(a, u);
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
                barExpectTx(fb, boxes * (uint32_t)(a.px + 2 * a.xHalo) * 2u * SX +
                                    (uint32_t)(dBoxes * (a.px + 2 * a.dHalo)) * 2u * SD);
            __syncwarp();
            for (int i = lane; i < dBoxes; i += 32) {
                const int r = i / a.dSlabs, c = i - r * a.dSlabs;
                tmaLoad4(ds + (uint32_t)i * a.dSlab, &dMap, c * SD, U.x0 - a.dHalo, U.y0 + r, U.img, fb);
            }
            for (int i = lane; i < xBoxes; i += 32) {
                const int j = i / a.xSlabs, c = i - j * a.xSlabs;
                if (needed(i)) tmaLoad4(xs + (uint32_t)i * a.xSlab, &xMap, c * SX, U.x0 - a.xHalo, U.y0 - 1 + j, U.img, fb);
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
            const uint32_t idesc = idescMnMajor(kM, WIDE ? 3 * a.cout : a.cout);
            const uint32_t cols = (uint32_t)a.cout;
            int k = 0, st = 0;
            uint32_t parity = 0, started = 0;
            for (int u = (int)blockIdx.x; u < a.units && ok; u += (int)gridDim.x, k++) {
                ok = waitPhase(base + Header::full + 8 * st, parity, abortFlag, limit);
                if (!ok) break;
                tcFenceAfter();
                const int rows = unitOf(a, u).rows;
                uint32_t xs = stage0 + (uint32_t)st * a.stageBytes, ds = xs + a.xBytes;
                for (int r = 0; r < rows; r++) {
                    const uint64_t dDesc = slabDescriptor<SD>(ds, WIDE ? 2u * SD : a.dSlab);
                    for (int b = b0; b < b1; b++)
                        issueRowK<SX, SD, WIDE>(a.px / 16, tmem + (uint32_t)(b - b0) * 3u * cols, cols,
                                          slabDescriptor<SX>(xs + (uint32_t)(b * (kM / SX)) * a.xSlab, a.xSlab), dDesc, idesc,
                                          started);
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
        if (ok && (int)blockIdx.x < a.units) {
            tcFenceAfter();
            for (int b = b0; b < b1; b++) {
                const int q = b * kM + quarter * 32 + lane;  // (dy, ci) of this thread's accumulator row
                const int dy = q / a.cin, ci = q % a.cin;
                for (int dx = 0; dx < 3; dx++) {
                    float* out = a.dw + ((size_t)(dy * 3 + (WIDE ? 2 - dx : dx)) * a.cin + ci) * a.cout;
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

template <int SX, int SD, bool WIDE>
cudaError_t launch(const CUtensorMap& xMap, const CUtensorMap& dMap, const WgradArgs& a, dim3 grid, uint32_t smemBytes,
                   cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(wgradTcKernel<SX, SD, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    wgradTcKernel<SX, SD, WIDE><<<grid, kThreads, smemBytes, stream>>>(xMap, dMap, a);
    return cudaGetLastError();
}
template <int SX>
cudaError_t launchD(int sd, const CUtensorMap& xMap, const CUtensorMap& dMap, const WgradArgs& a, dim3 grid,
                    uint32_t smemBytes, cudaStream_t stream) {
    if (a.dHalo)
        return sd == 64   ? launch<SX, 64, true>(xMap, dMap, a, grid, smemBytes, stream)
               : sd == 32 ? launch<SX, 32, true>(xMap, dMap, a, grid, smemBytes, stream)
                          : launch<SX, 16, true>(xMap, dMap, a, grid, smemBytes, stream);
    return sd == 64   ? launch<SX, 64, false>(xMap, dMap, a, grid, smemBytes, stream)
           : sd == 32 ? launch<SX, 32, false>(xMap, dMap, a, grid, smemBytes, stream)
                      : launch<SX, 16, false>(xMap, dMap, a, grid, smemBytes, stream);
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
    a.dHalo = a.dSlabs == 1 ? 1 : 0;  // the column taps along N (3 cout <= 192)
    a.xHalo = 1 - a.dHalo;
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
    const int most = std::max(1, std::max(1, sms) / slices);
    // Segment width, rows per stage and blocks per slice, by estimated cycles:
    // two stages have to fit; a block's units each cost the larger of their
    // MMAs (about 60 cycles each for N up to 64, 0.85 N above) and loads (20
    // bytes a cycle) and about 1,200 of latency; and every block adds its
    // accumulators to dw, about 800 bytes a cycle over all of them, which is what
    // limits the deep levels (128 -> 128 channels at 8 x 8: 29 MB from 147 blocks).
    const int n0 = a.dHalo ? 3 * cout : cout;
    const double mmaCycles = std::max(60.0, 0.85 * n0);
    const double addCycles = 36.0 * cin * cout / 800.0;
    double bestCost = -1.0;
    int splits = 1;
    for (int px = std::min(kM, (w + 15) / 16 * 16), next = 0; px >= 16; px = next) {
        next = px > 64 ? 64 : px > 32 ? 32 : px > 16 ? 16 : 0;
        const uint32_t xSlab = slabBytes(px + 2 * a.xHalo, sx), dSlab = slabBytes(px + 2 * a.dHalo, sd);
        const int tiles = (w + px - 1) / px;
        // A stage: rows + 2 rows of x, then the dY rows. The last M block may
        // read past the stacked rows, at most `over` bytes past x's part.
        const uint32_t over = (uint32_t)(a.mBlocks * (kM / sx) - 3 * a.xSlabs) * xSlab;
        for (int rows = 1; rows <= std::min(kMaxRows, h); rows++) {
            const uint32_t xPart = ((uint32_t)((rows + 2) * a.xSlabs) * xSlab + 1023u) & ~1023u;
            const uint32_t stage = (xPart + std::max(over, (uint32_t)(rows * a.dSlabs) * dSlab) + 1023u) & ~1023u;
            if (kHeader + 2u * stage > kSmemMax) break;
            const long long strips = (h + rows - 1) / rows, units = (long long)n * tiles * strips;
            if (units > 0x7FFFFFFFll) continue;
            const double mmas = (double)rows * a.blocksPerSlice * (a.dHalo ? 1 : 3) * (px / 16) * mmaCycles;
            const double loads = ((rows + 2.0) * (px + 2) * cin / slices + (double)rows * px * cout) * 2.0 / 20.0;
            const double unit = std::max(mmas, loads) + 1200.0;
            for (int s = most; s >= 1; s = s > 8 ? s * 3 / 4 : s - 1) {
                const long long per = (units + s - 1) / s;
                const double cost = (double)per * unit + s * addCycles;
                if (bestCost >= 0.0 && cost >= bestCost) continue;
                bestCost = cost;
                splits = (int)std::min<long long>(s, units);
                a.px = px; a.rows = rows;
                a.tilesPerRow = tiles; a.strips = (int)strips; a.units = (int)units;
                a.xSlab = xSlab; a.dSlab = dSlab;
                a.xBytes = xPart; a.stageBytes = stage;
            }
        }
    }
    if (bestCost < 0) return cudaErrorNotSupported;
    a.stages = 2;
    while (a.stages < kMaxStages && kHeader + (uint32_t)(a.stages + 1) * a.stageBytes <= kSmemMax) a.stages++;
    a.dw = dw;
    a.errorFlag = errorFlag;
    a.waitLimitNs = 1000000000ull;
    CUtensorMap xMap{}, dMap{};
    if (!makeActivationMap(&xMap, x, n, h, w, cin, sx, (uint32_t)(a.px + 2 * a.xHalo)) ||
        !makeActivationMap(&dMap, dy, n, h, w, cout, sd, (uint32_t)(a.px + 2 * a.dHalo)))
        return cudaErrorNotSupported;
    const dim3 grid((unsigned)splits, (unsigned)slices);
    const uint32_t smemBytes = kHeader + (uint32_t)a.stages * a.stageBytes;
    return sx == 64   ? launchD<64>(sd, xMap, dMap, a, grid, smemBytes, stream)
           : sx == 32 ? launchD<32>(sd, xMap, dMap, a, grid, smemBytes, stream)
                      : launchD<16>(sd, xMap, dMap, a, grid, smemBytes, stream);
}

}  // namespace rt
