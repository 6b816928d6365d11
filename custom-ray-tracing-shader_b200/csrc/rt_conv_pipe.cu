// Warp-specialised 3x3 convolution on the fifth-generation tensor cores,
// fed by TMA: the row-ring form of the denoiser's convolutions.
//
// Implicit GEMM as in rt_conv_tc.cuh: a tile is 128 consecutive output pixels
// of one image row (the MMA's M) and all output channels (N); K runs over
// the 9 taps and the input channels. A block owns strips of rows of one
// 128-pixel column of an image and walks them top to bottom, so every input
// row is staged once per strip and read by the three tiles that need it.
//
// Roles (6 warps):
//   warp 0     producer: TMA loads of the weights (once per block) and of the
//              input rows into a ring of R slots, each row as planes of 8
//              channels x 130 pixels x 16 bytes (the no-swizzle K-major
//              operand layout: core matrices of 8 pixels x 16 bytes, 128
//              bytes apart along M, one plane apart along K). For the
//              decoder's concatenated input [upsample2(low), skip] the skip
//              planes come from one tensor map and the low-resolution row
//              from another into a staging area, which the warp's lanes
//              expand (each low pixel to two) into the slot's first planes.
//   warp 1     MMA issuer (one thread) and tensor-memory owner: per tile 9
//              taps x cin/16 tcgen05.mma into one of two accumulators; a
//              commit tells the epilogue the accumulator is full and another
//              frees the ring slot of the row no later tile reads.
//              The A operand stays in shared memory: with A in tensor
//              memory (tcgen05.cp of each row's three shifted copies) an
//              MMA of 128 x N x 16 measured ~85 SM cycles against ~42 from
//              shared memory. Unsplit 32-channel layers use the stacked-row
//              issue instead (see Seg): per input row and column tap one MMA
//              over the three kernel rows' weights side by side into the
//              accumulator blocks of three output rows, so a row is read
//              by 3 cin/16 MMAs of N = 96 instead of 9 cin/16 of N = 32, and
//              its slot is freed as soon as they complete.
//   warps 2-5  epilogue: tcgen05.ld of the accumulator (warp w of the block
//              reads lanes 32 (w % 4) ...), which is then handed back to the issuer,
//              bias, ReLU and the store (BF16, or FP32 added to or written).
//   warp 6     a second MMA issuer where only one block fits per SM (a single
//              issuing thread per SM issues at about half the tensor pipe's
//              rate): the two issue alternate tiles from the same ring, each
//              into its own accumulators, and both release every row.
// Hand-offs are mbarriers only: full/empty per ring slot, full/empty per
// accumulator, one for the weights. Every wait is bounded by %globaltimer;
// a wait that runs out sets the block's abort flag and the error flag, every
// role leaves its loop, the producer waits (bounded) for its loads in
// flight, the issuer for its MMAs, and the tensor memory is freed.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <type_traits>
#include <vector>

#include "rt_conv_tc.cuh"

namespace rt {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kM = 128;                  // output pixels per tile
constexpr int kHalo = kM + 2;            // input pixels per staged row
constexpr int kLowHalo = kM / 2 + 2;     // low-resolution pixels per staged row
// Bytes of one 8-channel plane of a staged row (130 and 66 pixels x 16
// bytes), padded to 128 bytes: every TMA destination starts on a 128-byte
// boundary.
constexpr uint32_t kPlane = (kHalo * 16 + 127) / 128 * 128;        // 2,176
constexpr uint32_t kLowPlane = (kLowHalo * 16 + 127) / 128 * 128;  // 1,152
constexpr int kPipeThreads = 192;  // warps of one pipeline: producer, MMA issuer, 4 epilogue warps
// Threads of a block: the pipeline, a second issuer (warp 6) for ISS = 2,
// and with EPI = 8 four more epilogue warps (7-10) that drain the second
// half of each accumulator's columns.
__host__ __device__ constexpr int pipeThreads(int iss, int epi) { return kPipeThreads + 32 * (iss - 1) + 32 * (epi - 4); }
constexpr int kMinRing = 3;  // the rows a tile reads; 4 and more let the producer run ahead
constexpr int kMaxRing = 16;
constexpr int kMaxAcc = 8;   // tensor-memory accumulators per block (tiles between the issuer and the epilogue)
constexpr int kLowBufs = 4;  // staging rows of the low-resolution input (loads in flight ahead of the expansion)
constexpr uint32_t kPipeHeader = 512;    // mbarriers (the rest of the header: flags and biases)
constexpr uint32_t kHeader = 2048;       // barriers, flags and biases

// Staged-row layouts. SW = 0: planes of 8 channels x 130 pixels x 16 bytes,
// kPlane apart (no swizzle; one TMA box of 8 channels per plane). SW = 16,
// 32 or 64: slabs of SW channels, one TMA box each with the 32-, 64- or
// 128-byte swizzle, i.e. the K-major swizzled operand layout of that width
// (pixel rows of 2 SW bytes, 8-row groups 16 SW bytes apart), each slab on a
// 1024-byte boundary. A box of 8 channels moves 16 bytes per pixel; the TMA
// unit moved a 1080p row set of 32 channels in 44 us that way, in 27 us as
// 16-channel and 23 us as 32-channel swizzled boxes.
__host__ __device__ constexpr uint32_t slabBytes(int sw) { return ((uint32_t)(kHalo * 2 * sw) + 1023u) & ~1023u; }
// Descriptor units (16 bytes) from a staged row's start to the A operand of
// pixel shift dx (the tap's column) and K step k (16 channels).
template <int SW>
__host__ __device__ constexpr uint32_t aOffset(int dx, int k) {
    return SW == 0 ? (uint32_t)dx + (uint32_t)k * ((2u * kPlane) >> 4)
                   : (uint32_t)dx * (uint32_t)(SW / 8) + (uint32_t)(k / (SW / 16)) * (slabBytes(SW) >> 4) +
                         (uint32_t)(k % (SW / 16)) * 2u;
}
// The A descriptor of a staged row at `addr` (layout type in bits 61-63:
// 6 = 32-byte, 4 = 64-byte, 2 = 128-byte swizzle).
__host__ __device__ constexpr uint64_t rowDescriptor(uint32_t addr, int sw) {
    return sw == 0 ? ummaSmemDesc(addr, kPlane, 128u)
                   : ummaSmemDesc(addr, 16u, 16u * (uint32_t)sw) | ((uint64_t)(sw == 16 ? 6 : sw == 32 ? 4 : 2) << 61);
}
// Offset of the ring from the start of shared memory (its base is 1024-byte
// aligned; the kernel checks): the header, the weights, and for slabs the pad
// to a 1024-byte boundary.
__host__ __device__ constexpr uint32_t ringOffset(uint32_t weightBytes, int sw) {
    return sw ? (kHeader + weightBytes + 1023u) & ~1023u : kHeader + weightBytes;
}
// Staged row bytes of cin channels in layout sw.
__host__ __device__ constexpr uint32_t rowBytes(int cin, int sw) {
    return sw == 0 ? (((uint32_t)(cin / 8) * kPlane + 127u) & ~127u) : (uint32_t)(cin / sw) * slabBytes(sw);
}
// The layout of a layer's rows: the widest slab dividing cin, planes for
// the concatenated input (its low half is expanded into the planes).
__host__ __device__ constexpr int rowLayout(int cin, int lowChannels) {
    return lowChannels ? 0 : cin % 64 == 0 ? 64 : cin % 32 == 0 ? 32 : 16;
}

struct PipeArgs {
    int n, h, w, cin, cout, lowChannels;
    int coutTotal;  // output channels of the layer; a block computes cout of them, from (block % nSplits) * cout
    int nSplits;
    int tilesPerRow, stripRows, strips, units, ring;
    uint32_t weightBytes, slotBytes, lowSlotBytes, accCols, tmemCols;
    const float* bias;
    bf16* outB;
    float* outF;
    int relu, accumulate, reverseTaps;
    int* errorFlag;
    unsigned long long waitLimitNs;
    int probe;  // 1: the issuer first waits on a barrier nothing completes (tests the abort path)
    int nAcc;   // accumulators in tensor memory (2..kMaxAcc)
    int sw;     // staged-row layout (rowLayout)
    // Optional addend of the upsampled half of a decoder convolution, at half
    // resolution: 4 blocks of coutTotal channels per low pixel, block
    // (y % 2) * 2 + x % 2 for output pixel (x, y); added before bias and ReLU.
    const bf16* upAdd;
    long long upPixels;   // low pixels of upAdd (planes of 8 channels: see convTc)
    long long outPixels;  // > 0: BF16 output as planes of 8 channels over this many pixels
    ConvHead head;  // head.out set: the fused 1x1 output head (see ConvHead); activations not stored
    // Optional wait statistics (test hook), nanoseconds summed over blocks:
    // [0] producer waiting for a free slot, [1] producer waiting for a low
    // row, [2] issuer waiting for rows, [3] issuer waiting for a drained
    // accumulator, [4] epilogue waiting for a full accumulator (per warp),
    // [5] block lifetime, [6] stacked issuer inside its MMA issue, [7]
    // stacked issuer committing.
    unsigned long long* stats;
};

// Shared-memory header: mbarriers (8 bytes each) at full, empty, ...; then
// flags and the biases of the block's output channels.
struct Header {
    static constexpr uint32_t full = 0;                    // kMaxRing
    static constexpr uint32_t empty = 8 * kMaxRing;        // kMaxRing
    static constexpr uint32_t lowFull = 16 * kMaxRing;     // kLowBufs
    static constexpr uint32_t accFull = lowFull + 8 * kLowBufs;  // kMaxAcc
    static constexpr uint32_t accEmpty = accFull + 8 * kMaxAcc;
    static constexpr uint32_t drain = accEmpty + 8 * kMaxAcc;
    static constexpr uint32_t weightsFull = drain + 8;     // the weights (loaded once per block)
    static constexpr uint32_t weights = kPipeHeader;
    static constexpr uint32_t probe = weights + 8;
    static constexpr uint32_t tmemSlot = weights + 16;
    static constexpr uint32_t abort = weights + 20;
    static constexpr uint32_t bias = weights + 64;         // the block's output channels' biases (<= 128 floats)
    static constexpr uint32_t head = bias + 128 * 4;       // fused head: per channel {w0, w1, w2, 0} (<= 32 channels)
};
static_assert(Header::weightsFull + 8 <= kPipeHeader && Header::head + 32 * 16 <= kHeader, "header size");

__device__ __forceinline__ uint32_t smemAddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint64_t nowNs() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void barInit(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void barArrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void barExpectTx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool barTryWait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity), "r"(1000u)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool barTestWait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Bounded wait for the phase of parity `parity` to complete. Gives up when
// the block's abort flag is set or when limitNs pass (then sets the flag).
__device__ bool waitPhase(uint32_t bar, uint32_t parity, volatile int* abortFlag, uint64_t limitNs) {
    if (barTryWait(bar, parity)) return true;
    const uint64_t deadline = nowNs() + limitNs;
    for (;;) {
        if (barTryWait(bar, parity)) return true;
        if (*abortFlag) return false;
        if (nowNs() > deadline) { *abortFlag = 1; return false; }
    }
}
// The same for a whole warp: lane 0 waits and every lane gets its verdict,
// so the warp's control flow stays uniform (tcgen05.ld and __syncwarp need
// converged lanes).
__device__ __forceinline__ bool waitPhaseWarp(uint32_t bar, uint32_t parity, volatile int* abortFlag,
                                              uint64_t limitNs) {
    bool ok = true;
    if ((threadIdx.x & 31) == 0) ok = waitPhase(bar, parity, abortFlag, limitNs);
    return __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
}
// Bounded poll that ignores the abort flag (the drains on the abort path).
__device__ void pollPhase(uint32_t bar, uint32_t parity, uint64_t limitNs) {
    const uint64_t deadline = nowNs() + limitNs;
    while (!barTryWait(bar, parity) && nowNs() < deadline) {
    }
}

// TMA loads (no multicast; the tensor maps cover this GPU's memory only).
__device__ __forceinline__ void tmaLoad4(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                         uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n" ::"r"(dst),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tmaLoad3(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tcFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tcFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void mma(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tmemLoad16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmemWaitLoads() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// One tile's 9 taps x G2 MMAs (K steps of 16 channels), every descriptor a
// compile-time offset from the three row descriptors and the weights'. The
// K count must be a compile-time constant: with a runtime inner loop one
// thread issued an MMA per ~155 SM cycles, fully unrolled per ~60 (the tensor
// pipe itself takes ~42 per 128 x N x 16 with N <= 64).
template <int COUT, int G2, int SW>
__device__ __forceinline__ void issueTile(uint32_t acc, const uint64_t (&rowDesc)[3], uint64_t wDesc, uint32_t idesc) {
#pragma unroll
    for (int t = 0; t < 9; t++) {
#pragma unroll
        for (int k = 0; k < G2; k++) {
            const uint64_t aDesc = rowDesc[t / 3] + (uint64_t)aOffset<SW>(t % 3, k);
            const uint64_t bDesc = wDesc + (uint64_t)(((t * 2 * G2 + 2 * k) * COUT * 16) >> 4);
            mma(acc, aDesc, bDesc, idesc, (t > 0 || k > 0) ? 1u : 0u);
        }
    }
}
template <int COUT, int SW>
__device__ __forceinline__ void issueTileK(int G2, uint32_t acc, const uint64_t (&rowDesc)[3], uint64_t wDesc,
                                           uint32_t idesc) {
    switch (G2) {
        case 1: issueTile<COUT, 1, SW>(acc, rowDesc, wDesc, idesc); break;
        case 2: issueTile<COUT, 2, SW>(acc, rowDesc, wDesc, idesc); break;
        case 3: issueTile<COUT, 3, SW>(acc, rowDesc, wDesc, idesc); break;
        case 4: issueTile<COUT, 4, SW>(acc, rowDesc, wDesc, idesc); break;
        case 5: issueTile<COUT, 5, SW>(acc, rowDesc, wDesc, idesc); break;
        case 6: issueTile<COUT, 6, SW>(acc, rowDesc, wDesc, idesc); break;
        case 7: issueTile<COUT, 7, SW>(acc, rowDesc, wDesc, idesc); break;
        case 8: issueTile<COUT, 8, SW>(acc, rowDesc, wDesc, idesc); break;
        case 9: issueTile<COUT, 9, SW>(acc, rowDesc, wDesc, idesc); break;
        case 10: issueTile<COUT, 10, SW>(acc, rowDesc, wDesc, idesc); break;
        case 11: issueTile<COUT, 11, SW>(acc, rowDesc, wDesc, idesc); break;
        case 12: issueTile<COUT, 12, SW>(acc, rowDesc, wDesc, idesc); break;
        case 13: issueTile<COUT, 13, SW>(acc, rowDesc, wDesc, idesc); break;
        default: issueTile<COUT, 14, SW>(acc, rowDesc, wDesc, idesc); break;  // cin <= 224 (convPipeSupported)
    }
}
template <int COUT>
__device__ __forceinline__ void issueTileG(int G2, int sw, uint32_t acc, const uint64_t (&rowDesc)[3], uint64_t wDesc,
                                           uint32_t idesc) {
    switch (sw) {
        case 16: issueTileK<COUT, 16>(G2, acc, rowDesc, wDesc, idesc); break;
        case 32: issueTileK<COUT, 32>(G2, acc, rowDesc, wDesc, idesc); break;
        case 64: issueTileK<COUT, 64>(G2, acc, rowDesc, wDesc, idesc); break;
        default: issueTileK<COUT, 0>(G2, acc, rowDesc, wDesc, idesc); break;
    }
}

// The stacked-row form: an input row r feeds output rows r + 1, r and r - 1
// through the kernel rows dy = 0, 1, 2, so one MMA per column tap dx and K
// step multiplies the row (A, read once) by the three kernel rows' weights
// side by side along N (B: [dy = 2 | dy = 1 | dy = 0] x COUT, N = 3 COUT)
// into three consecutive accumulator blocks (output rows r - 1, r, r + 1) of
// a ring of blocks in tensor memory. Where that range wraps around the ring,
// or at a strip's first and last rows, the MMA covers fewer blocks (Seg: the
// first block's column, the B offset of its kernel row in descriptor units,
// the instruction descriptor for its width and the accumulate flag). An
// output row's first MMA (input row r + 1's dy = 0, dx = 0, first K step)
// starts its block from zero: that step issues the fresh block apart.
// Each output row thus receives the taps in the order t = 3 dy + dx with the
// K steps inner, the tap-per-tile form's order.
struct Seg { uint32_t d, b, id, acc; };
template <int COUT, int G2, int SW>
__device__ __forceinline__ void issueRowStacked(const Seg (&first)[3], int nFirst, const Seg (&rest)[2], int nRest,
                                                uint64_t aDesc, uint64_t wDesc) {
#pragma unroll
    for (int dx = 0; dx < 3; dx++) {
#pragma unroll
        for (int k = 0; k < G2; k++) {
            const uint64_t ad = aDesc + (uint64_t)aOffset<SW>(dx, k);
            // Weights: per (dx, plane g) a region of 3 COUT rows of 16 bytes.
            const uint64_t bd = wDesc + (uint64_t)(((dx * 2 * G2 + 2 * k) * 3 * COUT * 16) >> 4);
            if (dx == 0 && k == 0) {
#pragma unroll
                for (int s = 0; s < 3; s++)
                    if (s < nFirst) mma(first[s].d, ad, bd + first[s].b, first[s].id, first[s].acc);
            } else {
                mma(rest[0].d, ad, bd + rest[0].b, rest[0].id, 1u);
                if (nRest > 1) mma(rest[1].d, ad, bd + rest[1].b, rest[1].id, 1u);
            }
        }
    }
}
template <int COUT, int SW>
__device__ __forceinline__ void issueRowStackedK(int G2, const Seg (&first)[3], int nFirst, const Seg (&rest)[2],
                                                 int nRest, uint64_t aDesc, uint64_t wDesc) {
    switch (G2) {
        case 1: issueRowStacked<COUT, 1, SW>(first, nFirst, rest, nRest, aDesc, wDesc); break;
        case 2: issueRowStacked<COUT, 2, SW>(first, nFirst, rest, nRest, aDesc, wDesc); break;
        case 3: issueRowStacked<COUT, 3, SW>(first, nFirst, rest, nRest, aDesc, wDesc); break;
        case 4: issueRowStacked<COUT, 4, SW>(first, nFirst, rest, nRest, aDesc, wDesc); break;
        case 5: issueRowStacked<COUT, 5, SW>(first, nFirst, rest, nRest, aDesc, wDesc); break;
        case 6: issueRowStacked<COUT, 6, SW>(first, nFirst, rest, nRest, aDesc, wDesc); break;
        case 7: issueRowStacked<COUT, 7, SW>(first, nFirst, rest, nRest, aDesc, wDesc); break;
        default: issueRowStacked<COUT, 8, SW>(first, nFirst, rest, nRest, aDesc, wDesc); break;  // cin <= 128 (host check)
    }
}
template <int COUT>
__device__ __forceinline__ void issueRowStackedG(int G2, int sw, const Seg (&first)[3], int nFirst, const Seg (&rest)[2],
                                                 int nRest, uint64_t aDesc, uint64_t wDesc) {
    switch (sw) {
        case 16: issueRowStackedK<COUT, 16>(G2, first, nFirst, rest, nRest, aDesc, wDesc); break;
        case 32: issueRowStackedK<COUT, 32>(G2, first, nFirst, rest, nRest, aDesc, wDesc); break;
        case 64: issueRowStackedK<COUT, 64>(G2, first, nFirst, rest, nRest, aDesc, wDesc); break;
        default: issueRowStackedK<COUT, 0>(G2, first, nFirst, rest, nRest, aDesc, wDesc); break;
    }
}

// Unit u: image, column tile and strip of rows [y0, y1).
struct Unit { int img, x0, y0, y1; };
__device__ __forceinline__ Unit unitOf(const PipeArgs& a, int u) {
    const int strip = u % a.strips, xt = (u / a.strips) % a.tilesPerRow, img = u / (a.strips * a.tilesPerRow);
    const int y0 = strip * a.stripRows;
    return Unit{img, xt * kM, y0, min(a.h, y0 + a.stripRows)};
}

// The upsampled-half addend of output pixel (x, y) (see PipeArgs::upAdd),
// loaded before the epilogue waits for its accumulator so the load's latency
// overlaps the wait (COUT <= 64; wider layers take no addend).
__host__ __device__ constexpr int upWords(int cout) { return cout <= 64 ? cout / 8 : 1; }
template <int COUT>
__device__ __forceinline__ void loadUpAddend(const PipeArgs& a, int img, int y, int x, int nBase,
                                             uint4 (&u)[upWords(COUT)]) {
    // Planes of 8 channels over the low pixels: block (y % 2) * 2 + x % 2's
    // channels nBase ... are planes (block * coutTotal + nBase) / 8 + q.
    const size_t low = ((size_t)img * (a.h / 2) + y / 2) * (a.w / 2) + x / 2;
    const size_t plane0 = (size_t)(((y & 1) * 2 + (x & 1)) * a.coutTotal + nBase) / 8;
    const uint4* src = reinterpret_cast<const uint4*>(a.upAdd);
#pragma unroll
    for (int q = 0; q < upWords(COUT); q++) u[q] = __ldg(src + (plane0 + q) * (size_t)a.upPixels + low);
}
// How a tile's accumulators leave the block.
enum class Out {
    Rows,     // BF16 pixel rows
    RowsUp,   // the same with the upsampled addend
    Head,     // the fused 1x1 head
    General,  // FP32, or BF16 planes, with or without the addend
};
__device__ __forceinline__ Out outputForm(const PipeArgs& a) {
    return a.head.out ? Out::Head : a.outF || a.outPixels ? Out::General : a.upAdd ? Out::RowsUp : Out::Rows;
}
__device__ __forceinline__ float2 addPair(float2 x, float2 y) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;\n"
        : "=l"(r)
        : "l"(*reinterpret_cast<const unsigned long long*>(&x)), "l"(*reinterpret_cast<const unsigned long long*>(&y)));
    return *reinterpret_cast<const float2*>(&r);
}
// Bias, the addend, ReLU and the store of 16 output channels (c0 .. c0 + 15
// of the block's COUT) of one pixel, from 16 accumulator columns. The form is
// a template parameter, additions go two at a time (add.rn.f32x2) and ReLU
// follows the rounding to BF16 (the same values: rounding keeps the sign). With
// every form in one body the block issued 542 instructions per 32 pixels of 32
// channels and was idle on no unit long: 1080p 32 -> 32 69 us, now 58 (a copy of
// as many bytes takes 44), 16 -> 32 57 -> 50.
template <int COUT, Out FORM>
__device__ __forceinline__ void epilogueStore16(const PipeArgs& a, const uint32_t (&acc)[16], size_t pix, int c0,
                                                int nBase, const float* bias, const uint4 (&up)[upWords(COUT)],
                                                float2& headSum01, float& headSum2, const float4* headW) {
    float2 v[8];
    const float4* bias4 = reinterpret_cast<const float4*>(bias + c0);  // broadcast from shared memory
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float4 b = bias4[q];
        v[2 * q] = addPair(make_float2(__uint_as_float(acc[4 * q]), __uint_as_float(acc[4 * q + 1])), make_float2(b.x, b.y));
        v[2 * q + 1] = addPair(make_float2(__uint_as_float(acc[4 * q + 2]), __uint_as_float(acc[4 * q + 3])), make_float2(b.z, b.w));
    }
    if (COUT <= 64 && (FORM == Out::RowsUp || (FORM != Out::Rows && a.upAdd))) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&up[c0 / 8 + q]);
#pragma unroll
            for (int j = 0; j < 4; j++) v[4 * q + j] = addPair(v[4 * q + j], __bfloat1622float2(pairs[j]));
        }
    }
    if (FORM == Out::General && a.outF) {
        float4* o = reinterpret_cast<float4*>(a.outF + pix * a.coutTotal + nBase + c0);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            uint32_t words[8];
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const float2 lo = v[4 * q + j / 2], hi = v[4 * q + j / 2 + 1];
                float4 x = make_float4(lo.x, lo.y, hi.x, hi.y);
                if (a.relu) x = make_float4(fmaxf(x.x, 0.0f), fmaxf(x.y, 0.0f), fmaxf(x.z, 0.0f), fmaxf(x.w, 0.0f));
                if (a.accumulate) {
                    const float4 old = o[2 * q + j / 4];
                    x = make_float4(old.x + x.x, old.y + x.y, old.z + x.z, old.w + x.w);
                }
                words[j] = __float_as_uint(x.x); words[j + 1] = __float_as_uint(x.y);
                words[j + 2] = __float_as_uint(x.z); words[j + 3] = __float_as_uint(x.w);
            }
            storeWords8(o + 2 * q, words);
        }
        return;
    }
    __nv_bfloat162 pair[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        pair[j] = __floats2bfloat162_rn(v[j].x, v[j].y);
        if (a.relu) pair[j] = __hmax2(pair[j], __nv_bfloat162(__ushort_as_bfloat16(0), __ushort_as_bfloat16(0)));
    }
    if constexpr (FORM == Out::Head) {
        // The head reads the activations as BF16, channel by channel (its
        // weights from shared memory, one 16-byte broadcast per channel).
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const float2 both = __bfloat1622float2(pair[j / 2]);
            const float x = j & 1 ? both.y : both.x;
            const float4 wv = headW[c0 + j];
            headSum01 = addPair(headSum01, make_float2(__fmul_rn(x, wv.x), __fmul_rn(x, wv.y)));
            headSum2 += x * wv.z;
        }
    } else {
        uint32_t words[8];
#pragma unroll
        for (int j = 0; j < 8; j++) words[j] = *reinterpret_cast<uint32_t*>(&pair[j]);
        if (FORM == Out::General) {
#pragma unroll
            for (int q = 0; q < 2; q++)
                reinterpret_cast<uint4*>(a.outB)[((size_t)(nBase + c0) / 8 + q) * (size_t)a.outPixels + pix] =
                    make_uint4(words[4 * q], words[4 * q + 1], words[4 * q + 2], words[4 * q + 3]);
        } else {
            storeWords8(a.outB + pix * a.coutTotal + nBase + c0, words);
        }
    }
}

// ISS MMA issuers (warp 1, and warp 6 when ISS = 2) share the ring: issuer i
// issues the block's tiles t with t % ISS = i into its own accumulators, and
// every issuer releases every row (a slot's empty barrier counts ISS
// arrivals). Two issuers give a layer that fits one block per SM two issuing
// threads without a second ring.
// STACK: the stacked-row issue (one issuer; a.nAcc blocks of COUT columns).
template <int COUT, int ISS, bool STACK, int EPI>
__global__ void __launch_bounds__(pipeThreads(ISS, EPI), ISS > 1 ? 1 : (COUT <= 48 ? 4 : 2))
    convPipeKernel(const __grid_constant__ CUtensorMap inMap, const __grid_constant__ CUtensorMap lowMap,
                   const __grid_constant__ CUtensorMap wMap, PipeArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int me = (int)(threadIdx.x >> 5) == 6 ? 1 : 0;          // issuer index (warp 6 is the second issuer)
    const int warp = me ? 1 : (int)(threadIdx.x >> 5);            // role: 0 producer, 1 issuer, 2-5 epilogue
    const uint32_t base = smemAddr(smem);
    const uint32_t pb = base;  // barriers
    volatile int* abortFlag = reinterpret_cast<volatile int*>(smem + Header::abort);
    const uint32_t wAddr = base + kHeader;
    const uint32_t slotBytes = a.slotBytes;
    const uint32_t ringAddr = base + ringOffset(a.weightBytes, a.sw);  // slabs: on 1024-byte boundaries
    const uint32_t lowAddr = ringAddr + (uint32_t)a.ring * slotBytes;  // kLowBufs staging rows of the low input
    unsigned char* lowPtr = smem + (lowAddr - base);
    unsigned char* ringPtr = smem + (ringAddr - base);
    const uint64_t blockStart = a.stats ? nowNs() : 0;
    if (a.sw && (base & 1023u)) {  // swizzled slabs need a 1024-byte aligned base: report, touch nothing
        if (threadIdx.x == 0) atomicExch(a.errorFlag, 1);
        return;
    }
    // Planes of 8 channels: the low (upsampled) ones first in a slot, then
    // the full-resolution ones.
    const int G = a.cin / 8, Glow = a.lowChannels / 8, Gin = G - Glow;
    const int R = a.ring;
    const uint64_t limit = a.waitLimitNs;
    // The block's slice of output channels and its units (every nSplits-th
    // block shares a slice; the grid is a multiple of nSplits).
    const int nBase = (int)(blockIdx.x % (unsigned)a.nSplits) * COUT;
    const int firstUnit = (int)(blockIdx.x / (unsigned)a.nSplits);
    const int unitStride = (int)(gridDim.x / (unsigned)a.nSplits);

    if (threadIdx.x == 0) {
        for (int s = 0; s < R; s++) {
            barInit(pb + Header::full + 8 * s, Glow ? 2 : 1);
            barInit(pb + Header::empty + 8 * s, ISS);
        }
        for (int s = 0; s < kLowBufs; s++) barInit(pb + Header::lowFull + 8 * s, 1);
        for (int b = 0; b < ISS * a.nAcc; b++) {  // issuer i's accumulator b at i * nAcc + b
            barInit(pb + Header::accFull + 8 * b, 1);
            barInit(pb + Header::accEmpty + 8 * b, EPI);
        }
        barInit(pb + Header::drain, ISS);
        barInit(pb + Header::weightsFull, 1);
        barInit(base + Header::probe, 1);
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        // The weights, once per block, before the wait for the previous
        // kernel below: no convolution's weights are written by the kernel
        // launched just before it (they come from initialisation, the
        // optimiser or the merge of the two-pass form, each launched without
        // programmatic dependence, so complete before this kernel starts).
        // Tap-major ([tap][plane][cout][8]), or for the stacked form
        // [dx][plane][2 - dy][cout][8]. This thread is the producer's lane 0.
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&wMap) : "memory");
        const uint32_t wb = pb + Header::weightsFull;
        barExpectTx(wb, a.weightBytes);
        for (int t = 0; t < 9; t++)
            for (int g = 0; g < G; g++) {
                const int region = STACK ? ((t % 3) * G + g) * 3 + 2 - t / 3 : t * G + g;
                tmaLoad3(wAddr + (uint32_t)(region * COUT * 16), &wMap, g * 8, nBase, a.reverseTaps ? 8 - t : t, wb);
            }
    }
    if (threadIdx.x >> 5 == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + Header::tmemSlot),
                     "r"(a.tmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        // The next kernel in the stream may start its own setup now, and not
        // before this block holds its tensor memory: a block of the next
        // kernel on the same SM could take the columns first and keep them
        // while it waits for this kernel.
        asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    }
    // Programmatic dependent launch (the host launches with it): this block
    // waits for the previous kernel to complete before any other read of
    // global memory (input rows, bias, addend, the accumulated output).
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    float* sBias = reinterpret_cast<float*>(smem + Header::bias);
    for (int c = threadIdx.x; c < COUT; c += blockDim.x) sBias[c] = a.bias ? a.bias[nBase + c] : 0.0f;
    const float4* sHead = reinterpret_cast<const float4*>(smem + Header::head);
    if (a.head.out)
        for (int c = threadIdx.x; c < COUT && c < 32; c += blockDim.x)
            reinterpret_cast<float4*>(smem + Header::head)[c] =
                make_float4(a.head.wt[c * 3], a.head.wt[c * 3 + 1], a.head.wt[c * 3 + 2], 0.0f);
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + Header::tmemSlot);

    if (warp == 0) {
        // ---- producer ----
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&inMap) : "memory");
            if (Glow) asm volatile("prefetch.tensormap [%0];\n" ::"l"(&lowMap) : "memory");
        }
        // Rows are numbered in issue order q; row q sits in slot q % R, its
        // low-resolution part (concatenated input) in staging buffer
        // q % kLowBufs until the warp expands it into the slot. Rows whose
        // low part has landed are expanded as the producer goes (a test, not
        // a wait), so the loads of later rows are not held up by one row's
        // latency; a staging buffer is expanded before it is loaded again,
        // and every issued row is expanded before the producer blocks on a
        // slot (the issuer may be waiting for exactly those rows).
        int q = 0, expanded = 0;
        uint64_t waitSlotNs = 0, waitLowNs = 0;
        bool ok = true;
        auto lowLanded = [&](int e) -> bool {
            const uint32_t bar = pb + Header::lowFull + 8 * (e % kLowBufs), parity = (uint32_t)((e / kLowBufs) & 1);
            return __shfl_sync(0xFFFFFFFFu, lane == 0 ? (barTestWait(bar, parity) ? 1 : 0) : 0, 0) != 0;
        };
        auto expand = [&](int& e) -> bool {  // expands row e and advances e
            const uint64_t t1 = a.stats ? nowNs() : 0;
            if (!waitPhaseWarp(pb + Header::lowFull + 8 * (e % kLowBufs), (uint32_t)((e / kLowBufs) & 1), abortFlag, limit))
                return false;
            if (a.stats) waitLowNs += nowNs() - t1;
            const uint4* src = reinterpret_cast<const uint4*>(lowPtr + (size_t)(e % kLowBufs) * a.lowSlotBytes);
            uint4* dst = reinterpret_cast<uint4*>(ringPtr + (size_t)(e % R) * slotBytes);
            // Staged pixel p is input x0 - 1 + p, whose low-resolution pixel
            // floor((x0 - 1 + p) / 2) is staged at (p + 1) / 2 (x0 even).
            for (int g = 0; g < Glow; g++) {
                const uint4* srcPlane = src + g * (kLowPlane / 16);
                uint4* dstPlane = dst + g * (kPlane / 16);
#pragma unroll
                for (int k = 0; k < (kHalo + 31) / 32; k++) {
                    const int p = lane + 32 * k;
                    if (p < kHalo) dstPlane[p] = srcPlane[(p + 1) / 2];
                }
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) barArrive(pb + Header::full + 8 * (e % R));
            e++;
            return true;
        };
        for (int u = firstUnit; u < a.units && ok; u += unitStride) {
            const Unit U = unitOf(a, u);
            for (int r = U.y0 - 1; r <= U.y1 && ok; r++) {
                const int s = q % R;
                const uint32_t emptyBar = pb + Header::empty + 8 * s, emptyParity = (uint32_t)(((q / R) & 1) ^ 1);
                if (Glow) {
                    while (ok && expanded < q && lowLanded(expanded)) ok = expand(expanded);
                    while (ok && expanded <= q - kLowBufs) ok = expand(expanded);  // this row's staging buffer
                    const bool freeNow = __shfl_sync(0xFFFFFFFFu, lane == 0 ? (barTestWait(emptyBar, emptyParity) ? 1 : 0) : 0, 0) != 0;
                    while (ok && !freeNow && expanded < q) ok = expand(expanded);
                    if (!ok) break;
                }
                {
                    const uint64_t t1 = a.stats ? nowNs() : 0;
                    if (!waitPhaseWarp(emptyBar, emptyParity, abortFlag, limit)) { ok = false; break; }
                    if (a.stats) waitSlotNs += nowNs() - t1;
                }
                if (lane == 0) {
                    const uint32_t fb = pb + Header::full + 8 * s;
                    const uint32_t slot = ringAddr + (uint32_t)s * slotBytes;
                    barExpectTx(fb, (uint32_t)Gin * kHalo * 16u);  // the boxes' bytes (planes and slabs are padded)
                    if (a.sw) {
                        for (int j = 0; j < a.cin / a.sw; j++)
                            tmaLoad4(slot + (uint32_t)j * slabBytes(a.sw), &inMap, j * a.sw, U.x0 - 1, r, U.img, fb);
                    } else {
                        for (int g = 0; g < Gin; g++)
                            tmaLoad4(slot + (uint32_t)(Glow + g) * kPlane, &inMap, g * 8, U.x0 - 1, r, U.img, fb);
                    }
                    if (Glow) {
                        const uint32_t lb = pb + Header::lowFull + 8 * (q % kLowBufs);
                        const uint32_t ls = lowAddr + (uint32_t)(q % kLowBufs) * a.lowSlotBytes;
                        barExpectTx(lb, (uint32_t)Glow * kLowHalo * 16u);
                        for (int g = 0; g < Glow; g++)
                            tmaLoad4(ls + (uint32_t)g * kLowPlane, &lowMap, g * 8, U.x0 / 2 - 1, r >> 1, U.img, lb);
                    }
                }
                __syncwarp();
                q++;
            }
        }
        while (ok && Glow && expanded < q) ok = expand(expanded);
        // Every load issued must land before the block exits, also when the
        // issuer gave up before reading them: poll the phases of the weights,
        // the staging buffers and the last R slots (each the latest
        // phase of its barrier, so the parities are unambiguous). After a
        // failure, rows not expanded get their second arrival first so
        // their slot's phase can complete.
        if (!ok) *abortFlag = 1;
        if (lane == 0) {
            pollPhase(pb + Header::weightsFull, 0u, limit);
            for (int e = q > kLowBufs ? q - kLowBufs : 0; e < q && Glow; e++)
                pollPhase(pb + Header::lowFull + 8 * (e % kLowBufs), (uint32_t)((e / kLowBufs) & 1), limit);
            for (int e = q > R ? q - R : 0; e < q; e++) {
                if (Glow && e >= expanded) barArrive(pb + Header::full + 8 * (int)(e % R));
                pollPhase(pb + Header::full + 8 * (int)(e % R), (uint32_t)((e / R) & 1), limit);
            }
            if (a.stats) { atomicAdd(a.stats + 0, waitSlotNs); atomicAdd(a.stats + 1, waitLowNs); }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer ----
        // The issue rate of one thread bounds the tensor pipe here (an MMA of
        // 128 x COUT x 16 takes ~42 SM cycles; a single issuer that computes
        // descriptors with divisions per MMA issues one per ~100), so the
        // loop keeps ring positions as running 32-bit counters, makes the
        // three row descriptors once per tile and steps descriptors by
        // constants.
        bool ok = true;
        if (lane == 0) {
            const uint32_t idesc = ummaInstrDescBf16(kM, COUT);
            if (a.probe) ok = waitPhase(base + Header::probe, 0u, abortFlag, limit);
            if (ok)
                ok = waitPhase(pb + Header::weightsFull, 0u, abortFlag, limit);
            uint64_t waitRowNs = 0, waitAccNs = 0, issueNs = 0, commitNs = 0;
            const uint64_t wDesc = ummaSmemDesc(wAddr, COUT * 16u, 128u);
            const int G2 = G / 2;
            int rows = 0, tiles = 0, mine = 0;  // rows waited for, the block's tiles, this issuer's tiles
            int waitSlot = 0, relSlot = 0;      // next row to wait for / to release
            uint32_t waitParity = 0;
            int accB = 0;                       // this issuer's next accumulator (of nAcc)
            uint32_t accParity = 0;
            const int accBase = me * a.nAcc;
            auto nextRow = [&](int& slot) -> bool {
                const uint64_t t1 = a.stats ? nowNs() : 0;
                slot = waitSlot;
                const bool got = waitPhase(pb + Header::full + 8 * waitSlot, waitParity, abortFlag, limit);
                if (a.stats) waitRowNs += nowNs() - t1;
                if (++waitSlot == R) { waitSlot = 0; waitParity ^= 1u; }
                rows++;
                return got;
            };
            auto release = [&]() {
                commit(pb + Header::empty + 8 * relSlot);
                if (++relSlot == R) relSlot = 0;
            };
            if constexpr (STACK) {
                // Per input row i of a strip of S output rows (row y0 - 1 + i,
                // i = 0 .. S + 1): output rows jLo .. jHi of the strip, whose
                // blocks are (p0 + j) % NB for the strip's first block p0 (kept as
                // running counters); block p0 + i is fresh.
                const int NB = a.nAcc;
                const uint64_t wStack = ummaSmemDesc(wAddr, 3u * COUT * 16u, 128u);
                const uint32_t id0 = ummaInstrDescBf16(kM, 0);  // plus (N / 8) << 17 for N = blocks x COUT
                for (int u = firstUnit; u < a.units && ok; u += unitStride) {
                    const Unit U = unitOf(a, u);
                    const int S = U.y1 - U.y0;
                    int pLo = accB;  // block of output row jLo (running, no division)
                    for (int i = 0; i <= S + 1; i++) {
                        int slot = 0;
                        if (!nextRow(slot)) { ok = false; break; }
                        const bool fresh = i < S;
                        if (fresh) {
                            const uint64_t t1 = a.stats ? nowNs() : 0;
                            ok = waitPhase(pb + Header::accEmpty + 8 * accB, accParity ^ 1u, abortFlag, limit);
                            if (a.stats) waitAccNs += nowNs() - t1;
                            if (!ok) break;
                            tcFenceAfter();
                        }
                        const int jLo = i > 2 ? i - 2 : 0, jHi = i < S - 1 ? i : S - 1;
                        // Output rows lo .. hi (lo's block p) as one segment, or two where the ring wraps.
                        auto range = [&](int p, int lo, int hi, uint32_t accFlag, Seg& s0, Seg& s1) -> int {
                            const int len = hi - lo + 1, run = len < NB - p ? len : NB - p;
                            s0 = Seg{tmem + (uint32_t)(p * COUT), (uint32_t)((lo - i + 2) * COUT),
                                     id0 + ((uint32_t)(run * COUT / 8) << 17), accFlag};
                            s1 = Seg{tmem, (uint32_t)((lo + run - i + 2) * COUT),
                                     id0 + ((uint32_t)((len - run) * COUT / 8) << 17), accFlag};
                            return run < len ? 2 : 1;
                        };
                        Seg first[3], rest[2];
                        const int nRest = range(pLo, jLo, jHi, 1u, rest[0], rest[1]);
                        int nFirst = nRest;
                        first[0] = rest[0];
                        first[1] = rest[1];
                        if (fresh) {
                            // The fresh block (output row i = jHi) apart, from zero.
                            Seg fr, unused;
                            range(accB, jHi, jHi, 0u, fr, unused);  // jHi = i: the fresh block
                            if (jHi == jLo) {
                                first[0] = fr;
                                nFirst = 1;
                            } else {
                                nFirst = range(pLo, jLo, jHi - 1, 1u, first[0], first[1]) + 1;
                                if (nFirst == 3) first[2] = fr;
                                else first[1] = fr;
                            }
                        }
                        const uint64_t aDesc = rowDescriptor(ringAddr + (uint32_t)slot * slotBytes, a.sw);
                        const uint64_t t2 = a.stats ? nowNs() : 0;
                        issueRowStackedG<COUT>(G2, a.sw, first, nFirst, rest, nRest, aDesc, wStack);
                        const uint64_t t3 = a.stats ? nowNs() : 0;
                        release();  // row i: no later MMA reads it
                        if (i >= 2) {  // output row i - 2 = jLo has all its taps
                            commit(pb + Header::accFull + 8 * pLo);
                            pLo = pLo + 1 == NB ? 0 : pLo + 1;
                        }
                        if (a.stats) { issueNs += t3 - t2; commitNs += nowNs() - t3; }
                        if (fresh) {
                            mine++;
                            if (++accB == NB) { accB = 0; accParity ^= 1u; }
                        }
                    }
                }
            } else
            for (int u = firstUnit; u < a.units && ok; u += unitStride) {
                const Unit U = unitOf(a, u);
                int s0 = 0, s1 = 0, s2 = 0;  // slots of rows y - 1, y, y + 1
                ok = nextRow(s0) && nextRow(s1);
                for (int y = U.y0; y < U.y1 && ok; y++, tiles++) {
                    if (!nextRow(s2)) { ok = false; break; }
                    if (tiles % ISS == me) {
                        {
                            const uint64_t t1 = a.stats ? nowNs() : 0;
                            ok = waitPhase(pb + Header::accEmpty + 8 * (accBase + accB), accParity ^ 1u, abortFlag, limit);
                            if (a.stats) waitAccNs += nowNs() - t1;
                        }
                        if (!ok) break;
                        tcFenceAfter();
                        const uint32_t acc = tmem + (uint32_t)(accBase + accB) * a.accCols;
                        const uint64_t rowDesc[3] = {rowDescriptor(ringAddr + (uint32_t)s0 * slotBytes, a.sw),
                                                     rowDescriptor(ringAddr + (uint32_t)s1 * slotBytes, a.sw),
                                                     rowDescriptor(ringAddr + (uint32_t)s2 * slotBytes, a.sw)};
                        issueTileG<COUT>(G2, a.sw, acc, rowDesc, wDesc, idesc);
                        commit(pb + Header::accFull + 8 * (accBase + accB));
                        mine++;
                        if (++accB == a.nAcc) { accB = 0; accParity ^= 1u; }
                    }
                    release();  // row y - 1: no later tile reads it (this issuer's arrival)
                    s0 = s1;
                    s1 = s2;
                }
                if (!ok) break;
                release();  // rows y1 - 1 and y1 of the strip: no later tile reads them
                release();
            }
            if (ok) {
                // The commits' arrivals land after the MMAs complete: wait for
                // the last ones (the rows released last, the last
                // accumulators) before the block's shared memory goes away.
                for (int e = rows > R ? rows - R : 0; e < rows; e++)
                    pollPhase(pb + Header::empty + 8 * (e % R), (uint32_t)((e / R) & 1), limit);
                for (int t = mine > a.nAcc ? mine - a.nAcc : 0; t < mine; t++)
                    pollPhase(pb + Header::accFull + 8 * (accBase + t % a.nAcc), (uint32_t)((t / a.nAcc) & 1), limit);
            } else {
                *abortFlag = 1;
                // Wait (bounded) for every MMA issued so far.
                commit(pb + Header::drain);
                pollPhase(pb + Header::drain, 0u, limit);
            }
            if (a.stats) {
                atomicAdd(a.stats + 2, waitRowNs);
                atomicAdd(a.stats + 3, waitAccNs);
                atomicAdd(a.stats + 6, issueNs);
                atomicAdd(a.stats + 7, commitNs);
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue: warps 2-5 (and 7-10), lanes 32 * (warp % 4) ... ----
        // A warp may read only tensor-memory lanes 32 * (its warp index in
        // the block mod 4) ...: warps 2-5 cover the four quarters once, and
        // with EPI = 8 warps 7-10 once more; each set then drains half of
        // the accumulator's columns.
        const int quarter = (int)(threadIdx.x >> 5) & 3;
        constexpr int kChunks = COUT / 16 / (EPI / 4);  // 16-column chunks per warp
        const int chunk0 = EPI == 8 && (threadIdx.x >> 5) >= 7 ? kChunks : 0;
        // Chunks loaded before one wait: all of them (up to 5, else a divisor)
        // where registers allow (one or two blocks per SM), else one.
        constexpr int kGroup = !(ISS == 2 || COUT >= 64) ? 1
                               : kChunks <= 5 ? kChunks : kChunks % 4 == 0 ? 4 : kChunks % 3 == 0 ? 3 : 2;
        const Out form = outputForm(a);
        int bOf[ISS] = {};             // per issuer: next accumulator and its phase
        uint32_t parityOf[ISS] = {};
        int tile = 0;
        uint64_t waitNs = 0;
        bool ok = true;
        for (int u = firstUnit; u < a.units && ok; u += unitStride) {
            const Unit U = unitOf(a, u);
            for (int y = U.y0; y < U.y1; y++, tile++) {
                const int i = tile % ISS;
                const int b = i * a.nAcc + bOf[i];
                const uint32_t parity = parityOf[i];
                if (++bOf[i] == a.nAcc) { bOf[i] = 0; parityOf[i] ^= 1u; }
                const int x = U.x0 + quarter * 32 + lane;
                uint4 up[upWords(COUT)];
                if (COUT <= 64 && a.upAdd && x < a.w) loadUpAddend<COUT>(a, U.img, y, x, nBase, up);
                const uint64_t t1 = a.stats ? nowNs() : 0;
                if (!waitPhaseWarp(pb + Header::accFull + 8 * b, parity, abortFlag, limit)) { ok = false; break; }
                if (a.stats) waitNs += nowNs() - t1;
                tcFenceAfter();
                // 16 accumulator columns at a time: load, finish and store.
                const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)b * a.accCols;
                const size_t pix = ((size_t)U.img * a.h + y) * a.w + x;
                float2 headSum01 = make_float2(0.0f, 0.0f);
                float headSum2 = 0.0f;
                if (form == Out::Head) {
                    headSum01 = make_float2(__ldg(a.head.b), __ldg(a.head.b + 1));
                    headSum2 = __ldg(a.head.b + 2);
                }
                // Up to kGroup chunks of 16 columns loaded before one wait,
                // then finished and stored.
                auto drain = [&](auto formTag) {
                    constexpr Out FORM = decltype(formTag)::value;
#pragma unroll
                    for (int g = 0; g < kChunks; g += kGroup) {
                        uint32_t r[kGroup][16];
                        __syncwarp();  // the loads need converged lanes; the stores below diverge
#pragma unroll
                        for (int c = 0; c < kGroup; c++) tmemLoad16(taddr + (uint32_t)(16 * (chunk0 + g + c)), r[c]);
                        tmemWaitLoads();
#pragma unroll
                        for (int c = 0; c < kGroup; c++)
                            if (x < a.w)
                                epilogueStore16<COUT, FORM>(a, r[c], pix, 16 * (chunk0 + g + c), nBase, sBias, up, headSum01,
                                                            headSum2, sHead);
                    }
                };
                if (form == Out::Rows) drain(std::integral_constant<Out, Out::Rows>());
                else if (COUT <= 64 && form == Out::RowsUp) drain(std::integral_constant<Out, Out::RowsUp>());
                else if (COUT <= 32 && form == Out::Head) drain(std::integral_constant<Out, Out::Head>());
                else drain(std::integral_constant<Out, Out::General>());
                if (form == Out::Head && x < a.head.w && y < a.head.h) {
                    float* o = a.head.out + ((size_t)y * a.head.w + x) * 3;
                    o[0] = fmaxf(expm1f(headSum01.x), 0.0f);
                    o[1] = fmaxf(expm1f(headSum01.y), 0.0f);
                    o[2] = fmaxf(expm1f(headSum2), 0.0f);
                }
                tcFenceBefore();
                __syncwarp();
                if (lane == 0) barArrive(pb + Header::accEmpty + 8 * b);
            }
        }
        if (a.stats && lane == 0) atomicAdd(a.stats + 4, waitNs);
    }
    tcFenceBefore();
    __syncthreads();
    if (threadIdx.x == 0 && *abortFlag) atomicExch(a.errorFlag, 1);
    if (threadIdx.x == 0 && a.stats) atomicAdd(a.stats + 5, nowNs() - blockStart);
    if (threadIdx.x >> 5 == 1) {
        tcFenceAfter();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(a.tmemCols)
                     : "memory");
    }
}

// ---- host ----

PFN_cuTensorMapEncodeTiled_v12000 encodeTiled() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// Rank-4 or rank-3 BF16 tensor map, zero fill outside the tensor; no swizzle,
// or the swizzle of a slab of `sw` channels (rowLayout).
bool makeMap(CUtensorMap* map, const void* ptr, int rank, const uint64_t* dims, const uint64_t* strides,
             const uint32_t* box, int sw = 0) {
    auto fn = encodeTiled();
    if (!fn) return false;
    uint32_t elem[4] = {1, 1, 1, 1};
    const CUtensorMapSwizzle swizzle = sw == 16   ? CU_TENSOR_MAP_SWIZZLE_32B
                                       : sw == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                       : sw == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                                                  : CU_TENSOR_MAP_SWIZZLE_NONE;
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(ptr), dims, strides, box,
              elem, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int deviceSmCount() {
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms > 0 ? sms : 1;
}

template <int COUT, int ISS, bool STACK = false, int EPI = 4>
cudaError_t launchPipe(const CUtensorMap& inMap, const CUtensorMap& lowMap, const CUtensorMap& wMap,
                       const PipeArgs& a, int grid, uint32_t smemBytes, cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(convPipeKernel<COUT, ISS, STACK, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             227 * 1024);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    // Programmatic stream serialization: the kernel's setup may overlap the
    // previous kernel's tail (it waits with griddepcontrol.wait before
    // reading anything that kernel wrote).
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)pipeThreads(ISS, EPI));
    cfg.dynamicSmemBytes = smemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, convPipeKernel<COUT, ISS, STACK, EPI>, inMap, lowMap, wMap, a);
}

}  // namespace

namespace {
uint32_t pipeSmemBytes(int cin, int cout, int lowChannels, int ring, int sw) {
    const uint32_t lowSlot = ((uint32_t)(lowChannels / 8) * kLowPlane + 127u) & ~127u;
    return ringOffset(9u * (uint32_t)cin * (uint32_t)cout * 2u, sw) + (uint32_t)ring * rowBytes(cin, sw) +
           (uint32_t)kLowBufs * lowSlot;
}
}  // namespace

// Planes: the layer routing (convPipeSupported / convPipePreferred) does not
// depend on whether the swizzled slabs fit (a layer falls back to planes).
uint32_t convPipeSmemBytes(int cin, int cout, int lowChannels, int ring) {
    return pipeSmemBytes(cin, cout, lowChannels, ring, 0);
}

namespace {
bool knownCout(int c) { return c == 16 || c == 32 || c == 48 || c == 64 || c == 80 || c == 96 || c == 128; }
// Output-channel slices per layer: the fewest (1, 2, 3, 4, 6) whose slice is
// a supported width and whose weights fit beside a ring of kMinRing rows;
// 0 when none does.
int pickSplits(int cin, int cout, int lowChannels) {
    for (int s : {1, 2, 3, 4, 6})
        if (cout % s == 0 && knownCout(cout / s) &&
            convPipeSmemBytes(cin, cout / s, lowChannels, kMinRing) <= 227u * 1024u)
            return s;
    return 0;
}
}  // namespace

bool convPipeSupported(int cin, int cout, int lowChannels) {
    return cin >= 16 && cin <= 224 && cin % 16 == 0 && lowChannels % 16 == 0 && lowChannels < cin &&
           pickSplits(cin, cout, lowChannels) > 0;
}

bool convPipePreferred(int cin, int cout, int lowChannels) {
    if (!convPipeSupported(cin, cout, lowChannels)) return false;
    const int s = pickSplits(cin, cout, lowChannels);
    return convPipeSmemBytes(cin, cout / s, lowChannels, 4) <= 227u * 1024u;
}

cudaError_t convPipe(const bf16* in, const bf16* low, int lowChannels, int n, int h, int w, int cin,
                     const bf16* weights, bool reverseTaps, const float* bias, int coutTotal, bf16* outB, float* outF,
                     bool relu, bool accumulate, int* errorFlag, cudaStream_t stream, const ConvPipeTest* test,
                     const bf16* upAddend, const ConvHead* head, bool planarOut) {
    if (!low) lowChannels = 0;
    if (n < 1 || h < 1 || w < 1 || !convPipeSupported(cin, coutTotal, lowChannels) || (!outB && !outF && !head) ||
        (head && (!head->out || !head->wt || !head->b || n != 1 || head->h > h || head->w > w)) ||
        !errorFlag || (lowChannels && (h % 2 || w % 2)) ||
        (upAddend && (h % 2 || w % 2 || lowChannels || coutTotal > 64)) || (planarOut && (!outB || outF || head)))
        return cudaErrorNotSupported;
    const int nSplits = pickSplits(cin, coutTotal, lowChannels);
    if (head && (nSplits != 1 || coutTotal > 32)) return cudaErrorNotSupported;  // one pixel's channels in one thread
    const int cout = coutTotal / nSplits;  // output channels per block
    const int cinIn = cin - lowChannels;
    // convPipeReference(): tap-per-tile issue over rows staged as planes, the
    // form the stacked issue and the swizzled slabs are checked against.
    const bool reference = convPipeReference();
    int sw = (test ? test->planes != 0 : reference) ? 0 : rowLayout(cin, lowChannels);
    if (sw && pipeSmemBytes(cin, cout, lowChannels, 4, sw) > 227u * 1024u) sw = 0;  // slabs need a ring of 4 rows
    CUtensorMap inMap{}, lowMap{}, wMap{};
    {
        const uint64_t dims[4] = {(uint64_t)cinIn, (uint64_t)w, (uint64_t)h, (uint64_t)n};
        const uint64_t strides[3] = {(uint64_t)cinIn * 2, (uint64_t)w * cinIn * 2, (uint64_t)h * w * cinIn * 2};
        const uint32_t box[4] = {(uint32_t)(sw ? sw : 8), kHalo, 1, 1};
        if (!makeMap(&inMap, in, 4, dims, strides, box, sw)) return cudaErrorNotSupported;
    }
    if (lowChannels) {
        const uint64_t dims[4] = {(uint64_t)lowChannels, (uint64_t)(w / 2), (uint64_t)(h / 2), (uint64_t)n};
        const uint64_t strides[3] = {(uint64_t)lowChannels * 2, (uint64_t)(w / 2) * lowChannels * 2,
                                     (uint64_t)(h / 2) * (w / 2) * lowChannels * 2};
        const uint32_t box[4] = {8, kLowHalo, 1, 1};
        if (!makeMap(&lowMap, low, 4, dims, strides, box)) return cudaErrorNotSupported;
    } else {
        lowMap = inMap;
    }
    {
        // [9][coutTotal][cin]; a block loads the rows of its slice.
        const uint64_t dims[3] = {(uint64_t)cin, (uint64_t)coutTotal, 9};
        const uint64_t strides[2] = {(uint64_t)cin * 2, (uint64_t)coutTotal * cin * 2};
        const uint32_t box[3] = {8, (uint32_t)cout, 1};
        if (!makeMap(&wMap, weights, 3, dims, strides, box)) return cudaErrorNotSupported;
    }
    PipeArgs a{};
    a.n = n; a.h = h; a.w = w; a.cin = cin; a.cout = cout; a.lowChannels = lowChannels;
    a.coutTotal = coutTotal; a.nSplits = nSplits;
    a.tilesPerRow = (w + kM - 1) / kM;
    a.weightBytes = 9u * (uint32_t)cin * (uint32_t)cout * 2u;
    a.slotBytes = rowBytes(cin, sw);
    a.sw = sw;
    a.lowSlotBytes = ((uint32_t)(lowChannels / 8) * kLowPlane + 127u) & ~127u;
    a.accCols = 32;
    while (a.accCols < (uint32_t)cout) a.accCols <<= 1;
    a.nAcc = test && test->nAcc >= 2 && test->nAcc <= kMaxAcc ? test->nAcc : 2;
    auto tmemColumns = [&](int issuers) {
        uint32_t c = 32;
        while (c < (uint32_t)issuers * (uint32_t)a.nAcc * a.accCols) c <<= 1;
        return c;
    };
    a.tmemCols = tmemColumns(1);
    if (a.tmemCols > 512) return cudaErrorNotSupported;
    a.stats = test ? test->stats : nullptr;
    a.bias = bias; a.outB = outB; a.outF = outF; a.upAdd = upAddend;
    a.outPixels = planarOut ? (long long)n * h * w : 0;
    a.upPixels = (long long)n * (h / 2) * (w / 2);
    if (head) a.head = *head;
    a.relu = relu ? 1 : 0; a.accumulate = accumulate ? 1 : 0; a.reverseTaps = reverseTaps ? 1 : 0;
    a.errorFlag = errorFlag;
    a.waitLimitNs = test && test->waitLimitNs ? test->waitLimitNs : 1000000000ull;
    a.probe = test && test->probe ? 1 : 0;
    // Blocks per SM from shared and tensor memory at a ring of 4 rows (3
    // where 4 do not fit); then the largest ring (up to kMaxRing rows) that
    // keeps that many blocks per SM. Where one block fits per SM (one MMA
    // issuer per SM issues at about half the tensor pipe's rate), the block
    // runs two issuers on the same ring.
    const int sms = deviceSmCount();
    const uint32_t smemPerSm = 228u * 1024u, smemMax = 227u * 1024u;
    a.ring = pipeSmemBytes(cin, cout, lowChannels, 4, sw) <= smemMax ? 4 : kMinRing;
    int perSm = (int)(smemPerSm / (pipeSmemBytes(cin, cout, lowChannels, a.ring, sw) + 1024u));
    perSm = std::max(1, std::min({perSm, (int)(512u / a.tmemCols), 2048 / kPipeThreads}));
    if (test && test->blocksPerSm > 0 && test->blocksPerSm < perSm) perSm = test->blocksPerSm;
    const int force = test ? test->issuers : 0;  // 1 or 2 issuers
    const bool twoFit = tmemColumns(2) <= 512u && 2 * a.nAcc <= kMaxAcc;
    if (force == 2 && !twoFit) return cudaErrorNotSupported;
    // The stacked-row form (Cout 32 or 64 per block, no concatenated input):
    // one issuer, a ring of at least 4 accumulator blocks of cout columns.
    const int stackMode = test ? test->stacked : (reference ? 1 : 0);
    const bool stackFits = !lowChannels && (cout == 32 || cout == 64) && cin <= 128 && force != 2;
    // Measured per layer: the stacked form is faster for unsplit 32-channel
    // layers (1080p 16 -> 32: 78.6 -> 74.2 us, 32 -> 32: 98.9 -> 94.0), slower
    // for 64 output channels (64 -> 64 at 480x272: 31.4 -> 36.9) and for a
    // 32-channel slice of a split layer (128 -> 128 at 120x68: 19.2 -> 23.0), and
    // where one block fits per SM: there two issuers of the tap-per-tile form
    // issue faster than the stacked form's one (1080p 80 -> 32: 165 us against
    // 228; with two blocks, 48 -> 32 at 960x544, 36 against 35).
    const bool stackDefault = cout == 32 && nSplits == 1 && perSm > 1;
    if (stackMode == 2 && !stackFits) return cudaErrorNotSupported;
    const bool stacked = stackFits && (stackMode == 2 || (stackMode == 0 && stackDefault));
    const int issuers = !stacked && (force == 2 || (force == 0 && perSm == 1 && twoFit)) ? 2 : 1;
    a.tmemCols = tmemColumns(issuers);
    if (stacked) {
        auto colsFor = [](int per) {  // tensor-memory columns of a block at per blocks per SM
            uint32_t c = 512;
            while (c * (uint32_t)per > 512u) c >>= 1;
            return c;
        };
        while (perSm > 1 && colsFor(perSm) < 4u * (uint32_t)cout) perSm--;
        const uint32_t cols = colsFor(perSm);
        int nb = std::min<int>(kMaxAcc, (int)(cols / (uint32_t)cout));
        if (test && test->nAcc >= 3 && test->nAcc <= kMaxAcc && (uint32_t)test->nAcc * cout <= cols) nb = test->nAcc;
        a.nAcc = nb;
        a.accCols = (uint32_t)cout;
        a.tmemCols = 32;
        while (a.tmemCols < (uint32_t)(nb * cout)) a.tmemCols <<= 1;
    }
    while (a.ring < kMaxRing &&
           (uint32_t)perSm * (pipeSmemBytes(cin, cout, lowChannels, a.ring + 1, sw) + 1024u) <= smemPerSm &&
           pipeSmemBytes(cin, cout, lowChannels, a.ring + 1, sw) <= smemMax)
        a.ring++;
    if (test && test->ring >= kMinRing && test->ring <= kMaxRing) a.ring = test->ring;
    const uint32_t smemBytes = pipeSmemBytes(cin, cout, lowChannels, a.ring, sw);
    if (smemBytes > smemMax) return cudaErrorNotSupported;
    // Strips: balanced over the blocks (balancedStripRows); units that do
    // not divide evenly leave a last round on part of the GPU, strips too
    // long leave blocks idle. Every slice of output channels walks all units.
    const long long columns = (long long)n * a.tilesPerRow;
    const long long blocks = std::max<long long>(nSplits, (long long)sms * perSm / nSplits * nSplits);
    a.stripRows = balancedStripRows(columns * nSplits, h, blocks);
    if (test && test->stripRows > 0) a.stripRows = test->stripRows;
    a.strips = (h + a.stripRows - 1) / a.stripRows;
    a.units = (int)(columns * a.strips);
    const int grid = (int)std::min<long long>((long long)a.units * nSplits, blocks);
    // Eight epilogue warps where one block per SM drains wide accumulators
    // (two issuers, 96 or 128 columns); the fused head needs a pixel's
    // channels in one thread.
    const bool wideEpilogue = issuers == 2 && cout >= 96 && !head && !(test && test->epilogueWarps == 4);
    switch (cout) {
        case 16: return issuers == 2 ? launchPipe<16, 2>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                             : launchPipe<16, 1>(inMap, lowMap, wMap, a, grid, smemBytes, stream);
        case 32: return stacked ? launchPipe<32, 1, true>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                       : issuers == 2 ? launchPipe<32, 2>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                             : launchPipe<32, 1>(inMap, lowMap, wMap, a, grid, smemBytes, stream);
        case 48: return issuers == 2 ? launchPipe<48, 2>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                             : launchPipe<48, 1>(inMap, lowMap, wMap, a, grid, smemBytes, stream);
        case 64: return stacked ? launchPipe<64, 1, true>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                       : issuers == 2 ? launchPipe<64, 2>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                             : launchPipe<64, 1>(inMap, lowMap, wMap, a, grid, smemBytes, stream);
        case 80: return issuers == 2 ? launchPipe<80, 2>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                             : launchPipe<80, 1>(inMap, lowMap, wMap, a, grid, smemBytes, stream);
        case 96: return issuers == 2 ? (wideEpilogue ? launchPipe<96, 2, false, 8>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                                             : launchPipe<96, 2>(inMap, lowMap, wMap, a, grid, smemBytes, stream))
                             : launchPipe<96, 1>(inMap, lowMap, wMap, a, grid, smemBytes, stream);
        case 128: return issuers == 2 ? (wideEpilogue ? launchPipe<128, 2, false, 8>(inMap, lowMap, wMap, a, grid, smemBytes, stream)
                                              : launchPipe<128, 2>(inMap, lowMap, wMap, a, grid, smemBytes, stream))
                              : launchPipe<128, 1>(inMap, lowMap, wMap, a, grid, smemBytes, stream);
        default: return cudaErrorNotSupported;
    }
}

int convPipeWaitProbe() {
    // A 128 x 4 image of 16 channels, zero input and weights: the output is
    // ReLU(bias). First launch: the issuer waits on a barrier nothing
    // completes, with a 2 ms limit; the block must give up, report and free
    // its tensor memory. Second launch: the normal path on the same buffers.
    const int n = 1, h = 4, w = 128, cin = 16, cout = 32;
    bf16 *in = nullptr, *weights = nullptr, *out = nullptr;
    float* bias = nullptr;
    int* flag = nullptr;
    int ok = 0;
    std::vector<float> hostBias(cout);
    for (int c = 0; c < cout; c++) hostBias[c] = (float)(c % 7) - 2.5f;
    std::vector<bf16> hostOut((size_t)n * h * w * cout);
    int hostFlag = -1;
    cudaError_t e = cudaMalloc(&in, sizeof(bf16) * n * h * w * cin);
    if (e == cudaSuccess) e = cudaMalloc(&weights, sizeof(bf16) * 9 * cin * cout);
    if (e == cudaSuccess) e = cudaMalloc(&out, sizeof(bf16) * hostOut.size());
    if (e == cudaSuccess) e = cudaMalloc(&bias, sizeof(float) * cout);
    if (e == cudaSuccess) e = cudaMalloc(&flag, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(in, 0, sizeof(bf16) * n * h * w * cin);
    if (e == cudaSuccess) e = cudaMemset(weights, 0, sizeof(bf16) * 9 * cin * cout);
    if (e == cudaSuccess) e = cudaMemset(out, 0, sizeof(bf16) * hostOut.size());
    if (e == cudaSuccess) e = cudaMemset(flag, 0, sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpy(bias, hostBias.data(), sizeof(float) * cout, cudaMemcpyHostToDevice);
    ConvPipeTest probe{2000000ull, 1, 0, 0};
    if (e == cudaSuccess)
        e = convPipe(in, nullptr, 0, n, h, w, cin, weights, false, bias, cout, out, nullptr, true, false, flag, 0, &probe);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(&hostFlag, flag, sizeof(int), cudaMemcpyDeviceToHost);
    const bool reported = e == cudaSuccess && hostFlag == 1;
    if (e == cudaSuccess) e = cudaMemset(flag, 0, sizeof(int));
    if (e == cudaSuccess)
        e = convPipe(in, nullptr, 0, n, h, w, cin, weights, false, bias, cout, out, nullptr, true, false, flag, 0);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(&hostFlag, flag, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(hostOut.data(), out, sizeof(bf16) * hostOut.size(), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && reported && hostFlag == 0) {
        ok = 1;
        for (size_t i = 0; i < hostOut.size() && ok; i++)
            if (__bfloat162float(hostOut[i]) != fmaxf(hostBias[i % cout], 0.0f)) ok = 0;
    }
    cudaFree(in); cudaFree(weights); cudaFree(out); cudaFree(bias); cudaFree(flag);
    return e == cudaSuccess ? ok : 0;
}

}  // namespace rt
