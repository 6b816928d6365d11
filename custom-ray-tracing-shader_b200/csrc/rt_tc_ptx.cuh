// mbarrier, TMA and tcgen05 wrappers shared by the tensor-core kernels
// (sm_100a). TMA loads are never multicast; every wait is bounded.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <mutex>

#include "rt_conv_tc.cuh"

namespace rt {
namespace {

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
// Bounded wait for the phase of parity `parity` to complete. Gives up when
// the block's abort flag is set or when limitNs pass (then sets the flag).
__device__ __forceinline__ bool waitPhase(uint32_t bar, uint32_t parity, volatile int* abortFlag, uint64_t limitNs) {
    if (barTryWait(bar, parity)) return true;
    const uint64_t deadline = nowNs() + limitNs;
    for (;;) {
        if (barTryWait(bar, parity)) return true;
        if (*abortFlag) return false;
        if (nowNs() > deadline) { *abortFlag = 1; return false; }
    }
}
// The same for a whole warp: lane 0 waits and every lane gets its verdict.
__device__ __forceinline__ bool waitPhaseWarp(uint32_t bar, uint32_t parity, volatile int* abortFlag,
                                              uint64_t limitNs) {
    bool ok = true;
    if ((threadIdx.x & 31) == 0) ok = waitPhase(bar, parity, abortFlag, limitNs);
    return __shfl_sync(0xFFFFFFFFu, ok ? 1 : 0, 0) != 0;
}
// Bounded poll that ignores the abort flag (the drains on the abort path).
__device__ __forceinline__ void pollPhase(uint32_t bar, uint32_t parity, uint64_t limitNs) {
    const uint64_t deadline = nowNs() + limitNs;
    while (!barTryWait(bar, parity) && nowNs() < deadline) {
    }
}
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
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

inline PFN_cuTensorMapEncodeTiled_v12000 encodeTiled() {
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

// The swizzle whose span is a pixel row of `slab` channels (2 bytes each),
// and its layout type in bits 61-63 of a shared-memory matrix descriptor.
inline CUtensorMapSwizzle slabSwizzle(int slab) {
    return slab == 16 ? CU_TENSOR_MAP_SWIZZLE_32B : slab == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
}
__host__ __device__ constexpr uint64_t slabLayout(int slab) {
    return (uint64_t)(slab == 16 ? 6 : slab == 32 ? 4 : 2) << 61;
}
// The widest slab of 16, 32 or 64 channels dividing c.
inline int slabChannels(int c) { return c % 64 == 0 ? 64 : c % 32 == 0 ? 32 : 16; }

}  // namespace
}  // namespace rt
