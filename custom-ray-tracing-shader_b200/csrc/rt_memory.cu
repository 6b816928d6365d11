// Device memory of the library: cudaMalloc with a bounded cache of freed
// blocks (see rt_common.cuh).
//
// A scene load makes about 70 allocations and frees, a ray query or gradient
// call a handful; each cudaMalloc, cudaFree or cudaMallocHost costs 10 us to
// several hundred and cudaFree waits for the device every time. No work uses a
// block that is freed here (deviceFree), so handing it out again waits for
// nothing: waiting for the whole device would also fail, and break the capture,
// while another thread records a CUDA graph. Measured:
// loading 8,000 triangles took 20 ms of which the kernels 2, the million-
// triangle scene 54 ms of which upload and kernels 21.
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <list>
#include <mutex>
#include <unordered_map>

#include "rt_common.cuh"

namespace rt {
namespace {

// Bytes of freed blocks kept per device; the oldest go first. It covers what
// loads of a million triangles and their first full-HD frames free (about 1.5 GB
// each, in blocks of up to 300 MB that find their next use within a quarter of
// their size; with 2 GB kept a session's repeated loads took as long, a new
// session's first 21.5 ms against 18.7) and is 2% of the device's memory. Of the
// path buffers of a 16-path full-HD pass (20 blocks of 256 MB, freed after the
// scene's) as many stay as fit: giving them all back at once cost the next
// session's first such pass 3 to 390 ms, as the driver hands out new memory. A
// block of more than a quarter of the bound goes back at once.
constexpr size_t kCacheBytes = 4ull << 30;

// Blocks belong to the CUDA context they were allocated in. cudaDeviceReset
// (by a host with a runtime of its own) ends it with all its memory while
// sessions may still exist, so a block carries its context's number, which is
// never used again.
struct Block { void* p; size_t bytes; unsigned long long context; };
struct DeviceCache {
    std::list<Block> ready;  // oldest first
    size_t bytes = 0;
};
struct Owned { int device; size_t bytes; unsigned long long context; };

std::mutex g_lock;
std::unordered_map<int, DeviceCache>& caches() { static auto* m = new std::unordered_map<int, DeviceCache>; return *m; }
std::unordered_map<void*, Owned>& owned() { static auto* m = new std::unordered_map<void*, Owned>; return *m; }
int g_users = 0;

// Countdown of RtxDebugFailAllocation: when it reaches the call that brings
// it from 1 to 0, that allocation fails without calling cudaMalloc.
std::atomic<long long> g_failAllocationIn{0};

// Sizes in steps, so that blocks of similar requests are interchangeable.
size_t stepped(size_t bytes) {
    const size_t step = bytes < (2u << 20) ? 512 : 2u << 20;
    return (bytes + step - 1) / step * step;
}

// The number of the current device's context (made if need be); 0 where the
// driver does not say.
unsigned long long contextNumber() {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent getCurrent = nullptr;
    static GetId getId = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *a = nullptr, *b = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess &&
            cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess) {
            getCurrent = reinterpret_cast<GetCurrent>(a);
            getId = reinterpret_cast<GetId>(b);
        }
    });
    CUcontext context = nullptr;
    unsigned long long id = 0;
    if (!getCurrent || cudaFree(nullptr) != cudaSuccess || getCurrent(&context) != CUDA_SUCCESS || !context ||
        getId(context, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}
// With g_lock held: forgets the blocks of contexts that are gone.
void forget(DeviceCache& c, unsigned long long context) {
    for (auto it = c.ready.begin(); it != c.ready.end();) {
        if (it->context == context) { ++it; continue; }
        c.bytes -= it->bytes;
        it = c.ready.erase(it);
    }
}
// With g_lock held.
void evict(int device, DeviceCache& c, size_t keep) {
    if (c.bytes <= keep) return;
    int current = 0;
    const bool away = cudaGetDevice(&current) == cudaSuccess && current != device;
    if (away) cudaSetDevice(device);
    forget(c, contextNumber());
    if (away) cudaSetDevice(current);
    while (c.bytes > keep && !c.ready.empty()) {
        cudaFree(c.ready.front().p);
        c.bytes -= c.ready.front().bytes;
        c.ready.pop_front();
    }
}

}  // namespace

void setFailAllocation(int n) { g_failAllocationIn.store(n); }

cudaError_t deviceAllocBytes(void** p, size_t bytes) {
    *p = nullptr;
    long long n = g_failAllocationIn.load();
    while (n > 0 && !g_failAllocationIn.compare_exchange_weak(n, n - 1)) {
    }
    if (n == 1) return cudaErrorMemoryAllocation;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const size_t want = stepped(bytes ? bytes : 1);
    const unsigned long long context = contextNumber();
    std::lock_guard<std::mutex> guard(g_lock);
    DeviceCache& c = caches()[device];
    forget(c, context);
    // The smallest block that fits without wasting more than a quarter.
    auto fits = [&](const Block& b) { return b.bytes >= want && b.bytes - want <= (want / 4 > 65536 ? want / 4 : 65536); };
    auto best = c.ready.end();
    for (auto it = c.ready.begin(); it != c.ready.end(); ++it)
        if (fits(*it) && (best == c.ready.end() || it->bytes < best->bytes)) best = it;
    if (best != c.ready.end()) {
        *p = best->p;
        owned()[best->p] = Owned{device, best->bytes, context};
        c.bytes -= best->bytes;
        c.ready.erase(best);
        return cudaSuccess;
    }
    e = cudaMalloc(p, want);
    if (e == cudaErrorMemoryAllocation && c.bytes) {
        cudaGetLastError();
        evict(device, c, 0);
        e = cudaMalloc(p, want);
    }
    if (e != cudaSuccess) { *p = nullptr; return e; }
    owned()[*p] = Owned{device, want, context};
    return cudaSuccess;
}

void deviceFree(void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> guard(g_lock);
    auto it = owned().find(p);
    if (it == owned().end()) { cudaFree(p); return; }
    const Owned o = it->second;
    owned().erase(it);
    if (g_users == 0 || o.bytes > kCacheBytes / 4) { cudaFree(p); return; }
    DeviceCache& c = caches()[o.device];
    c.ready.push_back(Block{p, o.bytes, o.context});
    c.bytes += o.bytes;
    evict(o.device, c, kCacheBytes);
}

void trimDeviceMemory() {
    std::lock_guard<std::mutex> guard(g_lock);
    for (auto& entry : caches()) evict(entry.first, entry.second, 0);
}

DeviceMemoryUser::DeviceMemoryUser() {
    std::lock_guard<std::mutex> guard(g_lock);
    g_users++;
}
DeviceMemoryUser::~DeviceMemoryUser() {
    {
        std::lock_guard<std::mutex> guard(g_lock);
        if (--g_users > 0) return;
    }
    trimDeviceMemory();
}

}  // namespace rt
