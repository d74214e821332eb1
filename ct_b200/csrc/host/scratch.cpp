// Device memory that one operator call takes and gives back on its stream (view
// tables, the projector's volume copy, repacked rows): a stream-ordered pool per
// device that keeps up to kKeep bytes between calls. The device's default pool
// returns everything at each synchronisation, so that a program that waits for
// every call paid for mapping memory again each time (120 views of 200 x 150 into
// 96^3, filter and backprojection, each call waited for: 4.8 ms, with this pool 0.18
// ms; the smallest scan, 24 views of 32 x 20, 0.51 and 0.058 ms). The pool is the
// library's own: no setting of the default pool changes for the rest of the
// process. What it keeps idle is in nobody's way inside the process: the driver takes it
// for any allocation that is short (192 MB kept, 48 MB free: a cudaMalloc of 64 MB, and one of
// 100 MB more than is free by another allocator, succeed). For other processes, and
// for programs that plan by cudaMemGetInfo, ctb_release_scratch gives it back.

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <mutex>
#include <type_traits>

#include "../ctb_internal.h"

namespace ctb {

namespace {
// the driver's functions that the runtime has no counterpart of, null when not found
struct Driver {
    CUresult (*get_current)(CUcontext*) = nullptr;
    CUresult (*get_id)(CUcontext, unsigned long long*) = nullptr;
    CUresult (*primary_state)(CUdevice, unsigned*, int*) = nullptr;
    CUresult (*primary_retain)(CUcontext*, CUdevice) = nullptr;
    CUresult (*primary_release)(CUdevice) = nullptr;
};
const Driver& driver() {
    static Driver d;
    static std::once_flag once;
    std::call_once(once, [] {
        auto entry = [](const char* name, auto* fn) {
            void* p = nullptr;
            cudaDriverEntryPointQueryResult q;
            if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess &&
                q == cudaDriverEntryPointSuccess)
                *fn = reinterpret_cast<std::remove_pointer_t<decltype(fn)>>(p);
            else
                cudaGetLastError();
        };
        entry("cuCtxGetCurrent", &d.get_current);
        entry("cuCtxGetId", &d.get_id);
        entry("cuDevicePrimaryCtxGetState", &d.primary_state);
        entry("cuDevicePrimaryCtxRetain", &d.primary_retain);
        entry("cuDevicePrimaryCtxRelease", &d.primary_release);
    });
    return d;
}

// Whether the current context is the device's primary one (the one the CUDA runtime uses).
bool primary_context_current(int dev) {
    const Driver& d = driver();
    CUcontext cur = nullptr, primary = nullptr;
    unsigned flags = 0;
    int active = 0;
    if (!d.get_current || !d.primary_state || !d.primary_retain || !d.primary_release) return false;
    if (d.get_current(&cur) != CUDA_SUCCESS || d.primary_state(dev, &flags, &active) != CUDA_SUCCESS || !active)
        return false;
    if (d.primary_retain(&primary, dev) != CUDA_SUCCESS) return false;
    d.primary_release(dev);
    return cur == primary;
}
}  // namespace

unsigned long long current_context_id() {
    const Driver& d = driver();
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (!d.get_current || !d.get_id || d.get_current(&c) != CUDA_SUCCESS || !c || d.get_id(c, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

namespace {

constexpr uint64_t kKeep = uint64_t(256) << 20;

struct Pool {
    cudaMemPool_t pool = nullptr;
    unsigned long long ctx = 0;   // the context the pool belongs to
};
std::mutex g_pool_mtx;
std::map<int, Pool> g_pools;

// The current device's pool (null: none to be had, a capturing stream, whose
// allocations belong to its graph, or a context beside the device's primary one,
// where the device's default pool serves: a device has one pool of this library,
// however many contexts a program switches between).
cudaMemPool_t scratch_pool(cudaStream_t s) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return nullptr;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    const unsigned long long ctx = current_context_id();
    if (ctx == 0) return nullptr;
    std::lock_guard<std::mutex> lk(g_pool_mtx);
    Pool& p = g_pools[dev];
    if (p.pool && p.ctx == ctx) return p.pool;
    if (!primary_context_current(dev)) return nullptr;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    uint64_t keep = kKeep;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) cudaGetLastError();
    p.pool = pool;   // (the pool of a primary context that was reset went with it)
    p.ctx = ctx;
    return pool;
}

}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
    cudaMemPool_t pool = scratch_pool(s);
    if (!pool) return cudaMallocAsync(p, bytes, s);
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, s);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        scratch_trim();
        e = cudaMallocFromPoolAsync(p, bytes, pool, s);
    }
    return e;
}

void scratch_trim() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    const unsigned long long ctx = current_context_id();
    std::lock_guard<std::mutex> lk(g_pool_mtx);
    auto it = g_pools.find(dev);
    if (it == g_pools.end() || !it->second.pool || it->second.ctx != ctx) return;
    if (cudaMemPoolTrimTo(it->second.pool, 0) != cudaSuccess) cudaGetLastError();
}

cudaError_t device_alloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        scratch_trim();
        e = cudaMalloc(p, bytes);
    }
    return e;
}

}  // namespace ctb
