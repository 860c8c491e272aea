// Device memory of the library: one stream-ordered pool per device and context.
//
// cudaMalloc and cudaFree cost 0.05-0.2 ms each here and cudaFree now and then
// much more (an engine of 24 instances, ~30 arrays each, took 170-300 ms to
// fill and 210-1100 ms to empty, against 130 ms for 300 steps of it), and the
// default stream-ordered pool gives everything back at the next
// synchronisation, so a contraction that allocates its partial sums paid 4-5 ms
// per call for 1.5 ms of kernels.  This pool keeps a bounded amount instead:
// what is allocated plus kKeepEngine bytes while an engine of the device is
// alive, plus kKeepIdle bytes otherwise; the driver takes the rest back at the
// next synchronisation, which the calls that remove an instance or destroy an
// engine make at their end, so other allocators find it when they return.
//
// The pool is the library's own, so the device's default pool keeps the
// caller's settings.  It is found by device and context (a program may have
// several contexts on a device; a device reset makes a new one, and ids are not
// used again).  A stream that is being captured allocates
// from the default pool as any cudaMallocAsync does: the graph owns that
// memory.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <map>
#include <mutex>
#include <set>
#include <utility>

#include "../../include/phs.h"
#include "phs_common.cuh"

namespace phs {
namespace {

constexpr unsigned long long kKeepEngine = 4ull << 30;
constexpr unsigned long long kKeepIdle = 512ull << 20;

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    int engines = 0;
};
std::mutex g_pool_mu;
std::map<std::pair<int, unsigned long long>, DevicePool> g_pool;   // by device and context

bool context_id(unsigned long long* id) {
    static PFN_cuCtxGetId_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, []() {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuCtxGetId_v12000)p;
    });
    return fn != nullptr && fn(nullptr, id) == CUDA_SUCCESS;
}

// Bytes to hold on to from now on (g_pool_mu held).
void set_threshold(DevicePool& d) {
    unsigned long long used = 0;
    if (cudaMemPoolGetAttribute(d.pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) return;
    unsigned long long keep = used + (d.engines > 0 ? kKeepEngine : kKeepIdle);
    cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
}

// While it lives, this thread's calls neither fail for nor disturb a stream
// capture that another thread has under way.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The current device's pool, made on first use; nullptr when there is none to
// be had (the default pool serves then).  g_pool_mu held.
DevicePool* current_pool() {
    RelaxedCapture relaxed;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    if (cudaFree(nullptr) != cudaSuccess) return nullptr;   // the context exists from here on
    unsigned long long ctx = 0;
    if (!context_id(&ctx)) return nullptr;
    const auto it = g_pool.find({dev, ctx});
    if (it != g_pool.end()) return &it->second;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    DevicePool& d = g_pool[{dev, ctx}];
    d.pool = pool;
    set_threshold(d);
    return &d;
}

}  // namespace

cudaError_t dev_alloc(void** p, size_t bytes, cudaStream_t stream) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (stream != nullptr) {
        const cudaError_t e = cudaStreamIsCapturing(stream, &cap);
        if (e != cudaSuccess) return e;
    }
    cudaMemPool_t pool = nullptr;
    if (cap == cudaStreamCaptureStatusNone) {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        if (DevicePool* d = current_pool()) pool = d->pool;
    }
    const cudaError_t e = pool ? cudaMallocFromPoolAsync(p, bytes, pool, stream) : cudaMallocAsync(p, bytes, stream);
    // the caller reports it; the check after a later call's launches must not find it
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();
    return e;
}

void dev_free(void* p, cudaStream_t stream) {
    if (p) cudaFreeAsync(p, stream);
}

cudaError_t allow_dynamic_smem(const void* fn, size_t bytes) {
    static std::mutex mu;
    static std::set<std::pair<unsigned long long, const void*>> done;
    unsigned long long ctx = 0;
    std::lock_guard<std::mutex> lk(mu);
    const bool known = context_id(&ctx);
    if (known && done.count({ctx, fn})) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && known) done.insert({ctx, fn});
    return e;
}

void pool_update(int engines) {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    DevicePool* d = current_pool();
    if (!d) return;
    d->engines += engines;
    if (d->engines < 0) d->engines = 0;   // an engine made before a device reset
    set_threshold(*d);
}

}  // namespace phs
