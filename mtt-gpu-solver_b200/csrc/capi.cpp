// capi.cpp — status strings, version and the per-thread CUDA error slot.
#include <cuda.h>   // CUcontext / CUresult types only: the driver entry points are resolved at run time

#include <mutex>
#include <vector>

#include "mtt_common.h"

namespace mtt {
thread_local int g_last_cuda_error = 0;

// Unique id of the calling thread's current context (0 if none or if the
// driver does not offer the query).  Ids are never reused within a process,
// so a context created after a cudaDeviceReset always has a new one.  The two
// driver functions are resolved at run time, so the library does not link the
// driver and still loads on machines without one.
unsigned long long current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(f);
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(f);
    });
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (get_current && get_id && get_current(&c) == CUDA_SUCCESS && c && get_id(c, &id) == CUDA_SUCCESS) return id;
    return 0;
}

namespace {
// Scratch pools by device and context (a cudaDeviceReset replaces the context
// and ends its pools).  A context without an id, or one past the table's
// limit, has none and allocates from the device's default pool.
struct ScratchPool {
    int dev;
    unsigned long long ctx;
    cudaMemPool_t pool;
};
std::mutex g_scratch_mu;

cudaMemPool_t scratch_pool(bool create) {
    static std::vector<ScratchPool> pools;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    unsigned long long ctx = current_context_id();
    for (const ScratchPool& e : pools)
        if (ctx && e.dev == dev && e.ctx == ctx) return e.pool;
    if (!create || pools.size() >= 64) return nullptr;
    // another thread may be capturing a graph, which creating a pool must not end
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p = nullptr;
    cudaError_t e = cudaFree(nullptr);   // makes the device's context current
    if (e == cudaSuccess) e = cudaMemPoolCreate(&p, &props);
    if (e == cudaSuccess) {
        uint64_t keep = SCRATCH_KEEP;
        e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    ctx = current_context_id();
    if (e != cudaSuccess || !ctx) {
        cudaGetLastError();
        if (p) cudaMemPoolDestroy(p);
        return nullptr;
    }
    pools.push_back({dev, ctx, p});
    return p;
}
}  // namespace

int scratch_alloc(void** p, size_t bytes, cudaStream_t st) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    MTT_TRY_CUDA(cudaStreamIsCapturing(st, &cap));
    cudaMemPool_t pool = cap == cudaStreamCaptureStatusNone ? scratch_pool(true) : nullptr;
    return cuda_status(pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaMallocAsync(p, bytes, st));
}

int scratch_trim() {
    cudaMemPool_t pool = scratch_pool(false);
    return pool ? cuda_status(cudaMemPoolTrimTo(pool, 0)) : MTT_OK;
}
}  // namespace mtt

extern "C" const char* mtt_status_string(int status) {
    switch (status) {
        case MTT_OK: return "ok";
        case MTT_ERR_INVALID: return "invalid argument";
        case MTT_ERR_CUDA: return "CUDA error";
        case MTT_ERR_NOMEM: return "out of memory";
        case MTT_ERR_TIMEOUT: return "bounded device wait timed out";
        case MTT_ERR_IO: return "file missing, short or malformed";
        case MTT_ERR_UNSUPPORTED: return "unsupported size or feature";
        default: return "unknown status";
    }
}

extern "C" int mtt_last_cuda_error(void) { return mtt::g_last_cuda_error; }

extern "C" const char* mtt_version(void) { return "mtt-b200 0.1.0 (sm_100a)"; }
