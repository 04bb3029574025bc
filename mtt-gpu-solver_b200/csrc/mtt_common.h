// mtt_common.h — host-side status handling shared by the C ABI sources.
#pragma once
#include <cuda_runtime.h>
#include "../../include/mtt_b200.h"

namespace mtt {

// cudaError_t of the last failing CUDA call made by this host thread.
extern thread_local int g_last_cuda_error;

inline int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return MTT_OK;
    g_last_cuda_error = (int)e;
    return e == cudaErrorMemoryAllocation ? MTT_ERR_NOMEM : MTT_ERR_CUDA;
}

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Scratch of one call, allocated and freed in stream order (cudaFreeAsync).
// It comes from a library-owned pool per device that keeps up to
// SCRATCH_KEEP bytes between calls (mtt_trim_pool gives them back): the
// device's default pool returns its memory to the driver at the next
// synchronisation, and mapping it again cost 0.4 ms to several ms a call.
// While the stream is being captured the allocation is a plain graph node.
// The largest scratch of one call at the sizes in use is 239 MB (the flop
// matrices of 21 flops with all 1,326 combos); the flop-EV chain takes 134 MB.
constexpr size_t SCRATCH_KEEP = 256ull << 20;
int scratch_alloc(void** p, size_t bytes, cudaStream_t st);
template <typename T>
inline int scratch_alloc(T** p, size_t count, cudaStream_t st) {
    return scratch_alloc(reinterpret_cast<void**>(p), (count ? count : 1) * sizeof(T), st);
}
unsigned long long current_context_id();
int scratch_trim();   // returns what the current device's scratch pool keeps; the caller has synchronised

// Raises a kernel's limit on dynamic shared memory, where `need` is above the
// default (48 KB with the kernel's static part, at most 2.4 KB here), to 224 KB.
// Always to the same value: a limit set to one batch's need could be lowered by
// another thread's batch between this one's call and its launches, which then
// failed as invalid.  One call a kernel, and none for small needs: asking for
// the kernel's attributes first cost a solve 70 us.
constexpr size_t SMEM_FREE = 45 * 1024, SMEM_MOST = 224 * 1024;
template <typename... Args>
inline int allow_smem(void (*kernel)(Args...), size_t need) {
    if (need <= SMEM_FREE) return MTT_OK;
    return cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)(need > SMEM_MOST ? need : SMEM_MOST)));
}

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
inline long long ceil_div_ll(long long a, long long b) { return (a + b - 1) / b; }

}  // namespace mtt

#define MTT_TRY_CUDA(call)                                            \
    do {                                                              \
        int _mtt_s = ::mtt::cuda_status(call);                        \
        if (_mtt_s != MTT_OK) return _mtt_s;                          \
    } while (0)

#define MTT_TRY(call)                                                 \
    do {                                                              \
        int _mtt_s = (call);                                          \
        if (_mtt_s != MTT_OK) return _mtt_s;                          \
    } while (0)

// A launch's own error (bad configuration) surfaces right away.
#define MTT_CHECK_LAUNCH() MTT_TRY_CUDA(cudaGetLastError())
