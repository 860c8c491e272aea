// Shared definitions of the PyHeartSim B200 kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace phs {

constexpr int kThreads = 256;              // threads per CTA of the step kernel
constexpr int kWarps = kThreads / 32;
constexpr int kMaxRestart = 50;            // GMRES(m) restart bound (reference uses m = 50)
constexpr int kSlots = kMaxRestart + 2;    // FP64 partial sums per tile
constexpr int kPadVoxels = 1024;           // per-voxel engine arrays are padded to a multiple of this

// Record a CUDA error message (host side); defined in phs_capi.cu.
void set_last_error(const char* where, cudaError_t e);
// Record a plain error message for phs_last_error().
void set_last_message(const char* msg);

// Device memory from the library's pool of the current device, ordered on
// `stream` (phs_pool.cu); dev_free accepts null.  Memory allocated or filled on
// one stream is used on another only after a synchronisation or an event wait.
cudaError_t dev_alloc(void** p, size_t bytes, cudaStream_t stream);
void dev_free(void* p, cudaStream_t stream);
// The opt-in of kernel `fn` to `bytes` of dynamic shared memory, which holds per
// context: made once in each (so a call under capture that follows one outside
// makes no such call).
cudaError_t allow_dynamic_smem(const void* fn, size_t bytes);
// Sets how much the pool keeps; `engines`: engines made (+1) or destroyed (-1).
void pool_update(int engines);

}  // namespace phs

#define PHS_CUDA_TRY(expr)                                   \
    do {                                                     \
        cudaError_t _e = (expr);                             \
        if (_e != cudaSuccess) {                             \
            ::phs::set_last_error(#expr, _e);                \
            return _e == cudaErrorMemoryAllocation ? PHS_ERR_OOM : PHS_ERR_CUDA; \
        }                                                    \
    } while (0)
