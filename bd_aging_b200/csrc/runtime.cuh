// runtime.cuh -- host-side plumbing shared by the translation units of
// libbd_aging_b200: status mapping, per-call workspaces, launch checks.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>

#include "../../include/bd_aging.h"
#include "common.cuh"

namespace bd {

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// Identifier of the CUDA context current on the calling thread (initialising
// the current device's primary context if needed).  Context ids are unique
// for the life of the process, so a device reset, which destroys the primary
// context and every address in it, changes the id.  0 when none can be had.
unsigned long long current_context_id();

// What a synchronous mirror call needs on its device, one slot per call in
// flight: a status word and a result in host memory that the kernels write to
// directly (no clear before and no copy after them; the stream's
// synchronisation is all the call waits for), and the FP64 partial sums of the
// fixed-order reductions.  The slots are allocated on first use in each
// context (again after a device reset) and kept until exit.
constexpr int kWorkAccum = 2048;  // FP64 slots: one per reduction block
struct HostWords {
    unsigned status;  // kStat* bits
    double value;
};
struct CallSlot {
    HostWords *host = nullptr;     // host address
    HostWords *dev = nullptr;      // the same words as kernels see them
    double *accum = nullptr;       // kWorkAccum FP64 partial sums
    unsigned *counter = nullptr;   // finished blocks of a reduction, zero between calls
    CallStatus *status = nullptr;  // for the kernels, on the device
    void *state = nullptr;
    cudaStream_t stream;           // of the call's kernels
    bool waited = false;
    explicit CallSlot(cudaStream_t s);  // takes a free slot of the current context (waits when all are taken)
    ~CallSlot();                   // gives it back, after the call's kernels also where the call failed
    cudaError_t wait();            // for the call's kernels
    CallSlot(const CallSlot &) = delete;
    CallSlot &operator=(const CallSlot &) = delete;
    bool ok() const { return host != nullptr; }  // false: allocation failed
};

// Map the device status word to a BD_* code.  A non-finite position also
// piles particles into one cell, so it is reported before the overflow.
inline int status_from_bits(unsigned bits) {
    if (bits & kStatNumeric) return BD_ERR_NUMERIC;
    if (bits & kStatCellOverflow) return BD_ERR_CELL_OVERFLOW;
    if (bits & kStatTimeout) return BD_ERR_TIMEOUT;
    if (bits & kStatArg) return BD_ERR_ARG;
    return BD_OK;
}

#define BD_CUDA_TRY(expr)                                                                    \
    do {                                                                                     \
        cudaError_t _e = (expr);                                                             \
        if (_e != cudaSuccess) {                                                             \
            std::fprintf(stderr, "bd_aging_b200: %s failed: %s (%s:%d)\n", #expr,            \
                         cudaGetErrorString(_e), __FILE__, __LINE__);                        \
            return BD_ERR_CUDA;                                                              \
        }                                                                                    \
    } while (0)

#define BD_LAUNCH_CHECK() BD_CUDA_TRY(cudaPeekAtLastError())

inline int div_up(long a, long b) { return (int)((a + b - 1) / b); }

// Lets launches of `kern` take as much dynamic shared memory as the device
// gives a block; a launch passes what it needs, `bytes` at most (BD_ERR_CUDA
// when that does not fit).  The limit belongs to the kernel on its device, not
// to the engine or call that sets it: every caller sets the same value, so that
// none lowers it below what another's launches need.
template <class K>
inline int allow_smem(K kern, size_t bytes) {
    int dev = 0, most = 0;
    cudaFuncAttributes at;
    BD_CUDA_TRY(cudaGetDevice(&dev));
    BD_CUDA_TRY(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    BD_CUDA_TRY(cudaFuncGetAttributes(&at, kern));
    most -= (int)at.sharedSizeBytes;
    if (bytes > (size_t)most) return BD_ERR_CUDA;
    BD_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    return BD_OK;
}

}  // namespace bd
