// Shared helpers of the vtem_b200 CUDA library (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/vtem_b200.h"

#define VTB_API extern "C" __attribute__((visibility("default")))

namespace vtb {

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Records the CUDA error (if any) of the launch just issued and maps it to a
// status code.  Kernel launch errors are synchronous; execution faults are
// reported by the next synchronising call on the caller's side.
int launch_status();

void set_last_cuda_error(cudaError_t e);

// Polls after which a bounded device wait gives up: the process-wide value
// set by vtb_set_wait_limit, else the kernel's default.
uint32_t wait_limit(uint32_t default_polls);

constexpr int kNumSMs = 148;

// Dynamic shared memory allowed to the kernels whose need goes with the call's
// sizes.  The limit is an attribute of the kernel, shared by every host thread:
// set to one call's need, another thread's smaller call could lower it before the
// launch that needs it (which is then refused), so it is only ever set to this.
constexpr size_t kCallSmem = 200 * 1024;

template <typename Kernel>
inline cudaError_t allow_call_smem(Kernel* kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCallSmem);
}

inline int ceil_div(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// lower_bound of v in the sorted a[0..n) by one full warp: 32-way probes
// (three dependent rounds for 25k entries instead of fifteen), the same
// result on every lane.
__device__ __forceinline__ int warp_lower_bound(const int32_t* __restrict__ a, int n, int v) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;
    while (hi - lo > 32) {
        const int step = (hi - lo + 31) / 32;
        const int pos = lo + lane * step;
        const int c = __popc(__ballot_sync(full, pos < hi && a[pos] < v));
        if (c == 0) {
            hi = lo;
        } else {
            const int nlo = lo + (c - 1) * step + 1;
            hi = min(hi, lo + c * step);
            lo = nlo;
        }
    }
    const int pos = lo + lane;
    return lo + __popc(__ballot_sync(full, pos < hi && a[pos] < v));
}

}  // namespace vtb

#define VTB_CHECK_ARG(cond)            \
    do {                               \
        if (!(cond)) return VTB_BAD_ARG; \
    } while (0)

#define VTB_CUDA_TRY(expr)                     \
    do {                                       \
        cudaError_t _e = (expr);               \
        if (_e != cudaSuccess) {               \
            vtb::set_last_cuda_error(_e);      \
            return VTB_CUDA_ERR;               \
        }                                      \
    } while (0)
