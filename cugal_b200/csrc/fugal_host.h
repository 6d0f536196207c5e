// Host-side helpers shared by the .cu files: error reporting, argument checks,
// launch counting and the optional per-kernel event timing.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>

#include "../../include/fugal_b200.h"

namespace fugal {

// Record a message for fugal_last_error() and return `s`.
fugal_status fail(fugal_status s, const char* fmt, ...);

// Map a CUDA error to FUGAL_CUDA_ERROR (with message) or FUGAL_OK.
fugal_status cuda_check(cudaError_t e, const char* what);

// Check the launch that was just issued (cudaGetLastError).
inline fugal_status launch_check(const char* what) { return cuda_check(cudaGetLastError(), what); }

// Count one launch of `family`; if timing is enabled, bracket it with events.
class LaunchScope {
   public:
    LaunchScope(int family, cudaStream_t stream);
    ~LaunchScope();
    LaunchScope(const LaunchScope&) = delete;
    LaunchScope& operator=(const LaunchScope&) = delete;

   private:
    int family_;
    cudaStream_t stream_;
    cudaEvent_t start_ = nullptr;
};

// Fold completed timing events into the totals (non-blocking).
void timing_poll();

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Number of SMs of the current device (cached per device).
int sm_count();

// Failure-detection test hooks, read from the environment at each solve:
// FUGAL_TEST_WAIT_LIMIT_NS (limit of every bounded wait of a solve's kernels; unset: 0, the 2 s
// default), and a local row of CTA 0 whose first copy is armed for 16 bytes that never arrive, so
// that the waits on it run out (unset: -1, none): FUGAL_TEST_FAULT_ROW in sweeps over a 16-bit
// cost, FUGAL_TEST_FAULT_ROW_FP32 in the persistent kernels over FP32 rows.
unsigned long long test_wait_limit_ns();
int test_fault_row(bool fp32);
// FUGAL_TEST_FAULT_BARRIER (unset: 0, none): the last CTA of the adjoint's solve takes its wait on this
// barrier (counted from 1) as run out after it has arrived, so that the others may pass it.
int test_fault_barrier();

// Allow `fn` the largest dynamic shared memory the device gives a CTA next to its static arrays
// (an error if `bytes` is more).  The limit belongs to the function, not to a launch, and launches
// of several host threads may lie between a call and its own launch: a limit of the call's own
// size would take away what a larger one has asked for.
fugal_status allow_dynamic_smem(const void* fn, size_t bytes, const char* what);
template <typename... Args>
fugal_status allow_dynamic_smem(void (*fn)(Args...), size_t bytes, const char* what) {
    return allow_dynamic_smem(reinterpret_cast<const void*>(fn), bytes, what);
}

}  // namespace fugal

#define FUGAL_TRY(expr)                              \
    do {                                             \
        fugal_status _s = (expr);                    \
        if (_s != FUGAL_OK) return _s;               \
    } while (0)
