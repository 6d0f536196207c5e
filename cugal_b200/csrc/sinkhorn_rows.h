// Host interface of the row-owned persistent sweeps (sinkhorn_rows.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "fugal_host.h"

namespace fugal {

struct SolveState;

constexpr int kRowsMaxStages = 32;
constexpr int kRowsMaxSweeps = 4096;  // sweeps per launch

struct RowsArgs {
    const void* L;         // cost (FP32, or its 16-bit copy), n x ld
    long long ld;
    int n;
    int n_copy;            // columns copied per row (multiple of 16 bytes)
    int rows_per_cta;
    int stages;
    int resident;          // every row of a CTA has a stage of its own: copied once per launch
    int sweeps;            // sweeps this launch may run
    unsigned suspend_ns;
    float* b_buf;          // [2][n_pad] column duals of consecutive sweeps
    float* logcs;          // log column sums of the previous sweep
    float* b_next;         // b - log colsum: the next sweep's column duals without momentum
    float* a;              // row duals
    float* partials;       // [CTAs][n_pad]
    double* errs;          // [CTAs] column error of a sweep
    float* corrs;          // [CTAs] largest |column correction|
    long long n_pad;
    SolveState* st;
    // Failure-detection test hooks (host environment): the limit of every bounded
    // wait (0: the 2 s default), and a local row of CTA 0 whose first copy is armed
    // for 16 bytes more than it delivers (-1: none), so that the waits on it run out.
    unsigned long long wait_limit_ns;
    int fault_row;
};

struct RowsPlan {
    bool use = false;
    int dt = 0;
    int ept = 0;           // columns per thread
    int streams = 0;       // row streams (groups of warps) per CTA
    int ctas = 0;          // each writes one row of column partials
    int rows_per_cta = 0;
    int stages = 0;
    int resident = 0;
    size_t smem = 0;
};

// Plan for n columns of element type dt (FUGAL_F32, FUGAL_BF16, FUGAL_F16);
// use = false where these kernels do not apply.  Needs no device with device = false.
fugal_status make_rows_plan(int64_t n, int dt, RowsPlan& plan, bool device);

fugal_status launch_rows(const RowsPlan& plan, RowsArgs args, cudaStream_t stream, int family);

}  // namespace fugal
