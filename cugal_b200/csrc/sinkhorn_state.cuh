// State of a log-domain Sinkhorn solve and the device helpers its sweep kernels
// share (sinkhorn.cu: cluster sweeps; sinkhorn_rows.cu: row-owned sweeps).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>

#include "fugal_common.cuh"
#include "fugal_host.h"

namespace fugal {

struct SolveState {
    int it;          // index of the next sweep
    int done;        // set when the current phase has finished
    int final_it;    // index of the last sweep of the current phase
    int n_err;
    unsigned int ticket;
    int status;      // device-side error code (bounded waits)
    int max_it;      // phase ends after sweep max_it - 1
    int check;       // 1: main phase (convergence checks), 0: polish
    int eval_freq;
    int momentum_start;
    int main_final_it;
    int main_n_err;
    int polish_count;
    int exact_next;  // 1: the next sweep reduces rows with the exact (two-barrier) path
    float max_corr;  // max |log colsum| of the current sweep (as float bits, atomicMax)
    unsigned int arrivals;  // grid barrier of the row-owned sweeps (a multiple of their grid between kernels)
    double threshold;
    double omega;
    double err_accum;
    double last_err;
    double main_last_err;
    double polish_err;
    double errors[FUGAL_MAX_RECORDED_ERRORS];
};

FUGAL_DEVICE double lehmann_momentum(const SolveState* st) {
    return lehmann_omega(st->errors, st->n_err, st->eval_freq, st->momentum_start);
}

// End-of-sweep decision (single thread).
FUGAL_DEVICE void decide(SolveState* st, double err) {
    const int t = st->it;
    st->last_err = err;
    bool stop = false;
    if (st->check) {
        if (t % st->eval_freq == 0 && t != 0) {
            if (st->n_err < FUGAL_MAX_RECORDED_ERRORS) st->errors[st->n_err] = err;
            st->n_err += 1;
            if (err < st->threshold)
                stop = true;
            else
                st->omega = lehmann_momentum(st);
        }
    } else {
        st->polish_err = err;
        st->polish_count += 1;
    }
    if (!stop && t + 1 >= st->max_it) stop = true;
    if (st->status != 0) stop = true;  // a bounded wait timed out: end the phase
    if (stop) {
        st->done = 1;
        st->final_it = t;
        if (st->check) {
            st->main_final_it = t;
            st->main_n_err = st->n_err;
            st->main_last_err = err;
        }
    }
    st->it = t + 1;
}

// Largest |column correction| (nats) after which the next sweep uses the exact
// (max-stabilised) row reduction instead of the previous row normaliser.
constexpr float kFastPathLimit = 30.0f;

// One 16-byte chunk of T as float pairs (elements 2q, 2q+1 in .x, .y).
template <typename T> struct Pairs;
template <> struct Pairs<float> {
    FUGAL_DEVICE static void unpack(const uint4& r, float2* o) {
        o[0] = make_float2(__uint_as_float(r.x), __uint_as_float(r.y));
        o[1] = make_float2(__uint_as_float(r.z), __uint_as_float(r.w));
    }
};
template <> struct Pairs<__nv_bfloat16> {
    FUGAL_DEVICE static void unpack(const uint4& r, float2* o) {
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    }
};
template <> struct Pairs<__half> {
    FUGAL_DEVICE static void unpack(const uint4& r, float2* o) {
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    }
};

FUGAL_DEVICE float2 ex2_pair(float2 x) { return make_float2(ex2(x.x), ex2(x.y)); }

// 2^x for two lanes on the FMA pipe instead of MUFU (Cody-Waite style
// reduction): k = round(x) by the 1.5 * 2^23 rounding constant, f = x - k in
// [-1/2, 1/2], 2^f by a degree-6 polynomial, and k added to the result's
// exponent bits.  The coefficients were fitted for this file by Lawson's
// iteratively reweighted least squares, minimising the relative error on
// [-1/2, 1/2]: 1.9e-9 in exact arithmetic, under 8e-8 (about 1 ulp) with FP32
// Horner steps -- no worse than ex2.approx.  x is clamped to [-127, 127] (so a
// huge x still gives a huge finite value) and x < -126 gives 0, as
// ex2.approx.ftz flushes results below 2^-126; -inf gives 0.
FUGAL_DEVICE float2 ex2_poly_pair(float2 x) {
    const float2 xc = make_float2(fminf(fmaxf(x.x, -127.f), 127.f), fminf(fmaxf(x.y, -127.f), 127.f));
    const float2 rnd = make_float2(12582912.f, 12582912.f);  // 1.5 * 2^23
    const float2 t = __fadd2_rn(xc, rnd);                     // rnd + round(x)
    const float2 k = __fadd2_rn(t, make_float2(-12582912.f, -12582912.f));
    const float2 f = __ffma2_rn(k, make_float2(-1.f, -1.f), xc);  // x - k, exact
    float2 q = make_float2(1.534581242594868e-4f, 1.534581242594868e-4f);
    q = __ffma2_rn(q, f, make_float2(1.3399930903688073e-3f, 1.3399930903688073e-3f));
    q = __ffma2_rn(q, f, make_float2(9.618489071726799e-3f, 9.618489071726799e-3f));
    q = __ffma2_rn(q, f, make_float2(5.550328642129898e-2f, 5.550328642129898e-2f));
    q = __ffma2_rn(q, f, make_float2(2.4022646248340607e-1f, 2.4022646248340607e-1f));
    q = __ffma2_rn(q, f, make_float2(6.931471824645996e-1f, 6.931471824645996e-1f));
    q = __ffma2_rn(q, f, make_float2(1.f, 1.f));
    // the bits of t are those of rnd plus round(x); rnd's low 9 bits are 0, so
    // (bits(t) << 23) is round(x) << 23 modulo 2^32: round(x) added to the exponent
    float2 y;
    y.x = __int_as_float(__float_as_int(q.x) + (__float_as_int(t.x) << 23));
    y.y = __int_as_float(__float_as_int(q.y) + (__float_as_int(t.y) << 23));
    if (x.x < -126.f) y.x = 0.f;
    if (x.y < -126.f) y.y = 0.f;
    return y;
}

}  // namespace fugal
