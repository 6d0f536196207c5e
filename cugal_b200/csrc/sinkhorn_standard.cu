// Scaling-form Sinkhorn (the reference's SinkhornMethod.STANDARD,
// cugal/sinkhorn.py:122-144) and its Frank-Wolfe update (cugal/pred.py:77-86,
// 136-141), on the kernel matrix K = exp(-C/reg) (FP32, as the reference).
//
// Per iteration t the reference computes
//     v <- v^(1-w) (1 / (u K + eps))^w,   u <- u^(1-w) (1 / (K v + eps))^w,
// and at t % eval_freq == 0 (t = 0 included) the column-marginal error
//     sum_j | sum_i u_i K_ij v_j - 1 |,
// stopping below the threshold and updating the Lehmann factor w otherwise.
// The column sums u K of an iteration give both its error (with the current v) and
// the next v update.  u and v are read and written in place (warm start across
// solves, cugal/sinkhorn.py:51-65).  Two forms:
//   std_rows_kernel (up to 16384 columns): the whole solve in one persistent launch.
//   A CTA owns whole rows (row streams, ring of stages and column state of
//   sinkhorn_rows.cuh); a row is read once per iteration: its product with v gives
//   u_i, and u_i times the row, still in registers, goes into the column sums.
//   wider: round t launches column partial sums of u K, their FP64 merge with the
//   error and the decision on the device, the v update, and the row products K v with
//   the u update.  Rounds after the decision to stop return at once; the host polls
//   the stop flag with a lag of two rounds.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fugal_common.cuh"
#include "fugal_host.h"
#include "sinkhorn_rows.cuh"

namespace fugal {

constexpr float kStdEps = 1e-16f;  // M_EPS, cugal/sinkhorn.py:12
constexpr int kStdThreads = 256;
// Columns of the persistent form: what two streams of 64 columns a thread cover.  Against the launch
// form, us an iteration: n = 1000 8.6 and 34, 6000 40 and 101, 12288 108 and 306, and with one stage a
// stream left 12289 164 and 314, 16384 232 and 452.
constexpr int kStdRowsLimit = FUGAL_STANDARD_ROWS_MAX_N;

struct StdState {
    int done;
    int final_it;
    int n_err;
    int max_it;
    int eval_freq;
    int momentum_start;
    unsigned int ticket;
    int pad;
    double threshold;
    double omega;
    double err_accum;
    double last_err;
    double errors[FUGAL_MAX_RECORDED_ERRORS];
};

struct StdWs {
    StdState* st;
    float* colsum;    // [2][n_pad]: column sums (launch form); v of the pass before (persistent form, momentum)
    float* v_next;    // [n_pad]
    float* partials;  // [chunks][n], or [CTAs][n_pad]
    double* errs;     // [SMs]
    unsigned* sync;   // [2]: grid barrier, status
    size_t bytes;
};

int std_chunks(int64_t n) {
    const int col_blocks = static_cast<int>((n + kStdThreads - 1) / kStdThreads);
    int chunks = std::max(1, (sm_count() * 8) / std::max(1, col_blocks));
    return static_cast<int>(std::min<int64_t>(chunks, std::max<int64_t>(1, n / 8)));
}

StdWs std_layout(int64_t n, char* base) {
    StdWs w{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off = (off + bytes + 255) / 256 * 256;
        return p;
    };
    w.st = reinterpret_cast<StdState*>(take(sizeof(StdState)));
    const size_t n_pad = (static_cast<size_t>(n) + 63) / 64 * 64;
    w.colsum = reinterpret_cast<float*>(take(2 * n_pad * 4));
    w.v_next = reinterpret_cast<float*>(take(n_pad * 4));
    const size_t rows = std::max<size_t>(std_chunks(n), n <= kStdRowsLimit ? sm_count() : 0);
    w.partials = reinterpret_cast<float*>(take(rows * n_pad * 4));
    w.errs = reinterpret_cast<double*>(take(static_cast<size_t>(sm_count()) * 8));
    w.sync = reinterpret_cast<unsigned*>(take(2 * sizeof(unsigned)));
    w.bytes = off;
    return w;
}

__global__ void std_init_kernel(StdState* st, int max_it, int eval_freq, int momentum_start, double threshold) {
    st->done = 0;
    st->final_it = -1;
    st->n_err = 0;
    st->max_it = max_it;
    st->eval_freq = eval_freq;
    st->momentum_start = momentum_start;
    st->ticket = 0;
    st->threshold = threshold;
    st->omega = 1.0;
    st->err_accum = 0.0;
    st->last_err = 0.0;
}

// partials[c][j] = sum over rows of chunk c of u_i K_ij
__global__ void __launch_bounds__(kStdThreads) std_colpart_kernel(const float* __restrict__ K, long long ldk, int n,
                                                                  const float* __restrict__ u, int rows_per_chunk,
                                                                  float* __restrict__ partials,
                                                                  const StdState* st) {
    if (*reinterpret_cast<const volatile int*>(&st->done)) return;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int r0 = blockIdx.y * rows_per_chunk;
    const int r1 = min(n, r0 + rows_per_chunk);
    float acc = 0.f;
    for (int i = r0; i < r1; ++i) acc = fmaf(u[i], K[static_cast<size_t>(i) * ldk + j], acc);
    partials[static_cast<size_t>(blockIdx.y) * n + j] = acc;
}

// colsum_j = sum of the chunk partials (FP64); the error of iteration t-1 when
// it was an evaluation point; the last block takes the decision.
__global__ void __launch_bounds__(kStdThreads) std_merge_kernel(const float* __restrict__ partials, int chunks, int n,
                                                                const float* __restrict__ v, float* colsum,
                                                                StdState* st, int t) {
    __shared__ double red[32];
    __shared__ bool last;
    if (*reinterpret_cast<volatile int*>(&st->done)) return;
    const bool eval = t > 0 && ((t - 1) % st->eval_freq == 0);
    double err = 0.0;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        double c = 0.0;
        for (int k = 0; k < chunks; ++k) c += static_cast<double>(partials[static_cast<size_t>(k) * n + j]);
        const float cf = static_cast<float>(c);
        colsum[j] = cf;
        if (eval) err += fabs(static_cast<double>(v[j]) * static_cast<double>(cf) - 1.0);
    }
    err = block_sum(err, red);
    if (threadIdx.x == 0) {
        if (eval) atomicAdd(&st->err_accum, err);
        __threadfence();
        last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    st->ticket = 0;
    bool stop = false;
    if (eval) {
        const double e = *reinterpret_cast<volatile double*>(&st->err_accum);
        st->err_accum = 0.0;
        st->last_err = e;
        if (st->n_err < FUGAL_MAX_RECORDED_ERRORS) st->errors[st->n_err] = e;
        st->n_err += 1;
        if (e < st->threshold)
            stop = true;
        else
            st->omega = lehmann_omega(st->errors, st->n_err, st->eval_freq, st->momentum_start);
    }
    if (stop || t >= st->max_it) {
        st->done = 1;
        st->final_it = t - 1;
    }
}

// v_j <- v_j^(1-w) (1 / (colsum_j + eps))^w
__global__ void std_vupdate_kernel(const float* colsum, float* v, int n, const StdState* st) {
    if (*reinterpret_cast<const volatile int*>(&st->done)) return;
    const double w = st->omega;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const float x = 1.0f / (colsum[j] + kStdEps);
        v[j] = (w == 1.0) ? x : powf(v[j], static_cast<float>(1.0 - w)) * powf(x, static_cast<float>(w));
    }
}

// u_i <- u_i^(1-w) (1 / (sum_j K_ij v_j + eps))^w, one warp per row.
__global__ void __launch_bounds__(kStdThreads) std_rowdot_kernel(const float* __restrict__ K, long long ldk, int n,
                                                                 const float* __restrict__ v, float* u,
                                                                 const StdState* st) {
    if (*reinterpret_cast<const volatile int*>(&st->done)) return;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const double w = st->omega;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const float* row = K + static_cast<size_t>(i) * ldk;
        float acc = 0.f;
        for (int j = lane; j < n; j += 32) acc = fmaf(row[j], v[j], acc);
        acc = warp_sum(acc);
        if (lane == 0) {
            const float x = 1.0f / (acc + kStdEps);
            u[i] = (w == 1.0) ? x : powf(u[i], static_cast<float>(1.0 - w)) * powf(x, static_cast<float>(w));
        }
    }
}

// The record, if asked for.  A solve whose waits ran out has stopped anywhere in an iteration: its
// u and v become NaN, so that it cannot pass for a result where no record is read.
__global__ void std_end_kernel(const StdState* st, const unsigned* status, int n, float* u, float* v,
                               fugal_solve_record* rec) {
    if (*status != 0)
        for (int j = threadIdx.x; j < n; j += blockDim.x) u[j] = v[j] = NAN;
    if (rec == nullptr) return;
    if (threadIdx.x == 0) {
        rec->iteration_count = st->final_it + 1;
        rec->n_errors = min(st->n_err, FUGAL_MAX_RECORDED_ERRORS);
        rec->status = static_cast<int>(*status);
        rec->polish_count = 0;
        rec->last_error = st->last_err;
        rec->polish_error = 0.0;
    }
    for (int k = threadIdx.x; k < FUGAL_MAX_RECORDED_ERRORS; k += blockDim.x) rec->errors[k] = st->errors[k];
}

// out = exp(scale * C)
__global__ void exp_scale_kernel(const float* __restrict__ C, long long ldc, int n, float scale, float* out,
                                 long long ldo) {
    for (int i = blockIdx.y; i < n; i += gridDim.y)
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
            out[static_cast<size_t>(i) * ldo + j] = expf(C[static_cast<size_t>(i) * ldc + j] * scale);
}

// q = (K_ij v_j) u_i;  P += alpha (q - P);  gap += C (q - P)  (FP64)
__global__ void __launch_bounds__(kStdThreads) std_update_kernel(float* P, long long ldp, const float* K, long long ldk,
                                                                 const float* u, const float* v, const float* C,
                                                                 long long ldc, int n, float alpha, double* gap) {
    __shared__ double red[32];
    double g = 0.0;
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        const float ui = u[i];
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
            const float q = (K[static_cast<size_t>(i) * ldk + j] * v[j]) * ui;
            float* pp = P + static_cast<size_t>(i) * ldp + j;
            const float diff = q - *pp;
            g += static_cast<double>(C[static_cast<size_t>(i) * ldc + j]) * static_cast<double>(diff);
            *pp = fmaf(alpha, diff, *pp);
        }
    }
    g = block_sum(g, red);
    if (threadIdx.x == 0) atomicAdd(gap, g);
}

// ------------------------------------------------------------- persistent form

// Per iteration: one read of K (144 MB at n = 6000, 22 us at the copy peak) where the
// four launches of the other form read it twice (31 + 49 us) and paid their gaps: 101 us
// against 40 us an iteration at n = 6000.
struct StdRowsArgs {
    const float* K;
    long long ldk;
    int n;
    int n_copy;          // columns copied per row: a multiple of 4 within ldk
    int rows_per_cta;
    int stages;
    int resident;
    unsigned suspend_ns;
    float* u;
    float* v;
    float* v_next;       // 1 / (column sum + eps): the next v without momentum
    // n_pad columns on: v of the pass before (momentum).  (As a pointer to it, which the 16 places of
    // its reads fold differently, n = 6000 takes 53.8 instead of 40.0 us an iteration.)
    float* colsum;
    float* partials;
    double* errs;
    long long n_pad;
    StdState* st;
    unsigned* arrivals;
    int* status;
    unsigned long long wait_limit_ns;  // test hooks (test_fault_row in fugal_host.h)
    int fault_row;
};

// x^(1-w) y^w, the momentum update (w != 1)
FUGAL_DEVICE float std_blend(float x, float y, double w) {
    return powf(x, static_cast<float>(1.0 - w)) * powf(y, static_cast<float>(w));
}

__device__ __noinline__ void std_reduce_columns(const StdRowsArgs& p, bool eval, double (*colred)[128]) {
    __shared__ double red[32];
    const int per = columns_per_cta(p.n);
    const int j = blockIdx.x * per + threadIdx.x;
    const bool mine = static_cast<int>(threadIdx.x) < per && j < p.n;
    const float vj = mine && eval ? __ldcg(p.v + j) : 0.f;
    const double tot = own_column_sum(p.partials, p.n_pad, static_cast<int>(gridDim.x), p.n, colred);
    double err = 0.0;
    if (mine) {
        const float cf = static_cast<float>(tot);
        p.v_next[j] = 1.0f / (cf + kStdEps);
        if (eval) err = fabs(static_cast<double>(vj) * static_cast<double>(cf) - 1.0);
    }
    if (eval) {
        err = block_sum(err, red);
        if (threadIdx.x == 0) p.errs[blockIdx.x] = err;
    }
}

// The decision after the column sums of round t (thread 0 of every CTA, the same in all).
__device__ __noinline__ void std_decide(const StdRowsArgs& p, StdState* st, int t, bool eval) {
    if (threadIdx.x >= 32) return;
    double e = 0.0;
    float c;
    if (eval) grid_error(p.errs, nullptr, e, c);
    if (threadIdx.x != 0) return;
    bool stop = false;
    if (eval) {
        st->last_err = e;
        if (st->n_err < FUGAL_MAX_RECORDED_ERRORS) st->errors[st->n_err] = e;
        st->n_err += 1;
        if (e < st->threshold)
            stop = true;
        else
            st->omega = lehmann_omega(st->errors, st->n_err, st->eval_freq, st->momentum_start);
    }
    if (stop || t >= st->max_it) {
        st->done = 1;
        st->final_it = t - 1;
    }
}

template <int EPT, int GR>
__global__ void __launch_bounds__(kRowsThreads, 1) std_rows_kernel(const __grid_constant__ StdRowsArgs p) {
    constexpr int GT = kRowsThreads / GR;
    constexpr int GW = GT / 32;
    constexpr int COVER = GT * EPT;
    constexpr int NCH = EPT / 16;
    constexpr int H = EPT / 2;
    constexpr bool DUMP = rows_dump_bytes(GR, EPT) > 0;
    constexpr uint32_t TCOLS = ColumnState<EPT>::kTmemColumns;
    extern __shared__ __align__(128) unsigned char ring[];
    float* dump = reinterpret_cast<float*>(ring + static_cast<size_t>(p.stages) * COVER * sizeof(float));  // DUMP
    __shared__ uint64_t full[kRowsMaxStages];
    __shared__ int newest[kRowsMaxStages];  // phase of the newest copy into a stage (-1: none)
    __shared__ __align__(16) float red_s[GR][2][GW];
    __shared__ __align__(16) double colred[kRowsWarps][128];  // also where fewer than 8 streams meet
    __shared__ float u_s[kRowsMaxRows];
    __shared__ StdState ss;
    __shared__ uint32_t tmem_slot;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = tid / GT, gt = tid % GT, gw = warp % GW;
    const int n = p.n;
    const int row_begin = blockIdx.x * p.rows_per_cta;
    const int nrows = max(0, min(n, row_begin + p.rows_per_cta) - row_begin);
    const int NST = p.stages;
    for (int k = tid; k < static_cast<int>(sizeof(StdState) / 4); k += kRowsThreads)
        reinterpret_cast<int*>(&ss)[k] = reinterpret_cast<const int*>(p.st)[k];
    for (int i = tid; i < nrows; i += kRowsThreads) u_s[i] = p.u[row_begin + i];
    for (int s = 0; s < NST; ++s) {  // columns past n_copy are never copied
        float* row = reinterpret_cast<float*>(ring) + static_cast<size_t>(s) * COVER;
        for (int j = p.n_copy + tid; j < COVER; j += kRowsThreads) row[j] = 0.f;
    }
    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(&full[s], 1);
            newest[s] = -1;
        }
        fence_mbarrier_init();
    }
    if constexpr (TCOLS > 0) {
        if (warp == 0) {
            tmem_alloc(&tmem_slot, TCOLS);
            tmem_relinquish();
        }
        tmem_fence_before_sync();
    }
    __syncthreads();
    ColumnState<EPT> cols;
    if constexpr (TCOLS > 0) {
        tmem_fence_after_sync();
        cols.start(tmem_slot, warp);
    }

    // ring of whole rows: unit u (row u mod nrows) sits in stage u mod NST; see rows_kernel
    const uint32_t row_bytes = static_cast<uint32_t>(p.n_copy) * sizeof(float);
    auto issue = [&](int row, int s, uint32_t phase, bool first) {
        const uint32_t unmet = (first && blockIdx.x == 0 && row == p.fault_row) ? 16u : 0u;
        newest[s] = static_cast<int>(phase);
        mbar_arrive_expect_tx(&full[s], row_bytes + unmet);
        bulk_load(ring + static_cast<size_t>(s) * COVER * sizeof(float),
                  p.K + static_cast<unsigned long long>(static_cast<unsigned>(row_begin + row)) *
                            static_cast<unsigned long long>(p.ldk),
                  row_bytes, &full[s]);
    };
    if (tid == 0 && nrows > 0) {
        fence_proxy_async_smem();
        const int first = p.resident ? min(nrows, NST) : NST;
        for (int k = 0; k < first; ++k) issue(k % nrows, k, 0u, k < nrows);
    }
    int sbase = 0;
    uint32_t phbase = 0u;
    const int ahead = NST % max(1, nrows);
    auto column_of = [&](int e) { return ((e / 4) * GT + gt) * 4 + e % 4; };
    const bool ragged = (n & 3) != 0;
    unsigned arrivals = 0;
    bool alive = true;
    // round t: the pass over K of iteration t - 1 (t = 0: column sums with the given u),
    // then the error of that iteration, the decision, and v of iteration t
    for (int t = 0;; ++t) {
        const double omega = ss.omega;
        // ---- v of this pass: written by CTA 0, kept with the columns
        float4 v_raw[EPT / 4];  // all loads in flight
#pragma unroll
        for (int k = 0; k < EPT / 4; ++k) {
            const int j = column_of(4 * k);
            v_raw[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            // v_next is n_pad long, a multiple of 64 columns
            if (t > 0 && j < n) v_raw[k] = __ldcg(reinterpret_cast<const float4*>(p.v_next + j));
        }
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            float vv[16];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int j = column_of(16 * c + 4 * k);
                float4 v4 = v_raw[4 * c + k];
                if (t > 0 && j < n) {
                    float* e = reinterpret_cast<float*>(&v4);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (j + q >= n) {
                            e[q] = 0.f;
                        } else {
                            // with momentum every thread that needs v_j blends it from v's other copy
                            if (omega != 1.0) e[q] = std_blend(__ldcg(p.colsum + p.n_pad + j + q), e[q], omega);
                            if (blockIdx.x == 0 && g == 0) p.v[j + q] = e[q];
                        }
                    }
                }
                vv[4 * k] = v4.x;
                vv[4 * k + 1] = v4.y;
                vv[4 * k + 2] = v4.z;
                vv[4 * k + 3] = v4.w;
            }
            cols.set(c, vv);
        }
        cols.ready();

        float2 y[H];
        float wp = 0.f;
#pragma unroll
        for (int h = 0; h < H; ++h) y[h] = make_float2(0.f, 0.f);
        int s_cur = sbase + g;
        uint32_t ph = phbase;
        while (s_cur >= NST) {
            s_cur -= NST;
            ph ^= 1u;
        }
        int par = 0;
        for (int r = g; r < nrows; r += GR, par ^= 1) {
            const int s = s_cur;
            const float* stage = reinterpret_cast<const float*>(ring) + static_cast<size_t>(s) * COVER;
            const bool ok = (p.resident && t > 0) ||
                            mbar_wait<true>(&full[s], p.resident ? 0u : ph, p.status, p.suspend_ns, p.wait_limit_ns);
            cols.settle();
            float2 s2 = make_float2(0.f, 0.f), t2 = make_float2(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                cols.add(c, y + 8 * c, wp);
                float2 v2[8];
                cols.duals(c, v2);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float4 k4 = *reinterpret_cast<const float4*>(stage + ((c * 4 + i) * GT + gt) * 4);
                    if (ragged) {  // the copied row's last quad may hold anything past n
                        const int j = column_of(16 * c + 4 * i);
                        if (j + 1 >= n) k4.y = 0.f;
                        if (j + 2 >= n) k4.z = 0.f;
                        if (j + 3 >= n) k4.w = 0.f;
                    }
                    y[8 * c + 2 * i] = make_float2(k4.x, k4.y);
                    y[8 * c + 2 * i + 1] = make_float2(k4.z, k4.w);
                    s2 = __ffma2_rn(y[8 * c + 2 * i], v2[2 * i], s2);
                    t2 = __ffma2_rn(y[8 * c + 2 * i + 1], v2[2 * i + 1], t2);
                }
            }
            const float2 u2 = __fadd2_rn(s2, t2);
            const float part = warp_sum(u2.x + u2.y);
            if (lane == 0) red_s[g][par][gw] = part;
            if (!stream_and<GT>(ok, g)) {
                alive = false;
                break;
            }
            // the stage has been read by every thread of the stream
            if (gt == 0 && !p.resident) {
                int row = r + ahead;
                if (row >= nrows) row -= nrows;
                fence_proxy_async_smem();  // the reads of the stage precede the copy into it
                issue(row, s, ph ^ 1u, false);
            }
            if (t == 0) {
                wp = u_s[r];
            } else {
                const float x = 1.0f / (sum_warps<GW>(red_s[g][par]) + kStdEps);
                wp = x;
                if (omega != 1.0) {
                    wp = std_blend(u_s[r], x, omega);
                    stream_and<GT>(true, g);  // every thread has read u_s[r]
                }
                if (gt == GT - 32) {
                    u_s[r] = wp;
                    p.u[row_begin + r] = wp;
                }
            }
            s_cur += GR;
            while (s_cur >= NST) {
                s_cur -= NST;
                ph ^= 1u;
            }
        }
        // ---- column sums of the CTA
        {
            float* prow = p.partials + static_cast<size_t>(blockIdx.x) * p.n_pad;
            float* to = DUMP ? dump + static_cast<size_t>(g) * COVER : prow;
            cols.settle();
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                float acc[16];
                cols.total(c, y + 8 * c, wp, acc);
                if constexpr (GR > 1 && !DUMP) {
                    meet_streams<GR, GT, 4>(reinterpret_cast<float*>(colred), acc, c, g, gt, n, prow);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int j = column_of(16 * c + 4 * k);
                        if (j < n)
                            *reinterpret_cast<float4*>(to + j) =
                                make_float4(acc[4 * k], acc[4 * k + 1], acc[4 * k + 2], acc[4 * k + 3]);
                    }
                }
            }
            if constexpr (DUMP) {
                __syncthreads();
                for (int j = tid * 4; j < n; j += kRowsThreads * 4) {
                    float4 v[GR];
#pragma unroll
                    for (int k = 0; k < GR; ++k) v[k] = *reinterpret_cast<const float4*>(dump + k * COVER + j);
#pragma unroll
                    for (int o = 1; o < GR; o <<= 1) {
#pragma unroll
                        for (int k = 0; k < GR; k += 2 * o) {
                            v[k].x += v[k + o].x;
                            v[k].y += v[k + o].y;
                            v[k].z += v[k + o].z;
                            v[k].w += v[k + o].w;
                        }
                    }
                    *reinterpret_cast<float4*>(prow + j) = v[0];
                }
            }
        }
        arrivals += gridDim.x;
        if (!grid_barrier(p.arrivals, p.status, alive, arrivals, p.wait_limit_ns)) {
            alive = false;
            break;
        }
        const bool eval = t > 0 && ((t - 1) % ss.eval_freq == 0);
        std_reduce_columns(p, eval, colred);
        if (ss.momentum_start >= 0) {
            // v of this pass for the blend of the next one (CTA 0 overwrites p.v meanwhile)
            __syncthreads();
            const int per = columns_per_cta(n);
            const int j = blockIdx.x * per + tid;
            if (tid < per && j < n) p.colsum[p.n_pad + j] = __ldcg(p.v + j);
        }
        arrivals += gridDim.x;
        if (!grid_barrier(p.arrivals, p.status, true, arrivals, p.wait_limit_ns)) {
            alive = false;
            break;
        }
        std_decide(p, &ss, t, eval);
        if (!p.resident) {
            sbase += nrows;
            while (sbase >= NST) {
                sbase -= NST;
                phbase ^= 1u;
            }
        }
        __syncthreads();
        if (ss.done) break;
    }
    __syncthreads();
    if (tid == 0) {  // copies still in flight (bounded waits)
        for (int s = 0; s < NST; ++s)
            if (newest[s] >= 0)
                mbar_wait<true>(&full[s], static_cast<uint32_t>(newest[s]), p.status, p.suspend_ns, p.wait_limit_ns);
    }
    if (blockIdx.x == 0) {
        if (tid == 0) {
            p.st->done = 1;
            p.st->final_it = ss.final_it;
            p.st->n_err = ss.n_err;
            p.st->omega = ss.omega;
            p.st->last_err = ss.last_err;
        }
        for (int k = tid; k < min(ss.n_err, FUGAL_MAX_RECORDED_ERRORS); k += kRowsThreads) p.st->errors[k] = ss.errors[k];
    }
    if constexpr (TCOLS > 0) {
        tmem_fence_before_sync();
        __syncthreads();
        tmem_fence_after_sync();
        if (warp == 0) tmem_dealloc(tmem_slot, TCOLS);
    }
}

struct StdRowsPlan {
    bool use = false;
    int ept = 0, streams = 0, ctas = 0, rows_per_cta = 0, stages = 0, resident = 0;
    size_t smem = 0;
};
constexpr int kStdShapes[][2] = {{8, 16}, {8, 32}, {4, 32}, {4, 48}, {2, 32}, {2, 48}, {2, 64}};

using StdRowsFn = void (*)(StdRowsArgs);
StdRowsFn std_rows_fn(const StdRowsPlan& pl) {
    switch (pl.streams * 100 + pl.ept) {
        case 816: return std_rows_kernel<16, 8>;
        case 832: return std_rows_kernel<32, 8>;
        case 432: return std_rows_kernel<32, 4>;
        case 448: return std_rows_kernel<48, 4>;
        case 232: return std_rows_kernel<32, 2>;
        case 248: return std_rows_kernel<48, 2>;
        default: return std_rows_kernel<64, 2>;
    }
}

// Rows are copied in 16-byte pieces: K's rows aligned, n rounded up to 4 within ldk.  The vectors of
// the workspace are read 16 bytes at a time; the launch form needs 8-byte boundaries only.
StdRowsPlan std_rows_plan(int64_t n, int64_t ldk, const float* K, const void* workspace) {
    StdRowsPlan pl;
    if (n > kStdRowsLimit || (ldk % 4) != 0 || ldk < (n + 3) / 4 * 4 || !aligned16(K) || !aligned16(workspace))
        return pl;
    for (const auto& sh : kStdShapes)
        if (static_cast<int64_t>(kRowsThreads / sh[0]) * sh[1] >= n) {
            pl.streams = sh[0];
            pl.ept = sh[1];
            break;
        }
    const int want = static_cast<int>(std::min<int64_t>(sm_count(), n));
    pl.rows_per_cta = static_cast<int>((n + want - 1) / want);
    if (pl.rows_per_cta > kRowsMaxRows) return pl;
    pl.ctas = static_cast<int>((n + pl.rows_per_cta - 1) / pl.rows_per_cta);
    const size_t stage = static_cast<size_t>(kRowsThreads / pl.streams) * pl.ept * 4;
    const size_t dump = rows_dump_bytes(pl.streams, pl.ept);
    const size_t room = 227 * 1024 - kRowsStatic - dump;
    pl.stages = static_cast<int>(
        std::min<size_t>({room / stage, static_cast<size_t>(kRowsMaxStages), static_cast<size_t>(pl.rows_per_cta)}));
    pl.resident = pl.stages >= pl.rows_per_cta;
    if (!pl.resident) pl.stages -= pl.stages % pl.streams;  // a stage stays with its stream: see make_rows_plan
    if (pl.stages < 1) return pl;
    pl.smem = stage * pl.stages + dump;
    int dev = 0, coop = 0, blocks = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return pl;
    StdRowsFn fn = std_rows_fn(pl);
    if (allow_dynamic_smem(fn, pl.smem, "sinkhorn standard: shared memory") != FUGAL_OK ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, kRowsThreads, pl.smem) != cudaSuccess || blocks < 1) {
        (void)cudaGetLastError();
        return pl;
    }
    pl.use = true;
    return pl;
}

}  // namespace fugal

using namespace fugal;

extern "C" fugal_status fugal_sinkhorn_standard_workspace_size(int64_t n, size_t* bytes) {
    if (bytes == nullptr) return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_standard_workspace_size: null output");
    if (n <= 0 || n > (1ll << 30)) return fail(FUGAL_BAD_SHAPE, "fugal_sinkhorn_standard_workspace_size: bad n");
    *bytes = std_layout(n, nullptr).bytes;
    return FUGAL_OK;
}

namespace {
constexpr int kStdPinnedSlots = 64;
constexpr int kStdPollLag = 2;
thread_local int* g_std_pinned = nullptr;
thread_local int g_std_next = 0;
}  // namespace

extern "C" fugal_status fugal_sinkhorn_standard_solve(const float* K, int64_t ldk, int64_t n, float* u, float* v,
                                                      int max_iterations, double threshold, int eval_freq,
                                                      int momentum_start, void* record, void* workspace,
                                                      size_t workspace_bytes, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    size_t need = 0;
    FUGAL_TRY(fugal_sinkhorn_standard_workspace_size(n, &need));
    if (K == nullptr || u == nullptr || v == nullptr || workspace == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_standard_solve: null argument");
    if (ldk < n) return fail(FUGAL_BAD_SHAPE, "fugal_sinkhorn_standard_solve: ldk < n");
    if (max_iterations <= 0 || eval_freq <= 0)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_standard_solve: max_iterations and eval_freq must be positive");
    if (workspace_bytes < need)
        return fail(FUGAL_WORKSPACE_TOO_SMALL, "fugal_sinkhorn_standard_solve: workspace %zu < %zu", workspace_bytes,
                    need);
    StdWs w = std_layout(n, static_cast<char*>(workspace));
    const int nn = static_cast<int>(n);
    const int chunks = std_chunks(n);
    const int rows_per_chunk = (nn + chunks - 1) / chunks;
    const int vec_blocks = static_cast<int>(std::min<int64_t>((n + kStdThreads - 1) / kStdThreads, 4 * sm_count()));
    const int row_blocks = static_cast<int>(std::min<int64_t>((n * 32 + kStdThreads - 1) / kStdThreads, 16 * sm_count()));
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        std_init_kernel<<<1, 1, 0, stream>>>(w.st, max_iterations, eval_freq, momentum_start < 0 ? -1 : momentum_start,
                                             threshold);
        FUGAL_TRY(launch_check("sinkhorn standard: init"));
    }
    FUGAL_TRY(cuda_check(cudaMemsetAsync(w.sync, 0, 2 * sizeof(unsigned), stream), "sinkhorn standard: clear"));
    const StdRowsPlan plan = std_rows_plan(n, ldk, K, workspace);
    if (plan.use) {
        StdRowsArgs ra{};
        ra.K = K;
        ra.ldk = ldk;
        ra.n = nn;
        ra.n_copy = (nn + 3) / 4 * 4;
        ra.rows_per_cta = plan.rows_per_cta;
        ra.stages = plan.stages;
        ra.resident = plan.resident;
        ra.suspend_ns = kSuspendHintNs;
        ra.u = u;
        ra.v = v;
        ra.v_next = w.v_next;
        ra.colsum = w.colsum;
        ra.partials = w.partials;
        ra.errs = w.errs;
        ra.n_pad = (n + 63) / 64 * 64;
        ra.st = w.st;
        ra.arrivals = w.sync;
        ra.status = reinterpret_cast<int*>(w.sync + 1);
        ra.wait_limit_ns = test_wait_limit_ns();
        ra.fault_row = test_fault_row(true);
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        cfg.gridDim = dim3(plan.ctas, 1, 1);
        cfg.blockDim = dim3(kRowsThreads, 1, 1);
        cfg.dynamicSmemBytes = plan.smem;
        cfg.stream = stream;
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        {
            LaunchScope scope(FUGAL_KERNEL_SWEEP_F32, stream);
            FUGAL_TRY(cuda_check(cudaLaunchKernelEx(&cfg, std_rows_fn(plan), ra), "sinkhorn standard: rows"));
        }
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        std_end_kernel<<<1, 256, 0, stream>>>(w.st, w.sync + 1, nn, u, v, static_cast<fugal_solve_record*>(record));
        return launch_check("sinkhorn standard: record");
    }
    if (g_std_pinned == nullptr) {
        void* p = nullptr;
        FUGAL_TRY(cuda_check(cudaHostAlloc(&p, kStdPinnedSlots * sizeof(int), cudaHostAllocPortable),
                             "sinkhorn standard: pinned flags"));
        g_std_pinned = static_cast<int*>(p);
    }
    int* pinned = g_std_pinned + g_std_next;
    g_std_next = (g_std_next + 2) % kStdPinnedSlots;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    FUGAL_TRY(cuda_check(cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming), "sinkhorn standard: event"));
    FUGAL_TRY(cuda_check(cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming), "sinkhorn standard: event"));
    fugal_status status = FUGAL_OK;
    int slot = 0, poll_slot = -1, poll_t = 0;
    // round t evaluates iteration t-1 (if it was an evaluation point) and, unless
    // the solve stopped, runs iteration t
    for (int t = 0; t <= max_iterations && status == FUGAL_OK; ++t) {
        {
            LaunchScope scope(FUGAL_KERNEL_COLUMN_PASS, stream);
            std_colpart_kernel<<<dim3((nn + kStdThreads - 1) / kStdThreads, chunks), kStdThreads, 0, stream>>>(
                K, ldk, nn, u, rows_per_chunk, w.partials, w.st);
            status = launch_check("sinkhorn standard: column partials");
        }
        if (status != FUGAL_OK) break;
        {
            LaunchScope scope(FUGAL_KERNEL_FINALIZE, stream);
            std_merge_kernel<<<vec_blocks, kStdThreads, 0, stream>>>(w.partials, chunks, nn, v, w.colsum, w.st, t);
            status = launch_check("sinkhorn standard: merge");
        }
        if (status != FUGAL_OK || t == max_iterations) break;
        {
            LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
            std_vupdate_kernel<<<vec_blocks, kStdThreads, 0, stream>>>(w.colsum, v, nn, w.st);
            status = launch_check("sinkhorn standard: v update");
        }
        if (status != FUGAL_OK) break;
        {
            LaunchScope scope(FUGAL_KERNEL_SWEEP_F32, stream);
            std_rowdot_kernel<<<row_blocks, kStdThreads, 0, stream>>>(K, ldk, nn, v, u, w.st);
            status = launch_check("sinkhorn standard: u update");
        }
        if (status != FUGAL_OK) break;
        // poll the stop flag written by round t's decision, kStdPollLag rounds later
        if (poll_slot >= 0 && t - poll_t >= kStdPollLag) {
            status = cuda_check(cudaEventSynchronize(ev[poll_slot]), "sinkhorn standard: poll wait");
            timing_poll();
            const bool stop = status == FUGAL_OK && pinned[poll_slot] != 0;
            poll_slot = -1;
            if (stop) break;
        }
        if (poll_slot < 0 && t > 0 && (t - 1) % eval_freq == 0) {
            slot ^= 1;
            status = cuda_check(cudaMemcpyAsync(&pinned[slot], &w.st->done, sizeof(int), cudaMemcpyDeviceToHost, stream),
                                "sinkhorn standard: poll copy");
            if (status == FUGAL_OK) status = cuda_check(cudaEventRecord(ev[slot], stream), "sinkhorn standard: poll event");
            poll_slot = slot;
            poll_t = t;
        }
    }
    if (status == FUGAL_OK && record != nullptr) {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        std_end_kernel<<<1, 256, 0, stream>>>(w.st, w.sync + 1, nn, u, v, static_cast<fugal_solve_record*>(record));
        status = launch_check("sinkhorn standard: record");
    }
    cudaEventDestroy(ev[0]);
    cudaEventDestroy(ev[1]);
    return status;
}

extern "C" fugal_status fugal_exp_scale(const float* C, int64_t ldc, int64_t n, double scale, float* out, int64_t ldo,
                                        fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (C == nullptr || out == nullptr) return fail(FUGAL_BAD_ARGUMENT, "fugal_exp_scale: null argument");
    if (n <= 0 || ldc < n || ldo < n) return fail(FUGAL_BAD_SHAPE, "fugal_exp_scale: bad shape");
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    dim3 grid(static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 64)),
              static_cast<unsigned>(std::min<int64_t>(n, 65535)));
    exp_scale_kernel<<<grid, 256, 0, stream>>>(C, ldc, static_cast<int>(n), static_cast<float>(scale), out, ldo);
    return launch_check("fugal_exp_scale");
}

extern "C" fugal_status fugal_fw_update_standard(int64_t n, float* P, int64_t ldp, const float* K, int64_t ldk,
                                                 const float* u, const float* v, const float* C, int64_t ldc,
                                                 double alpha, double* gap, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (P == nullptr || K == nullptr || u == nullptr || v == nullptr || C == nullptr || gap == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_fw_update_standard: null argument");
    if (n <= 0 || ldp < n || ldk < n || ldc < n) return fail(FUGAL_BAD_SHAPE, "fugal_fw_update_standard: bad shape");
    FUGAL_TRY(cuda_check(cudaMemsetAsync(gap, 0, sizeof(double), stream), "fugal_fw_update_standard: clear gap"));
    LaunchScope scope(FUGAL_KERNEL_UPDATE, stream);
    dim3 grid(static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 16)),
              static_cast<unsigned>(std::min<int64_t>(n, 8 * sm_count())));
    std_update_kernel<<<grid, kStdThreads, 0, stream>>>(P, ldp, K, ldk, u, v, C, ldc, static_cast<int>(n),
                                                        static_cast<float>(alpha), gap);
    return launch_check("fugal_fw_update_standard");
}
