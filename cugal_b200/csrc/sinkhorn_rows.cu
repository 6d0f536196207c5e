// Row-owned, persistent log-domain Sinkhorn sweeps (see sinkhorn.cu for what a
// sweep is): one launch runs up to args.sweeps iteration boundaries.
//
// One 512-thread CTA per SM owns a block of whole rows.  Its 16 warps form
// `GR` row streams of 512 / GR threads; stream g takes rows g, g + GR, ... of the
// block, EPT columns per thread, so the row normaliser is a barrier of one
// stream and the streams hide part of each other's reduction and barrier latency.
// Running column sums and the column duals (b log2 e) of a thread's columns are
// registers up to EPT = 32, tensor memory above.  A row's exponentials stay in
// registers until the next row of the stream overwrites them chunk by chunk, each
// 16-column chunk being added into the column sums right before.  Rows stream
// through a ring of whole-row stages in shared memory (bulk copies); the cost does
// not depend on the duals, so the ring already fills with the next sweep's first rows
// while the CTAs exchange column sums.  When all rows of a CTA fit the ring they are
// copied once and stay.
//
// What bounds it: small n, the two grid exchanges (about 6 us a sweep, of which 1.4 us
// are each barrier and 2.2 us the FP64 column sums); from n = 3000 on the per-row
// chain of a stream (wait, exponentials, shuffles, barrier, reciprocal: about 1.5 us
// with 32 columns a thread) against MUFU and HBM.  Time per iteration, FP32, this
// kernel against a cluster sweep and a finalize kernel per iteration: n = 1000 7.8
// against 23.5 us, 4096 19.7 against 45.7, 8192 50.4 against 77.5 (41 us at the copy
// peak); BF16: 4096 18.6 against 37.6, 8192 41.1 against 62.1, 16384 119 against 158,
// 20011 217 against 275.  One exponential pair in 8 on the FMA pipe, worth 1.5% in the
// 64-column kernel, costs 2 to 7% here (instruction issue) and is not used.
//
// End of a sweep: every CTA writes its column sums; grid barrier; each CTA
// adds up its share of the columns in FP64 and writes log(colsum), its error and
// its largest correction; grid barrier; every CTA sums the errors in the same
// order and takes the same decision on its own copy of the solve state, which CTA
// 0 writes back when the launch ends.  The launch is cooperative, so all CTAs are
// resident; every wait is bounded, and a timed-out one ends the kernel with
// FUGAL_DEVICE_TIMEOUT in the state.
#include <algorithm>
#include <type_traits>

#include "fugal_common.cuh"
#include "sinkhorn_rows.cuh"
#include "sinkhorn_state.cuh"

namespace fugal {

// This CTA's share of the columns: log(colsum), the next duals, the CTA's error and
// largest correction.  (Not inlined: its registers would be live across the row loop.)
__device__ __noinline__ void reduce_columns(const RowsArgs& p, int t, double (*colred)[128]) {
    __shared__ double errred[kRowsWarps];
    __shared__ float corred[kRowsWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = columns_per_cta(p.n);
    const int j = blockIdx.x * per + tid;
    const bool mine = tid < per && j < p.n;
    float b_now = 0.f;
    if (mine) b_now = __ldcg(p.b_buf + (t & 1) * p.n_pad + j);
    const double tot = own_column_sum(p.partials, p.n_pad, static_cast<int>(gridDim.x), p.n, colred);
    double err = 0.0;
    float corr = 0.f;
    if (mine) {
        err = fabs(tot - 1.0);
        const float lg = static_cast<float>(log(fmax(tot, 1e-37)));
        p.logcs[j] = lg;
        p.b_next[j] = b_now - lg;  // the next sweep's dual without momentum
        corr = fabsf(lg);
    }
    const int used = (per + 31) / 32;  // warps that hold columns
    if (warp < used) {
        // (columns sit in lanes below `per`; adding the zeros of the others changes nothing)
        for (int o = per > 16 ? 16 : per > 8 ? 8 : per > 4 ? 4 : 2; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
        corr = warp_max_positive(corr);
        if (used == 1) {
            if (lane == 0) {
                p.errs[blockIdx.x] = err;
                p.corrs[blockIdx.x] = corr;
            }
        } else if (lane == 0) {
            errred[warp] = err;
            corred[warp] = corr;
        }
    }
    if (used > 1) {
        __syncthreads();
        if (tid == 0) {
            double e = 0.0;
            float c = 0.f;
            for (int w = 0; w < used; ++w) {
                e += errred[w];
                c = fmaxf(c, corred[w]);
            }
            p.errs[blockIdx.x] = e;
            p.corrs[blockIdx.x] = c;
        }
    }
}

// The decision at the end of a sweep, the same in every CTA (warp 0).
__device__ __noinline__ void take_decision(const RowsArgs& p, SolveState* ss) {
    if (threadIdx.x < 32) {
        double e;
        float c;
        grid_error(p.errs, p.corrs, e, c);
        if (threadIdx.x == 0) {
            decide(ss, e);
            // the next sweep may use the previous row normaliser as its reference
            // only if no column moves by more than kFastPathLimit nats
            ss->exact_next = (c * static_cast<float>(ss->omega) > kFastPathLimit || ss->omega != 1.0) ? 1 : 0;
        }
    }
}

template <typename T, int EPT, int GR>
__global__ void __launch_bounds__(kRowsThreads, 1) rows_kernel(const __grid_constant__ RowsArgs p) {
    constexpr int V = Vec<T>::N;                // elements per 16 bytes
    constexpr int GT = kRowsThreads / GR;       // threads per stream
    constexpr int GW = GT / 32;
    constexpr int COVER = GT * EPT;             // columns a stream covers
    constexpr int NCH = EPT / 16;
    constexpr int H = EPT / 2;
    constexpr bool F32 = sizeof(T) == 4;
    constexpr bool DUMP = rows_dump_bytes(GR, EPT) > 0;
    constexpr uint32_t TCOLS = ColumnState<EPT>::kTmemColumns;
    static_assert(EPT <= 64, "column sums and duals of every thread fit the tensor memory");
    static_assert(COVER * sizeof(T) <= 64 * 1024, "a stage holds one row");
    extern __shared__ __align__(128) unsigned char ring[];
    float* dump = reinterpret_cast<float*>(ring + static_cast<size_t>(p.stages) * COVER * sizeof(T));  // DUMP
    __shared__ uint64_t full[kRowsMaxStages];
    __shared__ __align__(16) float red_s[GR][2][GW];
    __shared__ __align__(16) float red_m[GR][2][GW];
    __shared__ __align__(16) double colred[kRowsWarps][128];  // also where fewer than 8 streams meet
    __shared__ float a_s[kRowsMaxRows];
    __shared__ SolveState ss;
    __shared__ int newest[kRowsMaxStages];  // phase of the newest copy into a stage (-1: none)
    __shared__ uint32_t tmem_slot;

    if (*reinterpret_cast<volatile int*>(&p.st->done)) return;  // uniform: written by an earlier kernel

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = tid / GT, gt = tid % GT, gw = warp % GW;
    const int n = p.n;
    const int row_begin = blockIdx.x * p.rows_per_cta;
    const int nrows = max(0, min(n, row_begin + p.rows_per_cta) - row_begin);
    const int NST = p.stages;
    const float2 log2e2 = make_float2(kLog2e, kLog2e);

    // this CTA's copy of the solve state, row duals, barriers, finite stage memory
    // (columns past n_copy are never copied), tensor memory
    for (int k = tid; k < static_cast<int>(sizeof(SolveState) / 4); k += kRowsThreads)
        reinterpret_cast<int*>(&ss)[k] = reinterpret_cast<const int*>(p.st)[k];
    for (int i = tid; i < nrows; i += kRowsThreads) a_s[i] = p.a[row_begin + i];
    {
        const int tail = COVER - p.n_copy;
        for (int s = 0; s < NST; ++s) {
            T* row = reinterpret_cast<T*>(ring) + static_cast<size_t>(s) * COVER;
            for (int j = tid; j < tail; j += kRowsThreads) row[p.n_copy + j] = from_float<T>(0.f);
        }
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

    // Ring of whole rows.  Unit u (row u mod nrows of sweep u / nrows) sits in stage
    // u mod NST; the stream that consumed it refills the stage with unit u + NST, which
    // within a sweep is that stream's own (NST is a multiple of GR) and in a later sweep
    // is waited for only after a barrier of the whole CTA: no wait is ever more than one
    // phase ahead of its barrier.
    const int sweeps = min(p.sweeps, ss.max_it - ss.it);
    const int units = p.resident ? nrows : nrows * sweeps;  // at most 256 kRowsMaxSweeps
    const uint32_t row_bytes = static_cast<uint32_t>(p.n_copy) * sizeof(T);
    auto issue = [&](int row, int s, uint32_t phase, bool first) {
        const uint32_t unmet = (first && blockIdx.x == 0 && row == p.fault_row) ? 16u : 0u;
        newest[s] = static_cast<int>(phase);
        mbar_arrive_expect_tx(&full[s], row_bytes + unmet);
        bulk_load(ring + static_cast<size_t>(s) * COVER * sizeof(T),
                  static_cast<const T*>(p.L) +
                      static_cast<unsigned long long>(static_cast<unsigned>(row_begin + row)) *
                          static_cast<unsigned>(p.ld),
                  row_bytes, &full[s]);
    };
    if (tid == 0) {
        fence_proxy_async_smem();  // the fill above precedes the copies
        const int first = min(units, NST);
        for (int u = 0; u < first; ++u) issue(u % nrows, u, 0u, u < nrows);
    }
    int ubase = 0;  // units consumed by finished sweeps
    int sbase = 0;        // their stage and phase: unit ubase + r sits in stage (sbase + r) mod NST
    uint32_t phbase = 0u;
    const int ahead = NST % max(1, nrows);  // row of unit u + NST, from u's row

    // The duals of this thread's columns; up to 32 columns they are fetched while warp
    // 0 still takes the decision of the sweep before.
    constexpr bool PREFETCH = EPT <= 32;
    float4 b_raw[EPT / 4];
    auto column_of = [&](int e) { return ((e / V) * GT + gt) * V + e % V; };
    // duals of sweep t before scaling: b_prev - omega logcs, or b_next, which the sweep
    // before wrote for omega = 1
    auto load_duals = [&](int e, int t, bool next, float omega) -> float4 {
        const int j = column_of(e);
        if (j >= n) return make_float4(0.f, 0.f, 0.f, 0.f);  // the vectors are n_pad long, a multiple of 64
        if (next) return __ldcg(reinterpret_cast<const float4*>(p.b_next + j));
        const float4 bp = __ldcg(reinterpret_cast<const float4*>(p.b_buf + ((t - 1) & 1) * p.n_pad + j));
        const float4 lc = __ldcg(reinterpret_cast<const float4*>(p.logcs + j));
        return make_float4(bp.x - omega * lc.x, bp.y - omega * lc.y, bp.z - omega * lc.z, bp.w - omega * lc.w);
    };
    const bool plain = ss.momentum_start < 0;  // omega stays 1

    unsigned arrivals = ss.arrivals - ss.arrivals % gridDim.x;  // a first barrier may already be filling
    bool alive = true;
    for (int sw = 0; sw < sweeps; ++sw) {
        const int t = ss.it;
        const float omega = static_cast<float>(ss.omega);
        const bool momentum = omega != 1.0f;
        const bool exact_only = ss.exact_next != 0 || momentum;  // uniform
        // ---- column duals of this sweep: b = b_prev - w log(colsum_prev), kept as b log2 e;
        //      -inf past n, so those columns contribute exactly 0
        {
            const bool next = plain && sw > 0;
            float* b_out = p.b_buf + (t & 1) * p.n_pad;
            if (!PREFETCH) {
#pragma unroll
                for (int k = 0; k < EPT / 4; ++k) b_raw[k] = load_duals(4 * k, t, next, omega);
            }
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                float bb[16];
                if (PREFETCH && !next) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) b_raw[4 * c + k] = load_duals(16 * c + 4 * k, t, false, omega);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int j = column_of(16 * c + 4 * k);
                    const float4 b = b_raw[4 * c + k];
                    if (blockIdx.x == 0 && g == 0 && j < n) *reinterpret_cast<float4*>(b_out + j) = b;
                    const float b4[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                    for (int w = 0; w < 4; ++w) bb[4 * k + w] = j + w < n ? b4[w] * kLog2e : -INFINITY;
                }
                cols.set(c, bb);
            }
            cols.ready();
        }

        float2 y[H];     // exponentials of the stream's last row, not yet in the column sums
        float wp = 0.f;  // and its weight 1 / (row sum)
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
            const T* stage = reinterpret_cast<const T*>(ring) + static_cast<size_t>(s) * COVER;
            // a resident row is waited for once per launch
            bool ok = (p.resident && sw > 0) ||
                      mbar_wait<true>(&full[s], p.resident ? 0u : ph, &p.st->status, p.suspend_ns, p.wait_limit_ns);
            cols.settle();
            auto release = [&]() {
                // (every thread of the stream has read the stage before the barrier just passed)
                if (gt == 0 && ubase + r + NST < units) {
                    int row = r + ahead;
                    if (row >= nrows) row -= nrows;
                    fence_proxy_async_smem();  // the reads of the stage precede the copy into it
                    issue(row, s, ph ^ 1u, false);
                }
            };
            float anew = 0.f, wr = 0.f;
            bool fast_ok = false;
            if (!exact_only) {
                // ---- fast path: y = 2^(L log2e + b [+ a_old log2e]), against the absorbed frame
                //      (16-bit) or the previous row normaliser (FP32)
                float2 s2 = make_float2(0.f, 0.f), t2 = make_float2(0.f, 0.f);
                const float ref = F32 ? a_s[r] * kLog2e : 0.f;
                const float2 ref2 = make_float2(ref, ref);
#pragma unroll
                for (int c = 0; c < NCH; ++c) {
                    cols.add(c, y + 8 * c, wp);
                    float2 bb[8];
                    cols.duals(c, bb);
#pragma unroll
                    for (int i = 0; i < 16 / V; ++i) {
                        float2 v2[V / 2];
                        Pairs<T>::unpack(
                            *reinterpret_cast<const uint4*>(stage + ((c * (16 / V) + i) * GT + gt) * V), v2);
#pragma unroll
                        for (int h = 0; h < V / 2; ++h) {
                            const int q = i * (V / 2) + h;
                            float2 b2 = bb[q];
                            if (F32) b2 = __fadd2_rn(b2, ref2);
                            const float2 x = __ffma2_rn(v2[h], log2e2, b2);
                            const float2 e = ex2_pair(x);
                            y[8 * c + q] = e;
                            if (q & 1)
                                t2 = __fadd2_rn(t2, e);
                            else
                                s2 = __fadd2_rn(s2, e);
                        }
                    }
                }
                const float2 u2 = __fadd2_rn(s2, t2);
                const float part = warp_sum(u2.x + u2.y);
                if (lane == 0) red_s[g][par][gw] = part;
                if (!stream_and<GT>(ok, g)) {
                    alive = false;
                    break;
                }
                const float S = sum_warps<GW>(red_s[g][par]);
                fast_ok = S > 1e-30f && S < 1e30f;  // uniform over the stream
                if (fast_ok) {
                    release();
                    if (gt == GT - 32) anew = (F32 ? a_s[r] : 0.f) - __log2f(S) * kLn2;
                    wr = __frcp_rn(S);
                }
            }
            if (!fast_ok) {
                // ---- exact path: row maximum, then the exponentials relative to it (the previous
                //      row dual is read before the barriers that precede its update)
                const float a_old = momentum ? a_s[r] : 0.f;
                if (exact_only) {  // the pending row (the fast path above has already added it)
#pragma unroll
                    for (int c = 0; c < NCH; ++c) cols.add(c, y + 8 * c, wp);
                }
                float mx = -INFINITY;
#pragma unroll
                for (int c = 0; c < NCH; ++c) {
                    float2 bb[8];
                    cols.duals(c, bb);
                    float2 v2[8];
                    load16<T, GT>(stage, c, gt, v2);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float2 x = __ffma2_rn(v2[q], log2e2, bb[q]);
                        y[8 * c + q] = x;
                        mx = fmaxf(mx, fmaxf(x.x, x.y));
                    }
                }
                mx = warp_max(mx);
                if (lane == 0) red_m[g][par][gw] = mx;
                if (!stream_and<GT>(ok, g)) {
                    alive = false;
                    break;
                }
                float M2 = -INFINITY;
#pragma unroll
                for (int w = 0; w < GW; ++w) M2 = fmaxf(M2, red_m[g][par][w]);
                const float base = (M2 == -INFINITY) ? 0.f : M2;
                const float2 nb = make_float2(-base, -base);
                float2 ssum = make_float2(0.f, 0.f);
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    y[h] = ex2_pair(__fadd2_rn(y[h], nb));
                    ssum = __fadd2_rn(ssum, y[h]);
                }
                const float part = warp_sum(ssum.x + ssum.y);
                if (lane == 0) red_s[g][par][gw] = part;
                stream_and<GT>(true, g);
                release();
                const float S = sum_warps<GW>(red_s[g][par]);
                const float lse = (M2 + log2f(S)) * kLn2;
                anew = momentum ? (1.f - omega) * a_old - omega * lse : -lse;
                wr = (M2 == -INFINITY) ? 0.f : ex2(M2 + anew * kLog2e);
            }
            if (gt == GT - 32) {  // not the warp that refills the stage
                a_s[r] = anew;
                p.a[row_begin + r] = anew;
            }
            wp = wr;
            s_cur += GR;
            while (s_cur >= NST) {
                s_cur -= NST;
                ph ^= 1u;
            }
        }

        // ---- this CTA's column sums: the streams' sums (the pending rows included) meet in
        //      shared memory, so that the grid exchanges one row per CTA
        {
            float* prow = p.partials + static_cast<size_t>(blockIdx.x) * p.n_pad;
            float* mine = DUMP ? dump + static_cast<size_t>(g) * COVER : prow;
            cols.settle();
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                float acc[16];
                cols.total(c, y + 8 * c, wp, acc);
                if constexpr (GR > 1 && !DUMP) {
                    meet_streams<GR, GT, V>(reinterpret_cast<float*>(colred), acc, c, g, gt, n, prow);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int j = column_of(16 * c + 4 * k);
                        if (j < n)  // partial rows are n_pad wide, a multiple of 64 columns
                            *reinterpret_cast<float4*>(mine + j) =
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
                    for (int o = 1; o < GR; o <<= 1) {  // neighbours first
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
        if (!grid_barrier(&p.st->arrivals, &p.st->status, alive, arrivals, p.wait_limit_ns)) {  // the same in every thread of the CTA
            alive = false;
            break;
        }
        reduce_columns(p, t, colred);
        arrivals += gridDim.x;
        if (!grid_barrier(&p.st->arrivals, &p.st->status, true, arrivals, p.wait_limit_ns)) {
            alive = false;
            break;
        }
        if (PREFETCH && plain) {
#pragma unroll
            for (int k = 0; k < EPT / 4; ++k) b_raw[k] = load_duals(4 * k, t + 1, true, 1.f);
        }
        take_decision(p, &ss);
        ubase += nrows;
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

    // Copies may be in flight (stages refilled ahead, or a timed-out wait): wait for
    // the newest copy of every stage (bounded) before its shared memory is released;
    // one that never completes does not hide the others.
    __syncthreads();
    if (tid == 0) {
        for (int s = 0; s < NST; ++s)
            if (newest[s] >= 0)
                mbar_wait<true>(&full[s], static_cast<uint32_t>(newest[s]), &p.st->status, p.suspend_ns,
                                p.wait_limit_ns);
        if (!alive) {
            p.st->done = 1;
            p.st->final_it = ss.it;
            if (ss.check) {
                p.st->main_final_it = ss.it;
                p.st->main_n_err = ss.n_err;
            }
            p.st->it = ss.it + 1;
        }
    }
    if (alive && blockIdx.x == 0) {
        // write the state back (not the error word and the barrier, which the CTAs share)
        SolveState* st = p.st;
        if (tid == 0) {
            st->it = ss.it;
            st->done = ss.done;
            st->final_it = ss.final_it;
            st->n_err = ss.n_err;
            st->main_final_it = ss.main_final_it;
            st->main_n_err = ss.main_n_err;
            st->polish_count = ss.polish_count;
            st->exact_next = ss.exact_next;
            st->omega = ss.omega;
            st->last_err = ss.last_err;
            st->main_last_err = ss.main_last_err;
            st->polish_err = ss.polish_err;
        }
        for (int k = tid; k < min(ss.n_err, FUGAL_MAX_RECORDED_ERRORS); k += kRowsThreads) st->errors[k] = ss.errors[k];
    }
    if constexpr (TCOLS > 0) {
        tmem_fence_before_sync();
        __syncthreads();
        tmem_fence_after_sync();
        if (warp == 0) tmem_dealloc(tmem_slot, TCOLS);
    }
}

namespace {

using RowsFn = void (*)(const RowsArgs);

template <typename T>
RowsFn rows_fn(int ept, int streams) {
    switch (streams * 100 + ept) {
        case 816: return rows_kernel<T, 16, 8>;
        case 832: return rows_kernel<T, 32, 8>;
        case 432: return rows_kernel<T, 32, 4>;
        case 448: return rows_kernel<T, 48, 4>;
    }
    if constexpr (sizeof(T) == 2) {
        switch (streams * 100 + ept) {
            case 464: return rows_kernel<T, 64, 4>;
            case 248: return rows_kernel<T, 48, 2>;
            case 264: return rows_kernel<T, 64, 2>;
            default: return rows_kernel<T, 48, 1>;
        }
    } else {
        return rows_kernel<T, 32, 2>;
    }
}

RowsFn rows_fn(const RowsPlan& pl) {
    if (pl.dt == FUGAL_F32) return rows_fn<float>(pl.ept, pl.streams);
    return pl.dt == FUGAL_BF16 ? rows_fn<__nv_bfloat16>(pl.ept, pl.streams) : rows_fn<__half>(pl.ept, pl.streams);
}

// (streams, columns per thread) in the order of the columns they cover,
// 512 / streams * ept: the narrowest that covers n.  Measured per iteration: BF16 at
// n = 8192 41.1 us as {4, 64}, 51.2 as {2, 32}; n = 6000 28.2 as {4, 48}, 39.1 as
// {2, 32}; n = 4096 18.6 as {4, 32}, 25.5 as {8, 64}.  FP32 rows of 6145 to 8192
// columns take two streams, so that two stages of 32 KB are left for each.  Wider
// rows: FP32 sweeps stay with the cluster kernel (an iteration takes 107 us at n = 8193, 145 at
// 12000, 190 at 16384, 800 at 32768: 38, 61, 87 and 82% of the copy peak); 16-bit ones of
// more than 24576 columns have too few stages left here (469 against 454 us at 32768).
struct RowsShape {
    int streams, ept;
};
constexpr RowsShape kShapes16[] = {{8, 16}, {8, 32}, {4, 32}, {4, 48}, {4, 64}, {2, 48}, {2, 64}, {1, 48}};
constexpr RowsShape kShapes32[] = {{8, 16}, {8, 32}, {4, 32}, {4, 48}, {2, 32}};

RowsShape rows_shape(int64_t n, int dt) {
    auto covers = [n](const RowsShape& sh) { return static_cast<int64_t>(kRowsThreads / sh.streams) * sh.ept >= n; };
    if (dt == FUGAL_F32) {
        for (const RowsShape& sh : kShapes32)
            if (covers(sh)) return sh;
    } else {
        for (const RowsShape& sh : kShapes16)
            if (covers(sh)) return sh;
    }
    return RowsShape{0, 0};
}

}  // namespace

fugal_status make_rows_plan(int64_t n, int dt, RowsPlan& pl, bool device) {
    pl = RowsPlan{};
    pl.dt = dt;
    const int es = dt == FUGAL_F32 ? 4 : 2;
    const RowsShape shape = rows_shape(n, dt);
    if (shape.streams == 0) return FUGAL_OK;
    pl.streams = shape.streams;
    pl.ept = shape.ept;
    const int sms = sm_count();
    const int want = static_cast<int>(std::min<int64_t>(sms, n));
    pl.rows_per_cta = static_cast<int>((n + want - 1) / want);
    if (pl.rows_per_cta > kRowsMaxRows) return FUGAL_OK;
    pl.ctas = static_cast<int>((n + pl.rows_per_cta - 1) / pl.rows_per_cta);
    const size_t stage = static_cast<size_t>(kRowsThreads / pl.streams) * pl.ept * es;
    const size_t dump = rows_dump_bytes(pl.streams, pl.ept);
    const size_t room = 227 * 1024 - kRowsStatic - dump;
    pl.stages = static_cast<int>(std::min<size_t>({room / stage, static_cast<size_t>(kRowsMaxStages),
                                                   static_cast<size_t>(pl.rows_per_cta)}));
    pl.resident = pl.stages >= pl.rows_per_cta;
    // A stage that is refilled within a sweep has to go back to the stream that emptied
    // it: a stream waiting for a copy two phases ahead of the stage's barrier would take
    // the phase before as its own (mbarrier waits see one parity bit).
    if (!pl.resident) pl.stages -= pl.stages % pl.streams;
    if (pl.stages < 1) return FUGAL_OK;
    pl.smem = stage * pl.stages + dump;
    if (device) {
        int dev = 0, coop = 0, blocks = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return FUGAL_OK;
        RowsFn fn = rows_fn(pl);
        FUGAL_TRY(allow_dynamic_smem(fn, pl.smem, "sinkhorn rows: shared memory"));
        FUGAL_TRY(cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, kRowsThreads, pl.smem),
                             "sinkhorn rows: occupancy"));
        if (blocks < 1) return FUGAL_OK;
    }
    pl.use = true;
    return FUGAL_OK;
}

fugal_status launch_rows(const RowsPlan& pl, RowsArgs args, cudaStream_t stream, int family) {
    args.rows_per_cta = pl.rows_per_cta;
    args.stages = pl.stages;
    args.resident = pl.resident;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(pl.ctas, 1, 1);
    cfg.blockDim = dim3(kRowsThreads, 1, 1);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LaunchScope scope(family, stream);
    return cuda_check(cudaLaunchKernelEx(&cfg, rows_fn(pl), args), "sinkhorn rows: launch");
}

}  // namespace fugal
