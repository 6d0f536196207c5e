// Exact linear assignment on the device, with the same mapping as
// scipy.optimize.linear_sum_assignment (the reference's HungarianMethod.SCIPY,
// cugal/pred.py:151-158; scipy 1.18.1 here).
//
// scipy solves the assignment with the shortest-augmenting-path method of
// D. F. Crouse, "On implementing 2D rectangular assignment algorithms", IEEE
// TAES 52(4), 2016: rows are added one at a time; for each, a Dijkstra search
// over reduced costs  minVal + c_ij - u_i - v_j  finds the cheapest path to a
// free column, then the duals u, v are updated and the path is augmented.  For
// the mapping to be identical to scipy's -- including which optimum it returns
// when several exist -- this kernel reproduces scipy's choices exactly:
//
//   * maximize: c = -P (the FP32 P converted to double first);
//   * the candidate columns are kept in a list that starts in descending column
//     order and loses the selected column by "swap with the last entry";
//   * each step selects the minimum shortest-path cost; among equal minima the
//     first one in list order, unless a later equal one is an unassigned
//     column, in which case the last such unassigned column;
//   * all arithmetic in double, in scipy's operation order (additions and
//     subtractions only, each rounded on its own).
//
// One CTA runs the outer loop over rows; each Dijkstra step scans the
// remaining columns with all its threads and reduces (cost, tie priority).  A cap on
// the total number of Dijkstra steps bounds the run time; hitting it is reported in
// the status word.
//
// Two kernels.  Up to 8192 columns (exact_lap_owned_kernel) every thread owns up to 8
// columns: their shortest-path costs, list positions and assigned rows are registers,
// the duals and the rest of the state shared memory, and a step is one coalesced read
// of a row of P, warp reductions on the cost's ordered bits and one barrier.  Above
// (exact_lap_kernel) the list and the per-column arrays are in global memory; the list
// order is restored after every row from an undo log, and shortest-path costs are
// invalidated by a row stamp.  Bound by latency (the next row is known only after the
// reduction): per step at n = 4096 2.7 us with the arrays in global memory, 1.4 us
// owned.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fugal_common.cuh"
#include "fugal_host.h"

namespace fugal {

constexpr int kExactThreads = 1024;

struct ExactWs {
    double* u;
    double* v;
    double* spc;    // shortest-path cost per column (valid when stamp == current row)
    int* stamp;
    int* path;
    int* col4row;
    int* row4col;
    int* remaining;
    int* sr_list;   // rows reached in the current search
    int* sc_list;   // columns reached (= removed from the list) in the current search
    int* undo_idx;  // list positions overwritten by those removals
    int* bad;       // count of invalid entries (NaN, or -inf cost)
    size_t bytes;
};

ExactWs exact_layout(int64_t n, char* base) {
    ExactWs w{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off = (off + bytes + 255) / 256 * 256;
        return p;
    };
    w.u = reinterpret_cast<double*>(take(n * 8));
    w.v = reinterpret_cast<double*>(take(n * 8));
    w.spc = reinterpret_cast<double*>(take(n * 8));
    w.stamp = reinterpret_cast<int*>(take(n * 4));
    w.path = reinterpret_cast<int*>(take(n * 4));
    w.col4row = reinterpret_cast<int*>(take(n * 4));
    w.row4col = reinterpret_cast<int*>(take(n * 4));
    w.remaining = reinterpret_cast<int*>(take(n * 4));
    w.sr_list = reinterpret_cast<int*>(take(n * 4));
    w.sc_list = reinterpret_cast<int*>(take(n * 4));
    w.undo_idx = reinterpret_cast<int*>(take(n * 4));
    w.bad = reinterpret_cast<int*>(take(4));
    w.bytes = off;
    return w;
}

// Invalid entries for scipy: NaN anywhere, or a cost of -inf (P = +inf when maximizing).
__global__ void exact_check_kernel(const float* __restrict__ P, long long ldp, int n, int maximize, int* bad) {
    int cnt = 0;
    for (int r = blockIdx.y; r < n; r += gridDim.y) {
        const float* row = P + static_cast<size_t>(r) * ldp;
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
            const float c = maximize ? -row[j] : row[j];
            if (c != c || c == -INFINITY) ++cnt;
        }
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(bad, cnt);
}

__global__ void exact_init_kernel(ExactWs w, int n) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        w.u[j] = 0.0;
        w.v[j] = 0.0;
        w.stamp[j] = -1;
        w.path[j] = -1;
        w.col4row[j] = -1;
        w.row4col[j] = -1;
        w.remaining[j] = n - 1 - j;  // descending column order, as scipy fills it
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *w.bad = 0;
}

// Selection key of a column in one Dijkstra step: smaller cost wins; among equal
// costs an unassigned column beats an assigned one, unassigned columns later in
// the list beat earlier ones and assigned columns earlier in the list beat later
// ones.  `prio` encodes that tie order (larger wins) and the list position.
struct Pick {
    double cost;
    int prio;
};
constexpr int kPrioBase = 1 << 30;
__device__ __forceinline__ int pick_prio(int pos, bool unassigned) {
    return unassigned ? kPrioBase + pos : kPrioBase - 1 - pos;
}
__device__ __forceinline__ int prio_pos(int prio) { return prio >= kPrioBase ? prio - kPrioBase : kPrioBase - 1 - prio; }
__device__ __forceinline__ Pick pick_better(Pick a, Pick b) {
    return (a.cost < b.cost || (a.cost == b.cost && a.prio > b.prio)) ? a : b;
}
__device__ __forceinline__ Pick pick_warp(Pick a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Pick b;
        b.cost = __shfl_xor_sync(0xffffffffu, a.cost, o);
        b.prio = __shfl_xor_sync(0xffffffffu, a.prio, o);
        a = pick_better(a, b);
    }
    return a;
}

__global__ void __launch_bounds__(kExactThreads) exact_lap_kernel(const float* __restrict__ P, long long ldp, int n,
                                                                  int maximize, long long max_steps, ExactWs w,
                                                                  long long* columns_out, long long* steps_out,
                                                                  int* status_out) {
    __shared__ Pick warp_best[kExactThreads / 32];
    __shared__ int s_i, s_sink, s_num, s_nsr, s_nsc, s_stop;
    __shared__ double s_min;
    __shared__ long long s_steps;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (*w.bad != 0) {
        if (tid == 0) {
            *status_out = FUGAL_NONFINITE;
            if (steps_out) *steps_out = 0;
        }
        return;
    }
    if (tid == 0) {
        s_steps = 0;
        s_stop = 0;
    }
    for (int cur = 0; cur < n; ++cur) {
        if (tid == 0) {
            s_i = cur;
            s_min = 0.0;
            s_sink = -1;
            s_num = n;
            s_nsr = 1;
            w.sr_list[0] = cur;
            s_nsc = 0;
        }
        __syncthreads();
        // ---- shortest augmenting path from row `cur`
        while (true) {
            const int i = s_i;
            const double min_val = s_min;
            const int num = s_num;
            const double ui = w.u[i];
            const float* prow = P + static_cast<size_t>(i) * ldp;
            Pick best{INFINITY, -1};
            for (int it = tid; it < num; it += kExactThreads) {
                const int j = w.remaining[it];
                const double p = static_cast<double>(prow[j]);
                const double c = maximize ? -p : p;
                const double r = __dsub_rn(__dsub_rn(__dadd_rn(min_val, c), ui), w.v[j]);
                double sp = (w.stamp[j] == cur) ? w.spc[j] : INFINITY;
                if (r < sp) {
                    w.path[j] = i;
                    w.spc[j] = r;
                    w.stamp[j] = cur;
                    sp = r;
                }
                best = pick_better(best, Pick{sp, pick_prio(it, w.row4col[j] < 0)});
            }
            best = pick_warp(best);
            if (lane == 0) warp_best[warp] = best;
            __syncthreads();
            if (warp == 0) {
                Pick b = warp_best[lane];
                b = pick_warp(b);
                if (lane == 0) {
                    const long long steps = ++s_steps;
                    if (b.cost == INFINITY || b.prio < 0) {
                        *status_out = FUGAL_BAD_ARGUMENT;  // infeasible: every remaining cost is +inf
                        s_stop = 1;
                    } else if (steps > max_steps) {
                        *status_out = FUGAL_ITER_LIMIT;
                        s_stop = 1;
                    } else {
                        const int idx = prio_pos(b.prio);
                        const int j = w.remaining[idx];
                        s_min = b.cost;
                        if (w.row4col[j] < 0) {
                            s_sink = j;
                        } else {
                            s_i = w.row4col[j];
                            w.sr_list[s_nsr++] = s_i;
                        }
                        w.undo_idx[s_nsc] = idx;
                        w.sc_list[s_nsc++] = j;
                        w.remaining[idx] = w.remaining[num - 1];
                        s_num = num - 1;
                    }
                }
            }
            __syncthreads();
            if (s_sink >= 0 || s_stop) break;
        }
        if (s_stop) break;
        // ---- duals (scipy: u[cur] += minVal; u[i] += minVal - spc[col4row[i]]; v[j] -= minVal - spc[j])
        const double min_val = s_min;
        for (int k = tid; k < s_nsr; k += kExactThreads) {
            const int i2 = w.sr_list[k];
            if (i2 == cur)
                w.u[i2] = __dadd_rn(w.u[i2], min_val);
            else
                w.u[i2] = __dadd_rn(w.u[i2], __dsub_rn(min_val, w.spc[w.col4row[i2]]));
        }
        for (int k = tid; k < s_nsc; k += kExactThreads) {
            const int j2 = w.sc_list[k];
            w.v[j2] = __dsub_rn(w.v[j2], __dsub_rn(min_val, w.spc[j2]));
        }
        __syncthreads();
        if (tid == 0) {
            // augment along the path
            int j = s_sink;
            while (true) {
                const int i2 = w.path[j];
                w.row4col[j] = i2;
                const int t = w.col4row[i2];
                w.col4row[i2] = j;
                j = t;
                if (i2 == cur) break;
            }
            // restore the candidate list to its state at the start of the row
            for (int k = s_nsc - 1; k >= 0; --k) w.remaining[w.undo_idx[k]] = w.sc_list[k];
        }
        __syncthreads();
    }
    if (s_stop) {
        if (tid == 0 && steps_out) *steps_out = s_steps;
        return;
    }
    for (int r = tid; r < n; r += kExactThreads) columns_out[r] = w.col4row[r];
    if (tid == 0) {
        *status_out = FUGAL_OK;
        if (steps_out) *steps_out = s_steps;
    }
}

// ---------------------------------------------------------------- owned columns

constexpr int kOwnedMaxN = 8192;
constexpr int kPathLog = 1024;  // rows of a search kept in shared memory (the rest in global)
constexpr int kNoRow = 0xffff;

// Order of doubles as unsigned integers, -0 and +0 alike (no NaN).
__device__ __forceinline__ unsigned long long ordered_bits(double x) {
    const long long b = __double_as_longlong(__dadd_rn(x, 0.0));
    return static_cast<unsigned long long>(b < 0 ? ~b : (b ^ static_cast<long long>(0x8000000000000000ull)));
}
__device__ __forceinline__ double from_ordered(unsigned long long k) {
    const long long b = static_cast<long long>(k);
    return __longlong_as_double(b < 0 ? (b ^ static_cast<long long>(0x8000000000000000ull)) : ~b);
}

struct OwnedPick {
    unsigned hi, lo;  // ordered_bits of the cost; all ones: no column
    int prio;         // -1: no column
    int column;
    int row;          // row assigned to the column (kNoRow: none)
};

// The best of the warp's picks (smallest cost, then largest priority), in every lane.
__device__ __forceinline__ OwnedPick best_of_warp(const OwnedPick& p) {
    OwnedPick b;
    b.hi = __reduce_min_sync(0xffffffffu, p.hi);
    b.lo = __reduce_min_sync(0xffffffffu, p.hi == b.hi ? p.lo : 0xffffffffu);
    const bool cheapest = p.hi == b.hi && p.lo == b.lo;
    b.prio = __reduce_max_sync(0xffffffffu, cheapest ? p.prio : -1);
    const int src = __ffs(__ballot_sync(0xffffffffu, cheapest && p.prio == b.prio)) - 1;
    b.column = __shfl_sync(0xffffffffu, p.column, src);
    b.row = __shfl_sync(0xffffffffu, p.row, src);
    return b;
}

size_t owned_smem(int64_t n) { return static_cast<size_t>(n) * (2 * 8 + 3 * 2) + 16; }

// Thread t owns columns t, t + 1024, ... (CPT of them).  A column's list position
// starts at n - 1 - j (descending order) in every search; "swap with the last entry"
// moves the column whose position is the last, which its owner sees by itself.
template <int CPT>
__global__ void __launch_bounds__(kExactThreads) exact_lap_owned_kernel(const float* __restrict__ P, long long ldp,
                                                                        int n, int maximize, long long max_steps,
                                                                        ExactWs w, long long* columns_out,
                                                                        long long* steps_out, int* status_out) {
    extern __shared__ __align__(16) unsigned char lap_smem[];
    double* v_s = reinterpret_cast<double*>(lap_smem);
    double* u_s = v_s + n;
    unsigned short* path_s = reinterpret_cast<unsigned short*>(u_s + n);
    unsigned short* row4col_s = path_s + n;
    unsigned short* col4row_s = row4col_s + n;
    __shared__ OwnedPick picks[2][kExactThreads / 32];
    __shared__ int log_row[kPathLog];
    __shared__ double log_cost[kPathLog];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (*w.bad != 0) {
        if (tid == 0) {
            *status_out = FUGAL_NONFINITE;
            if (steps_out) *steps_out = 0;
        }
        return;
    }
    for (int j = tid; j < n; j += kExactThreads) {
        v_s[j] = u_s[j] = 0.0;
        row4col_s[j] = col4row_s[j] = kNoRow;
    }
    __syncthreads();
    double spc[CPT];
    int pos[CPT];  // list position; -1: not a column; -2: reached in this search
    int row[CPT];  // row assigned to the column
    float pv[CPT]; // this step's row of P
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        const int j = tid + k * kExactThreads;
        row[k] = kNoRow;
        pv[k] = j < n ? P[j] : 0.f;
    }
    long long steps = 0;
    int par = 0;
    int failure = FUGAL_OK;
    for (int cur = 0; cur < n && failure == FUGAL_OK; ++cur) {
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int j = tid + k * kExactThreads;
            spc[k] = INFINITY;
            pos[k] = j < n ? n - 1 - j : -1;
        }
        int i = cur, num = n, reached = 0, sink = -1;
        double min_val = 0.0;
        // ---- shortest augmenting path from row `cur`
        while (true) {
            const double ui = u_s[i];
            OwnedPick mine{0xffffffffu, 0xffffffffu, -1, 0, kNoRow};
            double best = INFINITY;
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                if (pos[k] < 0) continue;
                const int j = tid + k * kExactThreads;
                const double p = static_cast<double>(pv[k]);
                const double c = maximize ? -p : p;
                const double r = __dsub_rn(__dsub_rn(__dadd_rn(min_val, c), ui), v_s[j]);
                if (r < spc[k]) {
                    spc[k] = r;
                    path_s[j] = static_cast<unsigned short>(i);
                }
                const int prio = pick_prio(pos[k], row[k] == kNoRow);
                if (mine.prio < 0 || spc[k] < best || (spc[k] == best && prio > mine.prio)) {
                    best = spc[k];
                    mine.prio = prio;
                    mine.column = j;
                    mine.row = row[k];
                }
            }
            if (mine.prio >= 0) {
                const unsigned long long key = ordered_bits(best);
                mine.hi = static_cast<unsigned>(key >> 32);
                mine.lo = static_cast<unsigned>(key);
            }
            const OwnedPick wb = best_of_warp(mine);
            if (lane == 0) picks[par][warp] = wb;
            __syncthreads();
            const OwnedPick b = best_of_warp(picks[par][lane]);
            par ^= 1;  // a warp is at most one step ahead of another: two buffers suffice
            const double cost = from_ordered((static_cast<unsigned long long>(b.hi) << 32) | b.lo);
            ++steps;
            if (b.prio < 0 || cost == INFINITY) {
                failure = FUGAL_BAD_ARGUMENT;  // infeasible: every remaining cost is +inf
                break;
            }
            if (steps > max_steps) {
                failure = FUGAL_ITER_LIMIT;
                break;
            }
            const int idx = prio_pos(b.prio);
            --num;
            min_val = cost;
            if (b.row == kNoRow) {
                sink = b.column;
            } else {
                i = b.row;
                // the next row, needed first thing in the next step
                const float* prow = P + static_cast<size_t>(i) * ldp;
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    const int j = tid + k * kExactThreads;
                    if (j < n) pv[k] = prow[j];
                }
                if (tid == 0) {
                    if (reached < kPathLog) {
                        log_row[reached] = i;
                        log_cost[reached] = cost;
                    } else {
                        w.sr_list[reached] = i;
                        w.spc[reached] = cost;
                    }
                }
                ++reached;
            }
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                if (tid + k * kExactThreads == b.column) pos[k] = -2;
                else if (pos[k] == num) pos[k] = idx;
            }
            if (sink >= 0) break;
        }
        if (failure != FUGAL_OK) break;
        // the next search's first row
        if (cur + 1 < n) {
            const float* prow = P + static_cast<size_t>(cur + 1) * ldp;
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                const int j = tid + k * kExactThreads;
                if (j < n) pv[k] = prow[j];
            }
        }
        // ---- duals (scipy: u[cur] += minVal; u[i] += minVal - spc[col4row[i]]; v[j] -= minVal - spc[j])
#pragma unroll
        for (int k = 0; k < CPT; ++k)
            if (pos[k] == -2) {
                const int j = tid + k * kExactThreads;
                v_s[j] = __dsub_rn(v_s[j], __dsub_rn(min_val, spc[k]));
            }
        __syncthreads();  // the log, the paths and every read of u are complete
        for (int s = tid; s < reached; s += kExactThreads) {
            const int i2 = s < kPathLog ? log_row[s] : w.sr_list[s];
            const double c2 = s < kPathLog ? log_cost[s] : w.spc[s];
            u_s[i2] = __dadd_rn(u_s[i2], __dsub_rn(min_val, c2));
        }
        if (tid == 0) {
            u_s[cur] = __dadd_rn(u_s[cur], min_val);
            int j = sink;
            while (true) {  // augment along the path
                const int i2 = path_s[j];
                row4col_s[j] = static_cast<unsigned short>(i2);
                const int t = col4row_s[i2];
                col4row_s[i2] = static_cast<unsigned short>(j);
                j = t;
                if (i2 == cur) break;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int j = tid + k * kExactThreads;
            if (j < n) row[k] = row4col_s[j];
        }
    }
    if (failure == FUGAL_OK)
        for (int r = tid; r < n; r += kExactThreads) columns_out[r] = col4row_s[r];
    if (tid == 0) {
        *status_out = failure;
        if (steps_out) *steps_out = steps;
    }
}

using OwnedFn = void (*)(const float*, long long, int, int, long long, ExactWs, long long*, long long*, int*);
OwnedFn owned_kernel(int64_t n) {
    if (n <= 1024) return exact_lap_owned_kernel<1>;
    if (n <= 2048) return exact_lap_owned_kernel<2>;
    if (n <= 4096) return exact_lap_owned_kernel<4>;
    return exact_lap_owned_kernel<8>;
}

}  // namespace fugal

using namespace fugal;

extern "C" fugal_status fugal_exact_lap_workspace_size(int64_t n, size_t* bytes) {
    if (bytes == nullptr) return fail(FUGAL_BAD_ARGUMENT, "fugal_exact_lap_workspace_size: null output");
    if (n <= 0 || n >= (1 << 30)) return fail(FUGAL_BAD_SHAPE, "fugal_exact_lap_workspace_size: bad n");
    *bytes = exact_layout(n, nullptr).bytes;
    return FUGAL_OK;
}

extern "C" fugal_status fugal_exact_lap(const float* P, int64_t ldp, int64_t n, int maximize, int64_t max_steps,
                                        int64_t* columns_out, int64_t* steps_out, int32_t* status_out,
                                        void* workspace, size_t workspace_bytes, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    size_t need = 0;
    FUGAL_TRY(fugal_exact_lap_workspace_size(n, &need));
    if (P == nullptr || columns_out == nullptr || status_out == nullptr || workspace == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_exact_lap: null argument");
    if (ldp < n) return fail(FUGAL_BAD_SHAPE, "fugal_exact_lap: ldp < n");
    if (max_steps <= 0) return fail(FUGAL_BAD_ARGUMENT, "fugal_exact_lap: max_steps must be positive");
    if (workspace_bytes < need)
        return fail(FUGAL_WORKSPACE_TOO_SMALL, "fugal_exact_lap: workspace %zu < %zu", workspace_bytes, need);
    ExactWs w = exact_layout(n, static_cast<char*>(workspace));
    const int nn = static_cast<int>(n);
    const int blocks = static_cast<int>(std::min<int64_t>((n + 255) / 256, 4 * sm_count()));
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        exact_init_kernel<<<blocks, 256, 0, stream>>>(w, nn);
        FUGAL_TRY(launch_check("fugal_exact_lap: init"));
    }
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        dim3 grid(static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 8)),
                  static_cast<unsigned>(std::min<int64_t>(n, 4 * sm_count())));
        exact_check_kernel<<<grid, 256, 0, stream>>>(P, ldp, nn, maximize ? 1 : 0, w.bad);
        FUGAL_TRY(launch_check("fugal_exact_lap: check"));
    }
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        long long* cols = reinterpret_cast<long long*>(columns_out);
        long long* steps = reinterpret_cast<long long*>(steps_out);
        if (n <= kOwnedMaxN) {
            OwnedFn fn = owned_kernel(n);
            const size_t smem = owned_smem(n);
            FUGAL_TRY(allow_dynamic_smem(fn, smem, "fugal_exact_lap: shared memory"));
            fn<<<1, kExactThreads, smem, stream>>>(P, ldp, nn, maximize ? 1 : 0, max_steps, w, cols, steps, status_out);
        } else {
            exact_lap_kernel<<<1, kExactThreads, 0, stream>>>(P, ldp, nn, maximize ? 1 : 0, max_steps, w, cols, steps,
                                                              status_out);
        }
        FUGAL_TRY(launch_check("fugal_exact_lap: solve"));
    }
    return FUGAL_OK;
}
