// Frank-Wolfe update and the reference-compatible elementwise / row kernels:
//   fugal_fw_update                    cugal/pred.py:133-141 on the absorbed cost
//   fugal_update_quasi_permutation_log cuda_kernels/update_quasi_permutation.cu:7-56
//   fugal_regularize                   cuda_kernels/regularize.cu:10-39
//   fugal_add_distance                 cuda_kernels/distance.cu:11-53
//   fugal_sinkhorn_log_step            cuda_kernels/sinkhorn_log.cu:8-66,100-114
//   fugal_sinkhorn_log_marginal        cuda_kernels/sinkhorn_log.cu:68-98
//   fugal_count_le                     cugal/pred.py:152-153
//   fugal_absorb_cost                  cugal/sinkhorn.py:98 and the duals folded in
// All reductions accumulate in FP64 and land in a caller-owned device double.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <initializer_list>

#include "fugal_common.cuh"
#include "fugal_host.h"

namespace fugal {

constexpr int kEwThreads = 256;

// Where the update records the plan's nonzero entries (fugal_fw_update_collect):
// per row k, counts[k] entries (column, q) at entries[k * slots ...] in no
// particular order (counts zeroed before the kernel; entries past `slots` are
// counted, not stored; the scatter checks counts and row sums).
struct PlanOut {
    int* counts;
    fugal_plan_entry* entries;
    int slots;
};

// q = exp(L + u_i + v_j); P += alpha (q - P); gap += (q - P) * (-reg (L - U_i - V_j)).
// Rows grid-strided over the blocks, each row's columns in chunks of 1024 (one
// float4 per thread per chunk); every block reduces its gap once at the end (one
// FP64 atomic per block).  EMIT: each q > 0 also takes a slot of its row through
// a global atomic on the row's count (a few per row, no barrier).
template <bool EMIT>
__global__ void __launch_bounds__(kEwThreads) fw_update_kernel(float* __restrict__ P, long long ldp,
                                                               const float* __restrict__ L, long long ldl,
                                                               const float* __restrict__ u,
                                                               const float* __restrict__ v,
                                                               const double* __restrict__ U,
                                                               const double* __restrict__ V, int n, float alpha,
                                                               double reg, double* gap, PlanOut plan) {
    __shared__ double red[32];
    constexpr int kChunk = kEwThreads * 4;
    double g = 0.0;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
      const float ui = u[i];
      const double Ui = U ? U[i] : 0.0;
      float* prow = P + static_cast<size_t>(i) * ldp;
    const float* lrow = L + static_cast<size_t>(i) * ldl;
      fugal_plan_entry* slots = EMIT ? plan.entries + static_cast<size_t>(i) * plan.slots : nullptr;
      auto record = [&](int j, float qv) {
          if constexpr (EMIT) {
              if (qv > 0.f) {
                  const int s = atomicAdd(&plan.counts[i], 1);
                  if (s < plan.slots) slots[s] = fugal_plan_entry{j, qv};
              }
          }
      };
      for (int j0 = threadIdx.x * 4; j0 < n; j0 += kChunk) {
        if (j0 + 4 <= n) {
            const float4 l4 = *reinterpret_cast<const float4*>(lrow + j0);
            float4 p4 = *reinterpret_cast<float4*>(prow + j0);
            const float4 v4 = *reinterpret_cast<const float4*>(v + j0);
            const float lv[4] = {l4.x, l4.y, l4.z, l4.w};
            const float vv[4] = {v4.x, v4.y, v4.z, v4.w};
            float pv[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float qv = expf(lv[q] + ui + vv[q]);
                const float diff = qv - pv[q];
                const double C = -reg * (static_cast<double>(lv[q]) - Ui - (V ? V[j0 + q] : 0.0));
                g += static_cast<double>(diff) * C;
                pv[q] = fmaf(alpha, diff, pv[q]);
                record(j0 + q, qv);
            }
            p4 = make_float4(pv[0], pv[1], pv[2], pv[3]);
            *reinterpret_cast<float4*>(prow + j0) = p4;
        } else {
            for (int j = j0; j < n; ++j) {
                const float qv = expf(lrow[j] + ui + v[j]);
                const float diff = qv - prow[j];
                const double C = -reg * (static_cast<double>(lrow[j]) - Ui - (V ? V[j] : 0.0));
                g += static_cast<double>(diff) * C;
                prow[j] = fmaf(alpha, diff, prow[j]);
                record(j, qv);
            }
        }
      }
    }
    g = block_sum(g, red);
    if (threadIdx.x == 0) atomicAdd(gap, g);
}

__global__ void commit_duals_kernel(const float* u, const float* v, double* U, double* V, int n) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        U[j] += static_cast<double>(u[j]);
        V[j] += static_cast<double>(v[j]);
    }
}

// The reference-compatible elementwise kernels walk rows grid-strided, a thread
// taking 4 consecutive columns with one 16-byte access each (VEC: aligned rows of
// whole quads), else one column per access (coalesced either way).  With 4 scalar
// accesses of stride 16 bytes per thread and one block per 1024 columns they ran at
// 23 to 70% of the copy peak at n = 8192 (update 177 us, regularize 326, distance 544).
constexpr int kEwCols = kEwThreads * 4;
inline dim3 ew_blocks(int64_t n) {
    const int64_t chunks = (n + kEwCols - 1) / kEwCols;
    const int64_t rows = std::max<int64_t>(1, std::min<int64_t>(n, (static_cast<int64_t>(sm_count()) * 32) / chunks));
    return dim3(static_cast<unsigned>(chunks), static_cast<unsigned>(rows));
}
// Column q (of 4) of this thread, and the access to its four columns of a row.
template <bool VEC>
FUGAL_DEVICE int ew_column(int q) {
    return VEC ? static_cast<int>(blockIdx.x) * kEwCols + static_cast<int>(threadIdx.x) * 4 + q
               : static_cast<int>(blockIdx.x) * kEwCols + q * kEwThreads + static_cast<int>(threadIdx.x);
}
template <bool VEC>
FUGAL_DEVICE void ew_load(const float* row, int n, float (&v)[4]) {
    if (VEC) {
        const int c = ew_column<true>(0);
        const float4 x = c < n ? *reinterpret_cast<const float4*>(row + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = ew_column<false>(q);
            v[q] = c < n ? row[c] : 0.f;
        }
    }
}
template <bool VEC>
FUGAL_DEVICE void ew_store(float* row, int n, const float (&v)[4]) {
    if (VEC) {
        const int c = ew_column<true>(0);
        if (c < n) *reinterpret_cast<float4*>(row + c) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = ew_column<false>(q);
            if (c < n) row[c] = v[q];
        }
    }
}

// Reference form: scaled = exp(K + v_c + u_r); gap += (scaled - P)(K * -reg); P += (scaled - P) alpha.
template <bool VEC>
__global__ void __launch_bounds__(kEwThreads) update_log_kernel(float* __restrict__ P, long long ldp,
                                                                const float* __restrict__ K, long long ldk,
                                                                const float* __restrict__ u,
                                                                const float* __restrict__ v, int n, float alpha,
                                                                float reg, double* gap) {
    __shared__ double red[32];
    double g = 0.0;
    float vv[4];
    ew_load<VEC>(v, n, vv);
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        float k[4], p[4];
        ew_load<VEC>(K + static_cast<size_t>(i) * ldk, n, k);
        ew_load<VEC>(P + static_cast<size_t>(i) * ldp, n, p);
        const float ui = u[i];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (ew_column<VEC>(q) >= n) continue;
            const float scaled = expf(k[q] + vv[q] + ui);
            const float diff = scaled - p[q];
            g += static_cast<double>(diff) * static_cast<double>(k[q] * -reg);
            p[q] = __fadd_rn(p[q], __fmul_rn(diff, alpha));
        }
        ew_store<VEC>(P + static_cast<size_t>(i) * ldp, n, p);
    }
    g = block_sum(g, red);
    if (threadIdx.x == 0) atomicAdd(gap, g);
}

// gradient += it - (2 it) * P, unfused IEEE operations in the reference's order.
template <bool VEC>
__global__ void __launch_bounds__(kEwThreads) regularize_kernel(float* G, long long ldg, const float* P, long long ldp,
                                                                int n, int it) {
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        float g[4], p[4];
        ew_load<VEC>(G + static_cast<size_t>(i) * ldg, n, g);
        ew_load<VEC>(P + static_cast<size_t>(i) * ldp, n, p);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float t = __fmul_rn(static_cast<float>(it * 2), p[q]);
            g[q] = __fadd_rn(g[q], __fsub_rn(static_cast<float>(it), t));
        }
        ew_store<VEC>(G + static_cast<size_t>(i) * ldg, n, g);
    }
}

// out[x][y] += sqrtf(sum_i (s[x][i] - t[y][i])^2), squares of FP32 differences summed in double
// (the reference accumulates into `auto sum = 0.0`).
template <bool VEC>
__global__ void __launch_bounds__(kEwThreads) add_distance_kernel(const float* s, const float* t, int n, float* out,
                                                                  long long ldo) {
    float f[4][4];  // features of this thread's columns
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int y = ew_column<VEC>(q);
#pragma unroll
        for (int k = 0; k < 4; ++k) f[q][k] = y < n ? t[4 * static_cast<size_t>(y) + k] : 0.f;
    }
    for (int x = blockIdx.y; x < n; x += gridDim.y) {
        float o[4], a[4];
        ew_load<VEC>(out + static_cast<size_t>(x) * ldo, n, o);
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = s[4 * static_cast<size_t>(x) + k];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            double sum = 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float d = a[k] - f[q][k];
                sum += __fmul_rn(d, d);
            }
            o[q] += sqrtf(static_cast<float>(sum));
        }
        ew_store<VEC>(out + static_cast<size_t>(x) * ldo, n, o);
    }
}

// A row of up to 8192 elements in registers: quad k of thread t starts
// at column 4 (256 k + t) with float4 loads (VEC), else column q 256 + t of each 1024.
constexpr int kRowThreads = 256;
template <bool VEC>
FUGAL_DEVICE int row_column(int k, int q) {
    return VEC ? (k * kRowThreads + static_cast<int>(threadIdx.x)) * 4 + q
               : (k * 4 + q) * kRowThreads + static_cast<int>(threadIdx.x);
}
template <bool VEC>
FUGAL_DEVICE float4 row_quad(const float* row, int k, int cols, float fill) {
    if (VEC) {  // cols is a multiple of 4
        const int c = row_column<true>(k, 0);
        return c < cols ? *reinterpret_cast<const float4*>(row + c) : make_float4(fill, fill, fill, fill);
    }
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = row_column<false>(k, q);
        v[q] = c < cols ? row[c] : fill;
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

// out[r] = (1-w) out[r] - w LSE_c(K[r,c] + add[c]) (w == 1 within 1e-4: out[r] = -LSE).
// One block per row, the row read once: QUADS float4 per thread stay in registers
// between the maximum and the exponentials (rows up to
// 8192), and longer rows (LONG) keep a running (max, sum) over pieces of 8192.
// Bound by HBM: 172 us with two scalar passes over a row, 52 us here at n = 8192 (268
// MB, 41 us at the copy peak).
template <int QUADS, bool VEC, bool LONG>
__global__ void __launch_bounds__(kRowThreads) log_step_kernel(const float* K, long long ldk, int cols,
                                                               const float* add, float* out, float w) {
    __shared__ float sm_m[kRowThreads / 32], sm_s[kRowThreads / 32];
    const int r = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float M = -INFINITY, S = 0.f;
    constexpr int PIECE = QUADS * 4 * kRowThreads;
    for (int c0 = 0; c0 < (LONG ? cols : 1); c0 += PIECE) {
        const float* row = K + static_cast<size_t>(r) * ldk + c0;
        const float* ad = add + c0;
        const int left = cols - c0;
        float4 x[QUADS];
#pragma unroll
        for (int k = 0; k < QUADS; ++k) x[k] = row_quad<VEC>(row, k, left, -INFINITY);
        float m = -INFINITY;
#pragma unroll
        for (int k = 0; k < QUADS; ++k) {
            const float4 a4 = row_quad<VEC>(ad, k, left, 0.f);
            x[k] = make_float4(x[k].x + a4.x, x[k].y + a4.y, x[k].z + a4.z, x[k].w + a4.w);
            m = fmaxf(m, fmaxf(fmaxf(x[k].x, x[k].y), fmaxf(x[k].z, x[k].w)));
        }
        m = warp_max(m);
        if (lane == 0) sm_m[warp] = m;
        __syncthreads();
        float Mp = M;
#pragma unroll
        for (int q = 0; q < kRowThreads / 32; ++q) Mp = fmaxf(Mp, sm_m[q]);
        const float base = (Mp == -INFINITY) ? 0.f : Mp;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < QUADS; ++k)
            s += (expf(x[k].x - base) + expf(x[k].y - base)) + (expf(x[k].z - base) + expf(x[k].w - base));
        s = warp_sum(s);
        if (lane == 0) sm_s[warp] = s;
        __syncthreads();
        float piece = 0.f;
#pragma unroll
        for (int q = 0; q < kRowThreads / 32; ++q) piece += sm_s[q];
        S = (LONG && c0 > 0 ? S * expf(M - base) : 0.f) + piece;  // (0 times 0 before any finite entry)
        M = Mp;
        if (LONG) __syncthreads();  // the next piece writes sm_m, sm_s
    }
    if (threadIdx.x == 0) {
        const float lse = M + logf(S);
        out[r] = (fabsf(w - 1.0f) < 1e-4f) ? -lse : (1.0f - w) * out[r] - w * lse;
    }
}

template <bool VEC>
void launch_log_step(int64_t rows, const float* K, int64_t ldk, int cols, const float* add, float* out, float w,
                     cudaStream_t stream) {
    const unsigned grid = static_cast<unsigned>(rows);
    if (cols <= 1024)
        log_step_kernel<1, VEC, false><<<grid, kRowThreads, 0, stream>>>(K, ldk, cols, add, out, w);
    else if (cols <= 2048)
        log_step_kernel<2, VEC, false><<<grid, kRowThreads, 0, stream>>>(K, ldk, cols, add, out, w);
    else if (cols <= 4096)
        log_step_kernel<4, VEC, false><<<grid, kRowThreads, 0, stream>>>(K, ldk, cols, add, out, w);
    else if (cols <= 8192)
        log_step_kernel<8, VEC, false><<<grid, kRowThreads, 0, stream>>>(K, ldk, cols, add, out, w);
    else
        log_step_kernel<8, VEC, true><<<grid, kRowThreads, 0, stream>>>(K, ldk, cols, add, out, w);
}

template <bool VEC>
__global__ void __launch_bounds__(kRowThreads) marginal_rows_kernel(const float* K, long long ldk, int n,
                                                                    const float* u, const float* v, double* result) {
    __shared__ double red[32];
    const int r = blockIdx.x;
    const float* row = K + static_cast<size_t>(r) * ldk;
    const float ur = u[r];
    double s = 0.0;
    const int quads = (n + 4 * kRowThreads - 1) / (4 * kRowThreads);
#pragma unroll 4
    for (int k = 0; k < quads; ++k) {
        const float4 x = row_quad<VEC>(row, k, n, 0.f), a = row_quad<VEC>(v, k, n, 0.f);
        const float e[4] = {x.x + ur + a.x, x.y + ur + a.y, x.z + ur + a.z, x.w + ur + a.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (row_column<VEC>(k, q) < n) s += static_cast<double>(expf(e[q]));
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) atomicAdd(result, fabs(s - 1.0));
}

// 32 columns per block (one per lane), 32 warps over the rows: enough loads in flight
// for few columns (153 us at n = 1024 with one thread per column).
__global__ void __launch_bounds__(1024) marginal_cols_kernel(const float* K, long long ldk, int n, const float* u,
                                                             const float* v, double* result) {
    __shared__ double part[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (c < n) {
        const float vc = v[c];
#pragma unroll 8
        for (int r = warp; r < n; r += 32) s += static_cast<double>(expf(K[static_cast<size_t>(r) * ldk + c] + u[r] + vc));
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 32; ++w) t += part[w][lane];
        const double dev = warp_sum(c < n ? fabs(t - 1.0) : 0.0);
        if (lane == 0) atomicAdd(result, dev);
    }
}

// K = scale * C and cost = (float)((K + U_i) + V_j) in FP64, zero in the padding columns
// [n, ldo): one pass (12 bytes an entry) for what was six elementwise passes with FP64
// intermediates (1.16 ms at n = 8192, 8 ms at 20011; 0.13 and 0.8 ms here).
template <bool VEC>
__global__ void __launch_bounds__(kEwThreads) absorb_cost_kernel(const float* __restrict__ C, long long ldc, int n,
                                                                 float scale, const double* __restrict__ U,
                                                                 const double* __restrict__ V, float* __restrict__ K,
                                                                 long long ldk, float* __restrict__ cost,
                                                                 long long ldo) {
    double vj[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) vj[q] = ew_column<VEC>(q) < n ? V[ew_column<VEC>(q)] : 0.0;
#pragma unroll 2
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        float c[4], o[4];
        ew_load<VEC>(C + static_cast<size_t>(i) * ldc, n, c);
        const double ui = U[i];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            c[q] = __fmul_rn(scale, c[q]);
            o[q] = ew_column<VEC>(q) < n ? static_cast<float>(static_cast<double>(c[q]) + ui + vj[q]) : 0.f;
        }
        if (K != nullptr) ew_store<VEC>(K + static_cast<size_t>(i) * ldk, n, c);
        ew_store<VEC>(cost + static_cast<size_t>(i) * ldo, static_cast<int>(ldo), o);
    }
}

template <bool VEC>
__global__ void __launch_bounds__(kEwThreads) count_le_kernel(const float* P, long long ldp, int n, float thr,
                                                              unsigned long long* count) {
    int c = 0;  // at most 4 n per thread
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        float p[4];
        ew_load<VEC>(P + static_cast<size_t>(i) * ldp, n, p);
#pragma unroll
        for (int q = 0; q < 4; ++q) c += (ew_column<VEC>(q) < n && p[q] <= thr) ? 1 : 0;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, static_cast<unsigned long long>(c));
}

fugal_status check_square(const void* p, int64_t ld, int64_t n, const char* who, const char* what) {
    if (p == nullptr) return fail(FUGAL_BAD_ARGUMENT, "%s: %s is null", who, what);
    if (n <= 0 || n > (1ll << 30)) return fail(FUGAL_BAD_SHAPE, "%s: bad n", who);
    if (ld < n) return fail(FUGAL_BAD_SHAPE, "%s: leading dimension of %s < n", who, what);
    return FUGAL_OK;
}

// 16-byte accesses: whole quads in every row of every operand.
struct EwRows {
    const void* p;
    int64_t ld;
};
bool ew_vec(int64_t n, std::initializer_list<EwRows> rows) {
    if ((n % 4) != 0) return false;
    for (const EwRows& r : rows)
        if ((r.ld % 4) != 0 || !aligned16(r.p)) return false;
    return true;
}

}  // namespace fugal

using namespace fugal;

namespace {

fugal_status fw_update(int64_t n, float* P, int64_t ldp, const float* cost32, int64_t ld32, const float* u,
                       const float* v, double* U, double* V, double alpha, double regularization, double* gap,
                       int commit, const PlanOut* plan, const char* who, cudaStream_t stream) {
    FUGAL_TRY(check_square(P, ldp, n, who, "P"));
    FUGAL_TRY(check_square(cost32, ld32, n, who, "cost32"));
    if (u == nullptr || v == nullptr || gap == nullptr) return fail(FUGAL_BAD_ARGUMENT, "%s: null duals or gap", who);
    if ((U == nullptr) != (V == nullptr)) return fail(FUGAL_BAD_ARGUMENT, "%s: give both U and V", who);
    if (commit && U == nullptr) return fail(FUGAL_BAD_ARGUMENT, "%s: commit needs U and V", who);
    if ((ldp % 4) || (ld32 % 4) || !aligned16(P) || !aligned16(cost32) || !aligned16(v))
        return fail(FUGAL_BAD_SHAPE, "%s: P, cost32, v need 16-byte rows", who);
    FUGAL_TRY(cuda_check(cudaMemsetAsync(gap, 0, sizeof(double), stream), who));
    {
        LaunchScope scope(FUGAL_KERNEL_UPDATE, stream);
        const int blocks = static_cast<int>(std::min<int64_t>(n, static_cast<int64_t>(sm_count()) * 8));
        if (plan != nullptr)
            fw_update_kernel<true><<<blocks, kEwThreads, 0, stream>>>(P, ldp, cost32, ld32, u, v, U, V,
                                                                      static_cast<int>(n), static_cast<float>(alpha),
                                                                      regularization, gap, *plan);
        else
            fw_update_kernel<false><<<blocks, kEwThreads, 0, stream>>>(P, ldp, cost32, ld32, u, v, U, V,
                                                                       static_cast<int>(n),
                                                                       static_cast<float>(alpha), regularization,
                                                                       gap, PlanOut{});
        FUGAL_TRY(launch_check(who));
    }
    if (commit) {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        const int blocks = static_cast<int>(std::min<int64_t>((n + 255) / 256, 1024));
        commit_duals_kernel<<<blocks, 256, 0, stream>>>(u, v, U, V, static_cast<int>(n));
        FUGAL_TRY(launch_check("fugal_fw_update: commit"));
    }
    return FUGAL_OK;
}

}  // namespace

extern "C" fugal_status fugal_fw_update(int64_t n, float* P, int64_t ldp, const float* cost32, int64_t ld32,
                                        const float* u, const float* v, double* U, double* V, double alpha,
                                        double regularization, double* gap, int commit, fugal_stream_t stream) {
    return fw_update(n, P, ldp, cost32, ld32, u, v, U, V, alpha, regularization, gap, commit, nullptr,
                     "fugal_fw_update", reinterpret_cast<cudaStream_t>(stream));
}

extern "C" fugal_status fugal_fw_update_collect(int64_t n, float* P, int64_t ldp, const float* cost32, int64_t ld32,
                                                const float* u, const float* v, double* U, double* V, double alpha,
                                                double regularization, double* gap, int commit, int32_t* plan_counts,
                                                fugal_plan_entry* plan_entries, int32_t slots,
                                                fugal_stream_t stream) {
    const char* who = "fugal_fw_update_collect";
    if (plan_counts == nullptr || plan_entries == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "%s: null plan buffers", who);
    if (slots < 1 || slots > 1024) return fail(FUGAL_BAD_ARGUMENT, "%s: slots must be in [1, 1024]", who);
    FUGAL_TRY(cuda_check(cudaMemsetAsync(plan_counts, 0, static_cast<size_t>(n) * sizeof(int32_t),
                                         reinterpret_cast<cudaStream_t>(stream)),
                         who));
    const PlanOut plan{plan_counts, plan_entries, slots};
    return fw_update(n, P, ldp, cost32, ld32, u, v, U, V, alpha, regularization, gap, commit, &plan, who,
                     reinterpret_cast<cudaStream_t>(stream));
}

extern "C" fugal_status fugal_update_quasi_permutation_log(float* P, int64_t ldp, const float* K, int64_t ldk,
                                                           const float* u, const float* v, int64_t n, float alpha,
                                                           float regularization, double* gap,
                                                           fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const char* who = "fugal_update_quasi_permutation_log";
    FUGAL_TRY(check_square(P, ldp, n, who, "P"));
    FUGAL_TRY(check_square(K, ldk, n, who, "K"));
    if (u == nullptr || v == nullptr || gap == nullptr) return fail(FUGAL_BAD_ARGUMENT, "%s: null argument", who);
    FUGAL_TRY(cuda_check(cudaMemsetAsync(gap, 0, sizeof(double), stream), who));
    LaunchScope scope(FUGAL_KERNEL_UPDATE, stream);
    const int ni = static_cast<int>(n);
    if (ew_vec(n, {{P, ldp}, {K, ldk}, {v, 4}}))
        update_log_kernel<true><<<ew_blocks(n), kEwThreads, 0, stream>>>(P, ldp, K, ldk, u, v, ni, alpha, regularization, gap);
    else
        update_log_kernel<false><<<ew_blocks(n), kEwThreads, 0, stream>>>(P, ldp, K, ldk, u, v, ni, alpha, regularization, gap);
    return launch_check(who);
}

extern "C" fugal_status fugal_regularize(float* gradient, int64_t ldg, const float* P, int64_t ldp, int64_t n,
                                         int iteration, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    FUGAL_TRY(check_square(gradient, ldg, n, "fugal_regularize", "gradient"));
    FUGAL_TRY(check_square(P, ldp, n, "fugal_regularize", "P"));
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    if (ew_vec(n, {{gradient, ldg}, {P, ldp}}))
        regularize_kernel<true><<<ew_blocks(n), kEwThreads, 0, stream>>>(gradient, ldg, P, ldp, static_cast<int>(n), iteration);
    else
        regularize_kernel<false><<<ew_blocks(n), kEwThreads, 0, stream>>>(gradient, ldg, P, ldp, static_cast<int>(n), iteration);
    return launch_check("fugal_regularize");
}

extern "C" fugal_status fugal_add_distance(const float* source, const float* target, int64_t n, float* out,
                                           int64_t ldo, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    FUGAL_TRY(check_square(out, ldo, n, "fugal_add_distance", "out"));
    if (source == nullptr || target == nullptr) return fail(FUGAL_BAD_ARGUMENT, "fugal_add_distance: null features");
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    if (ew_vec(n, {{out, ldo}}))
        add_distance_kernel<true><<<ew_blocks(n), kEwThreads, 0, stream>>>(source, target, static_cast<int>(n), out, ldo);
    else
        add_distance_kernel<false><<<ew_blocks(n), kEwThreads, 0, stream>>>(source, target, static_cast<int>(n), out, ldo);
    return launch_check("fugal_add_distance");
}

extern "C" fugal_status fugal_sinkhorn_log_step(const float* K, int64_t rows, int64_t cols, int64_t ldk,
                                                const float* add, float* out, float momentum,
                                                fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (K == nullptr || add == nullptr || out == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_log_step: null argument");
    if (rows <= 0 || cols <= 0 || ldk < cols || rows > (1ll << 31) - 1)
        return fail(FUGAL_BAD_SHAPE, "fugal_sinkhorn_log_step: bad shape");
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    // float4 rows need whole, aligned quads in K and add
    if ((cols % 4) == 0 && (ldk % 4) == 0 && aligned16(K) && aligned16(add))
        launch_log_step<true>(rows, K, ldk, static_cast<int>(cols), add, out, momentum, stream);
    else
        launch_log_step<false>(rows, K, ldk, static_cast<int>(cols), add, out, momentum, stream);
    return launch_check("fugal_sinkhorn_log_step");
}

extern "C" fugal_status fugal_sinkhorn_log_marginal(const float* K, int64_t n, int64_t ldk, const float* u,
                                                    const float* v, int axis, double* result,
                                                    fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    FUGAL_TRY(check_square(K, ldk, n, "fugal_sinkhorn_log_marginal", "K"));
    if (u == nullptr || v == nullptr || result == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_log_marginal: null argument");
    if (axis != 0 && axis != 1) return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_log_marginal: axis must be 0 or 1");
    FUGAL_TRY(cuda_check(cudaMemsetAsync(result, 0, sizeof(double), stream), "fugal_sinkhorn_log_marginal"));
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    const unsigned rows = static_cast<unsigned>(n);
    if (axis == 1 && (n % 4) == 0 && (ldk % 4) == 0 && aligned16(K) && aligned16(v))
        marginal_rows_kernel<true><<<rows, kRowThreads, 0, stream>>>(K, ldk, static_cast<int>(n), u, v, result);
    else if (axis == 1)
        marginal_rows_kernel<false><<<rows, kRowThreads, 0, stream>>>(K, ldk, static_cast<int>(n), u, v, result);
    else
        marginal_cols_kernel<<<static_cast<unsigned>((n + 31) / 32), 1024, 0, stream>>>(K, ldk, static_cast<int>(n), u,
                                                                                         v, result);
    return launch_check("fugal_sinkhorn_log_marginal");
}

extern "C" fugal_status fugal_absorb_cost(const float* C, int64_t ldc, int64_t n, double scale, const double* U,
                                          const double* V, float* K, int64_t ldk, float* cost32, int64_t ld32,
                                          fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const char* who = "fugal_absorb_cost";
    FUGAL_TRY(check_square(C, ldc, n, who, "C"));
    FUGAL_TRY(check_square(cost32, ld32, n, who, "cost32"));
    if (U == nullptr || V == nullptr) return fail(FUGAL_BAD_ARGUMENT, "%s: null duals", who);
    if (K != nullptr && ldk < n) return fail(FUGAL_BAD_SHAPE, "%s: ldk < n", who);
    if (ld32 > (1ll << 30)) return fail(FUGAL_BAD_SHAPE, "%s: ld32 too large", who);
    const float s = static_cast<float>(scale);
    const int ni = static_cast<int>(n);
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    if (ew_vec(n, {{C, ldc}, {K, K != nullptr ? ldk : 4}, {cost32, ld32}}))
        absorb_cost_kernel<true><<<ew_blocks(ld32), kEwThreads, 0, stream>>>(C, ldc, ni, s, U, V, K, ldk, cost32, ld32);
    else
        absorb_cost_kernel<false><<<ew_blocks(ld32), kEwThreads, 0, stream>>>(C, ldc, ni, s, U, V, K, ldk, cost32, ld32);
    return launch_check(who);
}

extern "C" fugal_status fugal_count_le(const float* P, int64_t ldp, int64_t n, float threshold, int64_t* count,
                                       fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    FUGAL_TRY(check_square(P, ldp, n, "fugal_count_le", "P"));
    if (count == nullptr) return fail(FUGAL_BAD_ARGUMENT, "fugal_count_le: null count");
    FUGAL_TRY(cuda_check(cudaMemsetAsync(count, 0, sizeof(int64_t), stream), "fugal_count_le"));
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    unsigned long long* total = reinterpret_cast<unsigned long long*>(count);
    if (ew_vec(n, {{P, ldp}}))
        count_le_kernel<true><<<ew_blocks(n), kEwThreads, 0, stream>>>(P, ldp, static_cast<int>(n), threshold, total);
    else
        count_le_kernel<false><<<ew_blocks(n), kEwThreads, 0, stream>>>(P, ldp, static_cast<int>(n), threshold, total);
    return launch_check("fugal_count_le");
}
