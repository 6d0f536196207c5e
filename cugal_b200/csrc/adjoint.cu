// Differentiation of the log-domain Sinkhorn solve (the plan P of
// cugal/sinkhorn.py:90-120 as a function of the cost C).
//
// At the converged potentials the plan P = exp(-C/reg + u 1^T + 1 v^T) has unit
// row and column sums.  Implicit differentiation of those constraints gives,
// for a loss L(P) with G = dL/dP,
//     a = (G o P) 1,  b = (G o P)^T 1,
//     [ I  P ; P^T  I ] [alpha; beta] = [a; b]      (consistent, one null vector [1; -1]),
//     dL/dK = P o (G - alpha 1^T - 1 beta^T),   dL/dC = -dL/dK / reg.
// The block system is symmetric positive semi-definite (eigenvalues 1 +- the
// singular values of P), so conjugate gradients solve it with one pass over P
// per iteration: the kernel below forms P y and P^T x from the same read.
//
// Kernels:
//   plan_kernel        P = exp(L + u_i + v_j) from the absorbed cost and duals;
//   matvec_part_kernel tiles of 64 rows x 1024 columns: row partials of P y and
//                      column partials of P^T x (P optionally weighted by G);
//   merge_add_kernel   FP64 sums of the partials;
//   cg_kernel          the whole conjugate-gradient solve in one launch;
//   adjoint_kernel     out = scale * P o (G - alpha_i - beta_j).
#include <cuda_runtime.h>

#include <algorithm>

#include "fugal_common.cuh"
#include "fugal_host.h"

namespace fugal {

constexpr int kMvRows = 64;
constexpr int kMvThreads = 256;
constexpr int kMvCols = kMvThreads * 4;

__global__ void plan_kernel(const float* __restrict__ L, long long ldl, int n, const float* __restrict__ u,
                            const float* __restrict__ v, float* __restrict__ P, long long ldp) {
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        const float ui = u[i];
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
            P[static_cast<size_t>(i) * ldp + j] = expf(L[static_cast<size_t>(i) * ldl + j] + ui + v[j]);
    }
}

// Block (cx, ry) covers rows [ry*64, +64) and columns [cx*1024, +1024); each
// thread owns 4 consecutive columns.  row_part[cx][i] = sum_j M_ij y_j over the
// block's columns, col_part[ry][j] = sum_i M_ij x_i over its rows, with
// M = P or P o W.
__global__ void __launch_bounds__(kMvThreads) matvec_part_kernel(const float* __restrict__ P, long long ldp,
                                                                 const float* __restrict__ W, long long ldw, int n,
                                                                 const double* __restrict__ x,
                                                                 const double* __restrict__ y, double* row_part,
                                                                 double* col_part) {
    __shared__ double red[kMvThreads / 32][kMvRows];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = blockIdx.y * kMvRows;
    const int j0 = blockIdx.x * kMvCols + threadIdx.x * 4;
    double yj[4], cs[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        yj[q] = (j0 + q < n) ? y[j0 + q] : 0.0;
        cs[q] = 0.0;
    }
    for (int r = 0; r < kMvRows; ++r) {
        const int i = r0 + r;
        double rs = 0.0;
        if (i < n) {
            const double xi = x[i];
            const float* prow = P + static_cast<size_t>(i) * ldp;
            const float* wrow = W ? W + static_cast<size_t>(i) * ldw : nullptr;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = j0 + q;
                if (j < n) {
                    double m = static_cast<double>(prow[j]);
                    if (wrow) m *= static_cast<double>(wrow[j]);
                    rs += m * yj[q];
                    cs[q] += m * xi;
                }
            }
        }
        rs = warp_sum(rs);
        if (lane == 0) red[warp][r] = rs;
    }
    __syncthreads();
    if (threadIdx.x < kMvRows) {
        const int i = r0 + threadIdx.x;
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kMvThreads / 32; ++w) s += red[w][threadIdx.x];
        if (i < n) row_part[static_cast<size_t>(blockIdx.x) * n + i] = s;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (j0 + q < n) col_part[static_cast<size_t>(blockIdx.y) * n + j0 + q] = cs[q];
}

__global__ void adjoint_kernel(const float* __restrict__ P, long long ldp, const float* __restrict__ G,
                               long long ldg, int n, const double* __restrict__ alpha,
                               const double* __restrict__ beta, double scale, float* __restrict__ out,
                               long long ldo) {
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        const double ai = alpha[i];
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
            const double p = static_cast<double>(P[static_cast<size_t>(i) * ldp + j]);
            const double g = static_cast<double>(G[static_cast<size_t>(i) * ldg + j]);
            out[static_cast<size_t>(i) * ldo + j] = static_cast<float>(scale * p * (g - ai - beta[j]));
        }
    }
}

// Backward of one half step of the unrolled log-domain iteration (no momentum).
// axis 1 (row half, out_i = -LSE_j(K_ij + other_j)):  E_ij = exp(K_ij + other_j + out_i),
//     gK_ij -= g_i E_ij,   g_other_j -= sum_i g_i E_ij        (column partials)
// axis 0 (column half, out_j = -LSE_i(K_ij + other_i)): E_ij = exp(K_ij + other_i + out_j),
//     gK_ij -= g_j E_ij,   g_other_i -= sum_j g_j E_ij        (row partials)
// A block covers ROWS rows x 1024 columns (4 consecutive columns per thread), bound by the
// chain of its FP64 exponentials and gK updates where blocks are few: at n = 1024 128 blocks of
// 8 rows, 16 of 64 (see unrolled_rows for the times).
template <int ROWS>
__global__ void __launch_bounds__(kMvThreads) unrolled_step_kernel(const float* __restrict__ K, long long ldk, int n,
                                                                   const float* __restrict__ out_dual,
                                                                   const float* __restrict__ other_dual,
                                                                   const double* __restrict__ g, int axis,
                                                                   float* __restrict__ gK, long long ldg,
                                                                   double* row_part, double* col_part) {
    __shared__ double red[kMvThreads / 32][ROWS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = blockIdx.y * ROWS;
    const int j0 = blockIdx.x * kMvCols + threadIdx.x * 4;
    double cs[4] = {0.0, 0.0, 0.0, 0.0};
    for (int r = 0; r < ROWS; ++r) {
        const int i = r0 + r;
        double rs = 0.0;
        if (i < n) {
            const float* krow = K + static_cast<size_t>(i) * ldk;
            float* grow = gK + static_cast<size_t>(i) * ldg;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = j0 + q;
                if (j < n) {
                    double e, w;
                    if (axis == 1) {
                        e = exp(static_cast<double>(krow[j]) + other_dual[j] + out_dual[i]);
                        w = g[i] * e;
                        cs[q] -= w;
                    } else {
                        e = exp(static_cast<double>(krow[j]) + other_dual[i] + out_dual[j]);
                        w = g[j] * e;
                        rs -= w;
                    }
                    grow[j] = static_cast<float>(static_cast<double>(grow[j]) - w);
                }
            }
        }
        if (axis == 0) {
            rs = warp_sum(rs);
            if (lane == 0) red[warp][r] = rs;
        }
    }
    if (axis == 0) {
        __syncthreads();
        if (threadIdx.x < ROWS) {
            const int i = r0 + threadIdx.x;
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kMvThreads / 32; ++w) s += red[w][threadIdx.x];
            if (i < n) row_part[static_cast<size_t>(blockIdx.x) * n + i] = s;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (j0 + q < n) col_part[static_cast<size_t>(blockIdx.y) * n + j0 + q] = cs[q];
    }
}

// out[k] += sum of the parts of column k (add), or = it: 32 columns per block, the
// parts over its 8 warps, eight loads in flight per lane.
__global__ void __launch_bounds__(256) merge_add_kernel(const double* __restrict__ part, int parts, int n, double* out,
                                                        int add) {
    __shared__ double red[8][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (k < n) {
        for (int p0 = warp; p0 < parts; p0 += 64) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = p0 + 8 * u < parts ? part[static_cast<size_t>(p0 + 8 * u) * n + k] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
    }
    red[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && k < n) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += red[w][lane];
        out[k] = add ? out[k] + t : t;
    }
}

// Conjugate gradients on [I P; P^T I] [alpha; beta] = [a; b] (alpha, beta from 0)
// in one persistent, cooperative launch: one 512-thread CTA per SM owns a block of
// rows (its entries of alpha) and a block of columns (its entries of beta).  Per
// iteration:
//   matvec   P y (complete for the CTA's rows) and the CTA's partial of P^T x, from
//            one read of its rows of P; the search direction's column half y sits in
//            every CTA's shared memory.  Grid barrier.
//   columns  the CTA's columns of P^T x, <p, A p>.  Grid barrier.
//   update   alpha/beta and the residual of the CTA's rows and columns, <r, r>.  Grid
//            barrier; every CTA then forms the new y itself from the residual.
// All vectors, sums and scalars are FP64, sums in a fixed order.  As a loop of
// launches an iteration was one matvec (38 us at n = 4096), 16 vector launches and a
// host round trip for the residual, 145 us; here about 20 us, bound by the L2 reads
// of P (67 MB) and the FP32 -> FP64 conversions (16 a clock per SM).
constexpr int kCgThreads = 512;
constexpr int kCgWarps = kCgThreads / 32;
constexpr int kCgRows = 8;         // rows in flight per thread
constexpr int kCgMaxN = 16384;     // y (8 bytes a column) fits the shared memory
constexpr int kCgMaxOwn = 128;     // rows and columns a CTA owns at most

struct CgArgs {
    const float* P;
    long long ldp;
    int n;
    int own;             // rows (and columns) per CTA
    const double* a;     // [n]
    const double* b;     // [n]
    double tol;
    int max_iter;
    double* alpha;       // [n]
    double* beta;        // [n]
    double* info;        // iterations, relative residual, status
    double* colpart;     // [CTAs][n]
    double* r_cols;      // [n] residual of the column half
    double* dots;        // [2][CTAs]
    unsigned* arrivals;
    int* status;
    unsigned long long wait_limit_ns;  // test hooks (test_wait_limit_ns, test_fault_barrier in fugal_host.h)
    int fault_barrier;
};

// Sums of 8 values over the 32 lanes of a warp: on return lane l holds the sum of
// value (l >> 2) in the low two bits' group (all four lanes alike).
FUGAL_DEVICE double warp_sum8(const double (&v)[8]) {
    const int lane = threadIdx.x & 31;
    double w4[4], w2[2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double send = (lane & 16) ? v[k] : v[k + 4];
        const double keep = (lane & 16) ? v[k + 4] : v[k];
        w4[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double send = (lane & 8) ? w4[k] : w4[k + 2];
        const double keep = (lane & 8) ? w4[k + 2] : w4[k];
        w2[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    const double send = (lane & 4) ? w2[0] : w2[1];
    double w = ((lane & 4) ? w2[1] : w2[0]) + __shfl_xor_sync(0xffffffffu, send, 4);
    w += __shfl_xor_sync(0xffffffffu, w, 2);
    w += __shfl_xor_sync(0xffffffffu, w, 1);
    return w;
}

// The sum of one value per CTA, the same in every thread of every CTA.  (`total` is not the scratch
// of a block_sum: the first warp of one that follows would write it under a slower warp's read.)
FUGAL_DEVICE double grid_total(const double* per_cta) {
    __shared__ double total;
    __syncthreads();  // the total before has been read
    if (threadIdx.x < 32) {
        double s = 0.0;
        const int ctas = static_cast<int>(gridDim.x);
        for (int k0 = threadIdx.x; k0 < ctas; k0 += 256) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = k0 + 32 * u < ctas ? __ldcg(per_cta + k0 + 32 * u) : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
        s = warp_sum(s);
        if (threadIdx.x == 0) total = s;
    }
    __syncthreads();
    return total;
}

template <bool VEC>
__global__ void __launch_bounds__(kCgThreads, 1) cg_kernel(const __grid_constant__ CgArgs p) {
    extern __shared__ __align__(16) double y_s[];  // [n rounded up to 2048]
    __shared__ double x_s[kCgMaxOwn], rx_s[kCgMaxOwn], zx_s[kCgMaxOwn], apx_s[kCgMaxOwn];
    __shared__ double ry_s[kCgMaxOwn], zy_s[kCgMaxOwn], apy_s[kCgMaxOwn];
    __shared__ double red[kCgWarps][kCgMaxOwn];
    __shared__ double scratch[32];
    constexpr int SPAN = kCgThreads * 4;  // columns a CTA covers at once
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = p.n;
    const int o0 = blockIdx.x * p.own;
    const int own = max(0, min(n, o0 + p.own) - o0);
    const int span_n = (n + SPAN - 1) / SPAN * SPAN;
    unsigned arrivals = 0;
    auto barrier = [&]() {  // false: a wait ran out; cg_end_kernel then leaves no result
        arrivals += gridDim.x;
        bool ok = grid_barrier(p.arrivals, p.status, true, arrivals, p.wait_limit_ns);
        if (p.fault_barrier > 0 && blockIdx.x == gridDim.x - 1 && arrivals == p.fault_barrier * gridDim.x) {
            if (tid == 0) report_error(p.status, FUGAL_DEVICE_TIMEOUT);
            ok = false;
        }
        return ok;
    };
    // column q of this thread in the span starting at c0
    auto column = [&](int c0, int q) { return VEC ? c0 + tid * 4 + q : c0 + q * kCgThreads + tid; };

    for (int j = tid; j < span_n; j += kCgThreads) y_s[j] = j < n ? p.b[j] : 0.0;
    double rr = 0.0;
    for (int k = tid; k < own; k += kCgThreads) {
        x_s[k] = rx_s[k] = p.a[o0 + k];
        ry_s[k] = p.b[o0 + k];
        zx_s[k] = zy_s[k] = 0.0;
        rr += rx_s[k] * rx_s[k] + ry_s[k] * ry_s[k];
    }
    rr = block_sum(rr, scratch);
    if (tid == 0) p.dots[blockIdx.x] = rr;
    if (!barrier()) return;
    double rs = grid_total(p.dots);
    const double norm = sqrt(rs);
    double rel = 0.0;
    int it = 0;
    if (norm > 0.0) {
        while (it < p.max_iter) {
            ++it;
            // ---- P y for the CTA's rows, partial P^T x
            for (int c0 = 0; c0 < n; c0 += SPAN) {
                double yq[4], cs[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int q = 0; q < 4; ++q) yq[q] = y_s[column(c0, q)];
                for (int r0 = 0; r0 < own; r0 += kCgRows) {
                    float4 m[kCgRows];
#pragma unroll
                    for (int r = 0; r < kCgRows; ++r) {
                        m[r] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (r0 + r < own) {
                            const float* row = p.P + static_cast<size_t>(o0 + r0 + r) * p.ldp;
                            if (VEC) {  // n is a multiple of 4
                                if (column(c0, 0) < n) m[r] = __ldg(reinterpret_cast<const float4*>(row + column(c0, 0)));
                            } else {
                                if (column(c0, 0) < n) m[r].x = __ldg(row + column(c0, 0));
                                if (column(c0, 1) < n) m[r].y = __ldg(row + column(c0, 1));
                                if (column(c0, 2) < n) m[r].z = __ldg(row + column(c0, 2));
                                if (column(c0, 3) < n) m[r].w = __ldg(row + column(c0, 3));
                            }
                        }
                    }
                    double rsum[kCgRows];
#pragma unroll
                    for (int r = 0; r < kCgRows; ++r) {
                        const double x = r0 + r < own ? x_s[r0 + r] : 0.0;
                        const double d0 = m[r].x, d1 = m[r].y, d2 = m[r].z, d3 = m[r].w;
                        rsum[r] = fma(d3, yq[3], fma(d2, yq[2], fma(d1, yq[1], d0 * yq[0])));
                        cs[0] = fma(d0, x, cs[0]);
                        cs[1] = fma(d1, x, cs[1]);
                        cs[2] = fma(d2, x, cs[2]);
                        cs[3] = fma(d3, x, cs[3]);
                    }
                    const double s = warp_sum8(rsum);
                    const int r = r0 + (lane >> 2);
                    if ((lane & 3) == 0 && r < own) red[warp][r] = (c0 == 0 ? 0.0 : red[warp][r]) + s;
                }
                double* cp = p.colpart + static_cast<size_t>(blockIdx.x) * n;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (column(c0, q) < n) cp[column(c0, q)] = cs[q];
            }
            if (!barrier()) return;
            // ---- A p on the CTA's rows and columns, <p, A p>
            double dot = 0.0;
            for (int k = tid; k < own; k += kCgThreads) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < kCgWarps; ++w) s += red[w][k];
                apx_s[k] = x_s[k] + s;
                dot += x_s[k] * apx_s[k];
            }
            __syncthreads();  // red is read
            for (int k0 = 0; k0 < own; k0 += 32) {
                const int k = k0 + lane;
                const int ctas = static_cast<int>(gridDim.x);
                double s = 0.0;
                if (k < own) {
                    for (int c0 = warp; c0 < ctas; c0 += 10 * kCgWarps) {
                        double v[10];
#pragma unroll
                        for (int u = 0; u < 10; ++u) {
                            const int c = c0 + u * kCgWarps;
                            v[u] = c < ctas ? __ldcg(p.colpart + static_cast<size_t>(c) * n + o0 + k) : 0.0;
                        }
#pragma unroll
                        for (int u = 0; u < 10; ++u) s += v[u];
                    }
                    red[warp][k] = s;
                }
            }
            __syncthreads();
            for (int k = tid; k < own; k += kCgThreads) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < kCgWarps; ++w) s += red[w][k];
                const double yk = y_s[o0 + k];
                apy_s[k] = s + yk;
                dot += yk * apy_s[k];
            }
            dot = block_sum(dot, scratch);
            if (tid == 0) p.dots[gridDim.x + blockIdx.x] = dot;
            if (!barrier()) return;
            const double step = rs / grid_total(p.dots + gridDim.x);
            // ---- solution and residual
            rr = 0.0;
            for (int k = tid; k < own; k += kCgThreads) {
                zx_s[k] += step * x_s[k];
                zy_s[k] += step * y_s[o0 + k];
                const double rx = rx_s[k] - step * apx_s[k], ry = ry_s[k] - step * apy_s[k];
                rx_s[k] = rx;
                ry_s[k] = ry;
                p.r_cols[o0 + k] = ry;
                rr += rx * rx + ry * ry;
            }
            rr = block_sum(rr, scratch);
            if (tid == 0) p.dots[blockIdx.x] = rr;
            if (!barrier()) return;
            const double rs_new = grid_total(p.dots);
            rel = sqrt(rs_new) / norm;
            if (rel < p.tol) break;
            const double ratio = rs_new / rs;
            rs = rs_new;
            for (int k = tid; k < own; k += kCgThreads) x_s[k] = rx_s[k] + ratio * x_s[k];
            for (int j = tid; j < n; j += kCgThreads) y_s[j] = __ldcg(p.r_cols + j) + ratio * y_s[j];
            __syncthreads();
        }
    }
    for (int k = tid; k < own; k += kCgThreads) {
        p.alpha[o0 + k] = zx_s[k];
        p.beta[o0 + k] = zy_s[k];
    }
    if (blockIdx.x == 0 && tid == 0) {
        p.info[0] = it;
        p.info[1] = rel;
    }
}

// The status that all CTAs of the solve share: a CTA may pass the last barrier while another one's wait
// on it runs out, so none of them can tell alone.
__global__ void __launch_bounds__(256) cg_end_kernel(const int* status, int n, double* alpha, double* beta,
                                                     double* info) {
    const int s = *status;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) {
        info[2] = s;
        if (s != 0) info[0] = info[1] = NAN;
    }
    if (s != 0 && k < n) alpha[k] = beta[k] = NAN;
}

inline dim3 ew2d(int64_t n) {
    return dim3(static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 32)),
                static_cast<unsigned>(std::min<int64_t>(n, 8 * sm_count())));
}

}  // namespace fugal

using namespace fugal;

extern "C" fugal_status fugal_sinkhorn_plan(const float* cost32, int64_t ld32, int64_t n, const float* u,
                                            const float* v, float* P, int64_t ldp, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (cost32 == nullptr || u == nullptr || v == nullptr || P == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_plan: null argument");
    if (n <= 0 || ld32 < n || ldp < n) return fail(FUGAL_BAD_SHAPE, "fugal_sinkhorn_plan: bad shape");
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    plan_kernel<<<ew2d(n), 256, 0, stream>>>(cost32, ld32, static_cast<int>(n), u, v, P, ldp);
    return launch_check("fugal_sinkhorn_plan");
}

namespace {
// Row partials of every column block and column partials of every row block of `rows` rows.
size_t partials_bytes(int64_t n, int rows) {
    const int64_t cb = (n + kMvCols - 1) / kMvCols, rb = (n + rows - 1) / rows;
    return static_cast<size_t>((cb + rb) * n) * 8 + 256;
}

// Rows of an unrolled step's block: the fewest of 8, 16, 32, 64 that leave at most 512 partial
// rows.  Small n needs the blocks, large n fewer partials to write and read (and to hold: n^2
// bytes with blocks of 8).  A row and a column half step together, us: n = 1024 41 with 8, 191
// with 64; 4096 163, 273; 8192 504 with 16, 537 with 8, 653 with 64; 16384 1942 with 32, 1970
// with 8, 1992 with 64.
int unrolled_rows(int64_t n) {
    int rows = 8;
    while (rows < kMvRows && n > 512 * rows) rows *= 2;
    return rows;
}
}  // namespace

extern "C" fugal_status fugal_plan_matvec_workspace_size(int64_t n, size_t* bytes) {
    if (bytes == nullptr) return fail(FUGAL_BAD_ARGUMENT, "fugal_plan_matvec_workspace_size: null output");
    if (n <= 0 || n > (1ll << 30)) return fail(FUGAL_BAD_SHAPE, "fugal_plan_matvec_workspace_size: bad n");
    *bytes = partials_bytes(n, kMvRows);
    return FUGAL_OK;
}

extern "C" fugal_status fugal_plan_matvec(const float* P, int64_t ldp, const float* W, int64_t ldw, int64_t n,
                                          const double* x, const double* y, double* Ptx, double* Py,
                                          void* workspace, size_t workspace_bytes, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    size_t need = 0;
    FUGAL_TRY(fugal_plan_matvec_workspace_size(n, &need));
    if (P == nullptr || x == nullptr || y == nullptr || Ptx == nullptr || Py == nullptr || workspace == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_plan_matvec: null argument");
    if (ldp < n || (W != nullptr && ldw < n)) return fail(FUGAL_BAD_SHAPE, "fugal_plan_matvec: bad leading dimension");
    if (workspace_bytes < need)
        return fail(FUGAL_WORKSPACE_TOO_SMALL, "fugal_plan_matvec: workspace %zu < %zu", workspace_bytes, need);
    const int nn = static_cast<int>(n);
    const int cb = static_cast<int>((n + kMvCols - 1) / kMvCols), rb = static_cast<int>((n + kMvRows - 1) / kMvRows);
    double* row_part = static_cast<double*>(workspace);
    double* col_part = row_part + static_cast<size_t>(cb) * n;
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        matvec_part_kernel<<<dim3(cb, rb), kMvThreads, 0, stream>>>(P, ldp, W, ldw, nn, x, y, row_part, col_part);
        FUGAL_TRY(launch_check("fugal_plan_matvec: partials"));
    }
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        const unsigned blocks = static_cast<unsigned>((n + 31) / 32);
        merge_add_kernel<<<blocks, 256, 0, stream>>>(row_part, cb, nn, Py, 0);
        merge_add_kernel<<<blocks, 256, 0, stream>>>(col_part, rb, nn, Ptx, 0);
        FUGAL_TRY(launch_check("fugal_plan_matvec: merge"));
    }
    return FUGAL_OK;
}

extern "C" fugal_status fugal_sinkhorn_adjoint(const float* P, int64_t ldp, const float* G, int64_t ldg, int64_t n,
                                               const double* alpha, const double* beta, double scale, float* out,
                                               int64_t ldo, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (P == nullptr || G == nullptr || alpha == nullptr || beta == nullptr || out == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_adjoint: null argument");
    if (n <= 0 || ldp < n || ldg < n || ldo < n) return fail(FUGAL_BAD_SHAPE, "fugal_sinkhorn_adjoint: bad shape");
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    adjoint_kernel<<<ew2d(n), 256, 0, stream>>>(P, ldp, G, ldg, static_cast<int>(n), alpha, beta, scale, out, ldo);
    return launch_check("fugal_sinkhorn_adjoint");
}

namespace {
int cg_ctas(int64_t n) { return static_cast<int>(std::min<int64_t>(sm_count(), n)); }
}  // namespace

extern "C" fugal_status fugal_sinkhorn_adjoint_solve_workspace_size(int64_t n, size_t* bytes) {
    if (bytes == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_adjoint_solve_workspace_size: null output");
    if (n <= 0 || n > FUGAL_ADJOINT_SOLVE_MAX_N)
        return fail(FUGAL_BAD_SHAPE, "fugal_sinkhorn_adjoint_solve_workspace_size: n must be in [1, %d]",
                    FUGAL_ADJOINT_SOLVE_MAX_N);
    // barrier and status words, dot products, column residual, column partials
    *bytes = 256 + static_cast<size_t>(2 * cg_ctas(n) + n + cg_ctas(n) * n) * 8;
    return FUGAL_OK;
}

extern "C" fugal_status fugal_sinkhorn_adjoint_solve(const float* P, int64_t ldp, int64_t n, const double* a,
                                                     const double* b, double tol, int max_iter, double* alpha,
                                                     double* beta, double* info, void* workspace,
                                                     size_t workspace_bytes, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const char* who = "fugal_sinkhorn_adjoint_solve";
    static_assert(kCgMaxN == FUGAL_ADJOINT_SOLVE_MAX_N, "the header's limit");
    size_t need = 0;
    FUGAL_TRY(fugal_sinkhorn_adjoint_solve_workspace_size(n, &need));
    if (P == nullptr || a == nullptr || b == nullptr || alpha == nullptr || beta == nullptr || info == nullptr ||
        workspace == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "%s: null argument", who);
    if (ldp < n) return fail(FUGAL_BAD_SHAPE, "%s: ldp < n", who);
    if (workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 7u) != 0)
        return fail(FUGAL_WORKSPACE_TOO_SMALL, "%s: workspace %zu < %zu bytes", who, workspace_bytes, need);
    CgArgs args{};
    args.P = P;
    args.ldp = ldp;
    args.n = static_cast<int>(n);
    int ctas = cg_ctas(n);
    args.own = static_cast<int>((n + ctas - 1) / ctas);
    if (args.own > kCgMaxOwn) return fail(FUGAL_UNSUPPORTED, "%s: too few SMs for n = %lld", who, (long long)n);
    ctas = static_cast<int>((n + args.own - 1) / args.own);
    args.a = a;
    args.b = b;
    args.tol = tol;
    args.max_iter = max_iter;
    args.alpha = alpha;
    args.beta = beta;
    args.info = info;
    char* w = static_cast<char*>(workspace);
    args.arrivals = reinterpret_cast<unsigned*>(w);
    args.status = reinterpret_cast<int*>(w + 8);
    args.dots = reinterpret_cast<double*>(w + 256);
    args.r_cols = args.dots + 2 * cg_ctas(n);
    args.colpart = args.r_cols + n;
    args.wait_limit_ns = test_wait_limit_ns();
    args.fault_barrier = test_fault_barrier();
    FUGAL_TRY(cuda_check(cudaMemsetAsync(w, 0, 256, stream), who));
    // float4 rows: aligned, and whole quads (else one column per lane and load)
    const bool vec = (n % 4) == 0 && (ldp % 4) == 0 && aligned16(P);
    void (*fn)(CgArgs) = vec ? cg_kernel<true> : cg_kernel<false>;
    const size_t span = kCgThreads * 4;
    const size_t smem = (static_cast<size_t>(n) + span - 1) / span * span * 8;
    FUGAL_TRY(allow_dynamic_smem(fn, smem, who));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(kCgThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        FUGAL_TRY(cuda_check(cudaLaunchKernelEx(&cfg, fn, args), who));
    }
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    cg_end_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(args.status, args.n, alpha, beta, info);
    return launch_check(who);
}

extern "C" fugal_status fugal_sinkhorn_unrolled_workspace_size(int64_t n, size_t* bytes) {
    if (bytes == nullptr) return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_unrolled_workspace_size: null output");
    if (n <= 0 || n > (1ll << 30)) return fail(FUGAL_BAD_SHAPE, "fugal_sinkhorn_unrolled_workspace_size: bad n");
    *bytes = partials_bytes(n, unrolled_rows(n));
    return FUGAL_OK;
}

extern "C" fugal_status fugal_sinkhorn_unrolled_step_backward(const float* K, int64_t ldk, int64_t n,
                                                              const float* out_dual, const float* other_dual,
                                                              const double* g, int axis, float* gK, int64_t ldg,
                                                              double* g_other, void* workspace,
                                                              size_t workspace_bytes, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    size_t need = 0;
    FUGAL_TRY(fugal_plan_matvec_workspace_size(n, &need));
    if (K == nullptr || out_dual == nullptr || other_dual == nullptr || g == nullptr || gK == nullptr ||
        g_other == nullptr || workspace == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_unrolled_step_backward: null argument");
    if (axis != 0 && axis != 1) return fail(FUGAL_BAD_ARGUMENT, "fugal_sinkhorn_unrolled_step_backward: axis 0 or 1");
    if (ldk < n || ldg < n) return fail(FUGAL_BAD_SHAPE, "fugal_sinkhorn_unrolled_step_backward: bad shape");
    if (workspace_bytes < need)
        return fail(FUGAL_WORKSPACE_TOO_SMALL, "fugal_sinkhorn_unrolled_step_backward: workspace too small");
    const int nn = static_cast<int>(n);
    int rows = unrolled_rows(n);  // larger blocks where the workspace holds fewer partials
    while (rows < kMvRows && partials_bytes(n, rows) > workspace_bytes) rows *= 2;
    const int cb = static_cast<int>((n + kMvCols - 1) / kMvCols), rb = static_cast<int>((n + rows - 1) / rows);
    double* row_part = static_cast<double*>(workspace);
    double* col_part = row_part + static_cast<size_t>(cb) * n;
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        auto kernel = rows == 8    ? unrolled_step_kernel<8>
                      : rows == 16 ? unrolled_step_kernel<16>
                      : rows == 32 ? unrolled_step_kernel<32>
                                   : unrolled_step_kernel<kMvRows>;
        kernel<<<dim3(cb, rb), kMvThreads, 0, stream>>>(K, ldk, nn, out_dual, other_dual, g, axis, gK, ldg, row_part,
                                                        col_part);
        FUGAL_TRY(launch_check("fugal_sinkhorn_unrolled_step_backward"));
    }
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        const unsigned blocks = static_cast<unsigned>((n + 31) / 32);
        if (axis == 0)
            merge_add_kernel<<<blocks, 256, 0, stream>>>(row_part, cb, nn, g_other, 1);
        else
            merge_add_kernel<<<blocks, 256, 0, stream>>>(col_part, rb, nn, g_other, 1);
        FUGAL_TRY(launch_check("fugal_sinkhorn_unrolled_step_backward: merge"));
    }
    return FUGAL_OK;
}
