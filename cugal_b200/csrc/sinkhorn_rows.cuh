// Device pieces shared by the row-owned persistent Sinkhorn kernels (sinkhorn_rows.cu,
// log domain; sinkhorn_standard.cu, scaling form): row streams, per-thread column state,
// the FP64 reduction of the CTAs' column sums.
#pragma once

#include <type_traits>

#include "fugal_common.cuh"
#include "sinkhorn_rows.h"
#include "sinkhorn_state.cuh"

namespace fugal {

constexpr int kRowsThreads = 512;
constexpr int kRowsWarps = kRowsThreads / 32;
constexpr int kRowsMaxRows = 256;      // rows per CTA the row-dual staging holds
constexpr int kRowsStatic = 24 * 1024; // shared memory kept for the static arrays
// Eight streams (rows of up to 4096 columns) leave room for all their column sums next to the
// stages; fewer meet 8 columns per thread at a time in `colred` (meet_streams).
constexpr size_t rows_dump_bytes(int streams, int ept) {
    return streams == 8 ? static_cast<size_t>(kRowsThreads) * ept * 4 : 0;
}

// Barrier over the GT threads of stream g; true if every thread voted true.
template <int GT>
FUGAL_DEVICE bool stream_and(bool ok, int g) {
    if constexpr (GT == kRowsThreads) {
        return __syncthreads_and(ok) != 0;
    } else {
        uint32_t out;
        asm volatile(
            "{\n .reg .pred p, q;\n"
            " setp.ne.u32 q, %1, 0;\n"
            " barrier.cta.red.and.aligned.pred p, %2, %3, q;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(out)
            : "r"(static_cast<uint32_t>(ok)), "r"(g + 1), "n"(GT)
            : "memory");
        return out != 0;
    }
}

// Sum of GW per-warp values in a fixed pairwise order.
template <int GW>
FUGAL_DEVICE float sum_warps(const float* r) {
    if constexpr (GW == 2) {
        const float2 a = *reinterpret_cast<const float2*>(r);
        return a.x + a.y;
    } else {
        float s[GW / 4];
#pragma unroll
        for (int i = 0; i < GW / 4; ++i) {
            const float4 a = reinterpret_cast<const float4*>(r)[i];
            s[i] = (a.x + a.y) + (a.z + a.w);
        }
        if constexpr (GW == 4) return s[0];
        else if constexpr (GW == 8) return s[0] + s[1];
        else return (s[0] + s[1]) + (s[2] + s[3]);
    }
}

// 16 elements of a staged row (chunk c of this thread) as 8 float pairs.
template <typename T, int GT>
FUGAL_DEVICE void load16(const T* stage, int c, int gt, float2* v) {
    constexpr int V = Vec<T>::N;
#pragma unroll
    for (int i = 0; i < 16 / V; ++i)
        Pairs<T>::unpack(*reinterpret_cast<const uint4*>(stage + ((c * (16 / V) + i) * GT + gt) * V), v + i * V / 2);
}

// Column sums and column duals (b log2 e) of a thread's EPT columns: in registers
// up to 32 columns, else in tensor memory, 16 columns per access.
template <int EPT, bool REG = (EPT <= 32)>
struct ColumnState;

template <int EPT>
struct ColumnState<EPT, true> {
    static constexpr uint32_t kTmemColumns = 0;
    float2 sum[EPT / 2], dual[EPT / 2];
    FUGAL_DEVICE void start(uint32_t, int) {}
    // 16 duals b of chunk c; their sums start at 0
    FUGAL_DEVICE void set(int c, const float* b) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            dual[8 * c + q] = make_float2(b[2 * q], b[2 * q + 1]);
            sum[8 * c + q] = make_float2(0.f, 0.f);
        }
    }
    FUGAL_DEVICE void ready() {}
    FUGAL_DEVICE void settle() {}
    FUGAL_DEVICE void duals(int c, float2* b) const {
#pragma unroll
        for (int q = 0; q < 8; ++q) b[q] = dual[8 * c + q];
    }
    // adds the pending row's chunk y (weight w) to the sums of chunk c
    FUGAL_DEVICE void add(int c, const float2* y, float w) {
#pragma unroll
        for (int q = 0; q < 8; ++q) sum[8 * c + q] = __ffma2_rn(y[q], make_float2(w, w), sum[8 * c + q]);
    }
    FUGAL_DEVICE void total(int c, const float2* y, float w, float* out) {
        add(c, y, w);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            out[2 * q] = sum[8 * c + q].x;
            out[2 * q + 1] = sum[8 * c + q].y;
        }
    }
};

template <int EPT>
struct ColumnState<EPT, false> {
    static constexpr uint32_t kTmemColumns = 512;  // 4 warps per lane quarter x (sums + duals) x EPT <= 64
    uint32_t tsum, tdual;
    FUGAL_DEVICE void start(uint32_t base, int warp) {
        tsum = base + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + static_cast<uint32_t>((warp >> 2) * EPT);
        tdual = tsum + static_cast<uint32_t>((kRowsThreads / 128) * EPT);
    }
    FUGAL_DEVICE void set(int c, const float* b) {
        float z[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) z[k] = 0.f;
        tmem_st16(tdual + 16 * c, b);
        tmem_st16(tsum + 16 * c, z);
    }
    FUGAL_DEVICE void ready() { tmem_wait_st(); }
    // Tensor memory orders a load after a store of the same thread only through a wait: called
    // once per row before its sums are added to and once before they are read out, when the
    // stores of the row before have a reduction and a barrier behind them.
    FUGAL_DEVICE void settle() { tmem_wait_st(); }
    FUGAL_DEVICE void duals(int c, float2* b) const {
        float v[16];
        tmem_ld16(tdual + 16 * c, v);
#pragma unroll
        for (int q = 0; q < 8; ++q) b[q] = make_float2(v[2 * q], v[2 * q + 1]);
    }
    FUGAL_DEVICE void total(int c, const float2* y, float w, float* out) {
        tmem_ld16(tsum + 16 * c, out);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float2 a2 = __ffma2_rn(y[q], make_float2(w, w), make_float2(out[2 * q], out[2 * q + 1]));
            out[2 * q] = a2.x;
            out[2 * q + 1] = a2.y;
        }
    }
    FUGAL_DEVICE void add(int c, const float2* y, float w) {
        float acc[16];
        total(c, y, w, acc);
        tmem_st16(tsum + 16 * c, acc);
    }
};

// The column sums of GR = 2 or 4 streams: every thread holds 16 sums (chunk c) of its
// stream; their totals go to prow, neighbouring streams first.  8 columns of every thread
// meet at a time, 8 GT consecutive ones, in 16 KB of shared memory.  A partial row per
// stream instead made the exchange half of a sweep at n = 8192 BF16 (4 streams): the CTAs'
// FP64 sums 16400 cycles and the writes 8000, against 8200 and 5000.
// Neighbours first is a choice among orders that are equally exact.  It is kept fixed because an
// alignment at a small regularization follows the last bits: over 150 steps on the 1000-node
// Newman-Watts graph eight orders ended at node accuracies 2 points apart, and two of the eight left
// the 1.5 points around the reference's result that tests/test_gpu_accuracy.py allows.
template <int GR, int GT, int V>
FUGAL_DEVICE void meet_streams(float* meet, const float* acc, int c, int g, int gt, int n, float* prow) {
    static_assert(GR == 2 || GR == 4, "a thread adds 8 / GR columns, at least 2");
    constexpr int W = 8 / GR;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        __syncthreads();  // the columns before have been read
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int at = (4 * k / V) * GT * V + gt * V + 4 * k % V;
            const float* a4 = acc + 8 * h + 4 * k;
            *reinterpret_cast<float4*>(meet + g * GT * 8 + at) = make_float4(a4[0], a4[1], a4[2], a4[3]);
        }
        __syncthreads();
        const int at = static_cast<int>(threadIdx.x) * W;
        const int j = (16 * c + 8 * h) * GT + at;
        float v[GR][W];
#pragma unroll
        for (int k = 0; k < GR; ++k) {
#pragma unroll
            for (int q = 0; q < W; q += 2) {
                const float2 f = *reinterpret_cast<const float2*>(meet + k * GT * 8 + at + q);
                v[k][q] = f.x;
                v[k][q + 1] = f.y;
            }
        }
#pragma unroll
        for (int o = 1; o < GR; o <<= 1) {
#pragma unroll
            for (int k = 0; k < GR; k += 2 * o) {
#pragma unroll
                for (int q = 0; q < W; ++q) v[k][q] += v[k + o][q];
            }
        }
        if (j < n) {  // partial rows are n_pad wide, a multiple of 64 columns
#pragma unroll
            for (int q = 0; q < W; q += 2) *reinterpret_cast<float2*>(prow + j + q) = make_float2(v[0][q], v[0][q + 1]);
        }
    }
}

// FP64 sums of this CTA's share of the columns over `parts` partial rows: on return
// thread t < 4 * per holds the sum of column 4 * per * blockIdx.x + t (others: 0).
// Lanes of a warp: cgp column quads (a power of two) x the rest over partial rows;
// all of a thread's loads in flight (they come from L2): at most 4 up to 8192 columns
// on 148 SMs, 10 per round above.  Grids of at least n / 256 CTAs.
FUGAL_DEVICE int columns_per_cta(int n) {
    const int quads = (n + 3) / 4;
    return 4 * ((quads + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x));
}
FUGAL_DEVICE double own_column_sum(const float* partials, long long n_pad, int parts, int n,
                                   double (*colred)[128]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quads = (n + 3) / 4;
    const int per = columns_per_cta(n) / 4;
    int cgp = 1;
    while (cgp < per) cgp <<= 1;
    const int cg = tid & (cgp - 1);
    const int q0 = blockIdx.x * per;
    const bool mine = cg < per && q0 + cg < quads;
    const int step = kRowsThreads / cgp;
    double cs[4] = {0.0, 0.0, 0.0, 0.0};
    const float* src = partials + (q0 + cg) * 4;
    auto add_rows = [&](auto unroll) {
        constexpr int U = decltype(unroll)::value;
        for (int k0 = tid / cgp; k0 < parts; k0 += U * step) {
            float4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = k0 + u * step;
                v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (mine && k < parts)
                    v[u] = __ldcg(reinterpret_cast<const float4*>(src + static_cast<size_t>(k) * n_pad));
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k0 + u * step < parts) {
                    cs[0] += v[u].x;
                    cs[1] += v[u].y;
                    cs[2] += v[u].z;
                    cs[3] += v[u].w;
                }
            }
        }
    };
    if (parts <= 4 * step) add_rows(std::integral_constant<int, 4>{});
    else add_rows(std::integral_constant<int, 10>{});
    for (int o = cgp; o < 32; o <<= 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) cs[q] += __shfl_xor_sync(0xffffffffu, cs[q], o);
    }
    // cgp <= 32: lane l < cgp of every warp holds quad l; cgp = 64: warps alternate quads 0..31, 32..63
    if (lane < cgp) {
#pragma unroll
        for (int q = 0; q < 4; ++q) colred[warp][lane * 4 + q] = cs[q];
    }
    __syncthreads();
    if (tid >= per * 4) return 0.0;
    // pairwise over the warps (the upper half is empty at cgp = 64)
    double h[kRowsWarps];
#pragma unroll
    for (int w = 0; w < kRowsWarps; ++w)
        h[w] = cgp <= 32 ? colred[w][tid] : (w < kRowsWarps / 2 ? colred[2 * w + (tid >> 7)][tid & 127] : 0.0);
#pragma unroll
    for (int o = kRowsWarps / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int w = 0; w < o; ++w) h[w] += h[w + o];
    }
    return h[0];
}

// The sum of errs and the maximum of corrs over the CTAs, the same in every CTA
// (warp 0; all loads in flight up to 256 CTAs).
FUGAL_DEVICE void grid_error(const double* errs, const float* corrs, double& e, float& c) {
    constexpr int U = 8;
    const int lane = threadIdx.x & 31;
    const int ctas = static_cast<int>(gridDim.x);
    e = 0.0;
    c = 0.f;
    for (int k0 = lane; k0 < ctas; k0 += 32 * U) {
        double ev[U];
        float cv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + 32 * u;
            ev[u] = k < ctas ? __ldcg(errs + k) : 0.0;
            cv[u] = corrs != nullptr && k < ctas ? __ldcg(corrs + k) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            e += ev[u];
            c = fmaxf(c, cv[u]);
        }
    }
    e = warp_sum(e);
    c = warp_max_positive(c);
}

}  // namespace fugal
