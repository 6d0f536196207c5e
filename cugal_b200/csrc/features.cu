// Graph structure kernels: CSR construction and the four FUGAL node features.
//   fugal_create_adjacency            cuda_kernels/adjacency.cu:163-259 (CUB sort + row pointers)
//   fugal_graph_features              cuda_kernels/feature_extraction.cu:13-84
//   fugal_average_neighbor_features   cuda_kernels/feature_extraction.cu:86-125
//
// Triangle counts are integer and exact: t(v) = sum over u in N(v) of
// |N(v) & N(u)|, one warp per 32 consecutive CSR edges (v, u) whatever rows they
// belong to, so a hub's edges spread over many warps; the lanes share each
// intersection (the elements of the shorter list, searched in the longer one).
// The clustering ratio uses the IEEE-rounded FP32 division.  Neighbour averages
// keep the reference's sequential FP32 sum in CSR order (one warp per vertex, the
// values fetched by its lanes), so they are bit-reproducible.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "fugal_common.cuh"
#include "fugal_host.h"

namespace fugal {

__device__ __forceinline__ int lower_bound(const int* __restrict__ col, int lo, int hi, int x) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (col[mid] < x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Vertices of up to this degree have counts below 2^32: a list of d entries meets d others, each in
// at most d places.
constexpr int kMaxDegree32 = 65535;

__global__ void __launch_bounds__(256) clear_counts_kernel(int n, unsigned* tri, unsigned* carry) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) tri[v] = carry[v] = 0u;
}

// Adds to tri[v] the common neighbours of the edges (v, u) of one chunk of 32 edges.
// Count: 64-bit counts (long long), or 32-bit ones with the wraps of rows longer than
// kMaxDegree32 (parallel edges: a simple graph of 65536 vertices has none) in `carry`.  Lists
// of up to 32 entries are intersected in registers (five shuffles a binary search);
// longer ones are searched in memory by lanes that share the shorter list.  One warp
// per vertex, lanes over its neighbours, left a power-law graph's hubs to single
// warps: 904 us at 65536 vertices of mean degree 16.
template <typename Count>
__global__ void __launch_bounds__(256) triangle_kernel(const int* __restrict__ col, const int* __restrict__ rp, int n,
                                                       Count* tri, unsigned* carry) {
    const int lane = threadIdx.x & 31;
    const int nnz = rp[n];
    const long long chunk = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const long long chunks = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
    for (long long ch = chunk; ch * 32 < nnz; ch += chunks) {
        const int e0 = static_cast<int>(ch * 32), e1 = min(nnz, e0 + 32);
        // this lane's edge: its neighbour and the neighbour's list
        const int u = e0 + lane < e1 ? col[e0 + lane] : 0;
        const int us = e0 + lane < e1 ? rp[u] : 0, ue = e0 + lane < e1 ? rp[u + 1] : 0;
        int v = lower_bound(rp, 0, n + 1, e0 + 1) - 1;  // the row of edge e0 (rp[v] <= e0 < rp[v + 1])
        int e = e0;
        while (e < e1) {
            const int s = rp[v], t = rp[v + 1];
            if (t <= e) {
                ++v;
                continue;
            }
            const int d = t - s;
            const int a = (d <= 32 && lane < d) ? col[s + lane] : INT_MAX;
            const int stop = min(t, e1);
            Count count = 0;
            for (; e < stop; ++e) {
                const int bs = __shfl_sync(0xffffffffu, us, e - e0), be = __shfl_sync(0xffffffffu, ue, e - e0);
                const int db = be - bs;
                if (d <= 32 && db <= 32) {
                    const int b = lane < db ? col[bs + lane] : INT_MAX;
                    const int x = db < d ? b : a, hay = db < d ? a : b;  // shorter in longer, INT_MAX past the end
                    int pos = 0;                                         // entries of hay below x
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1) {
                        const int y = __shfl_sync(0xffffffffu, hay, pos + step - 1);
                        if (y < x) pos += step;
                    }
                    const int y = __shfl_sync(0xffffffffu, hay, pos);
                    count += (x != INT_MAX && y == x) ? 1 : 0;
                } else {
                    int ss = s, st = t, ls = bs, lt = be;  // shorter, longer
                    if (db < d) {
                        ss = bs; st = be; ls = s; lt = t;
                    }
                    for (int k = ss + lane; k < st; k += 32) {
                        const int x = col[k];
                        const int q = lower_bound(col, ls, lt, x);
                        count += (q < lt && col[q] == x) ? 1 : 0;
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
            if (lane == 0 && count) {
                if (sizeof(Count) == 8 || d <= kMaxDegree32) {
                    atomicAdd(&tri[v], count);
                } else if (atomicAdd(&tri[v], count) > ~count) {
                    atomicAdd(&carry[v], 1u);
                }
            }
            ++v;
        }
    }
}

// 32-bit counts lie in clustering, their carries in degrees (read as the floats that they are
// overwritten with, so that the compiler keeps the order).
template <typename Count>
__global__ void clustering_kernel(const int* __restrict__ rp, int n, const Count* tri, float* clustering,
                                  float* degrees, int* degree_counts) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const int d = rp[v + 1] - rp[v];
        long long t = static_cast<long long>(tri[v]);
        if (sizeof(Count) == 4 && d > kMaxDegree32) t += static_cast<long long>(__float_as_uint(degrees[v])) << 32;
        degrees[v] = static_cast<float>(d);
        if (degree_counts) degree_counts[v] = d;
        const float denom = static_cast<float>(static_cast<long long>(d) * (d - 1));
        clustering[v] = (t == 0 || d < 2) ? 0.0f : __fdiv_rn(static_cast<float>(t), denom);
    }
}

// Counts without a buffer of 64-bit ones and vertices whose count may pass 32 bits.
__global__ void graph_features_kernel(const int* __restrict__ col, const int* __restrict__ rp, int n,
                                      float* clustering, float* degrees, int* degree_counts) {
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
        const int s = rp[v], e = rp[v + 1];
        const int d = e - s;
        long long t = 0;
        for (int idx = s + lane; idx < e; idx += 32) {
            const int u = col[idx];
            const int us = rp[u], ue = rp[u + 1];
            int as = s, ae = e, bs = us, be = ue;  // search the shorter list in the longer
            if (ue - us < e - s) {
                as = us; ae = ue; bs = s; be = e;
            }
            int cnt = 0;
            for (int k = as; k < ae; ++k) {
                const int x = col[k];
                const int pos = lower_bound(col, bs, be, x);
                cnt += (pos < be && col[pos] == x) ? 1 : 0;
            }
            t += cnt;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) {
            degrees[v] = static_cast<float>(d);
            if (degree_counts) degree_counts[v] = d;
            const float denom = static_cast<float>(static_cast<long long>(d) * (d - 1));
            clustering[v] = (t == 0 || d < 2) ? 0.0f : __fdiv_rn(static_cast<float>(t), denom);
        }
    }
}

// One warp per vertex: lanes fetch 32 neighbours' values (the next 32 already in
// flight), then every lane adds them in CSR order.
__global__ void average_neighbor_kernel(const int* __restrict__ col, const int* __restrict__ rp, int n,
                                        const float* __restrict__ f, float* avg) {
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
        const int s = rp[v], e = rp[v + 1];
        float sum = 0.0f;
        float x = s + lane < e ? f[col[s + lane]] : 0.0f;
        for (int k = s; k < e; k += 32) {
            const float next = k + 32 + lane < e ? f[col[k + 32 + lane]] : 0.0f;
            const int cnt = min(32, e - k);
            if (cnt == 32) {
#pragma unroll
                for (int q = 0; q < 32; ++q) sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, x, q));
            } else {
                for (int q = 0; q < cnt; ++q) sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, x, q));
            }
            x = next;
        }
        const int d = e - s;
        if (lane == 0) avg[v] = d == 0 ? 0.0f : __fdiv_rn(sum, static_cast<float>(d));
    }
}

// ---------------------------------------------------------------- CSR build

__global__ void count_rows_kernel(const int* edges, long long m, int n, int* counts, int* bad) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m; e += (long long)gridDim.x * blockDim.x) {
        const int x = edges[2 * e], y = edges[2 * e + 1];
        if (x < 0 || x >= n || y < 0 || y >= n) {
            atomicExch(bad, 1);
            continue;
        }
        atomicAdd(&counts[y], 1);
    }
}

// Exclusive scan of counts[0..n) into rp[0..n], 1024 counts per block (more above 262144); a
// block first adds up all counts before its own, 4 n bytes at most, read by all SMs at once.
// 7 us at n = 65536, 51 when one block walked all counts.
constexpr int kScanBlocks = 256;

// Inclusive scan of one value per thread over a 1024-thread block; returns the block's total in `total`.
__device__ __forceinline__ int block_scan_1024(int x, int* warp_tot, int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        warp_tot[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    total = warp_tot[31];
    incl += warp > 0 ? warp_tot[warp - 1] : 0;
    __syncthreads();  // warp_tot is read
    return incl;
}

__global__ void __launch_bounds__(1024) scan_rows_kernel(const int* counts, int n, int* rp, int* cursor) {
    __shared__ int warp_tot[32];
    const int per = (n + gridDim.x - 1) / gridDim.x;  // counts per block: 1024 unless there are too many
    const int begin = min(n, static_cast<int>(blockIdx.x) * per), end = min(n, begin + per);
    int sum = 0;
#pragma unroll 8
    for (int i = threadIdx.x; i < begin; i += 1024) sum += counts[i];
    int carry = 0;
    block_scan_1024(sum, warp_tot, carry);
    for (int base = begin; base < end; base += 1024) {
        const int i = base + threadIdx.x;
        const int x = i < end ? counts[i] : 0;
        int total = 0;
        const int excl = carry + block_scan_1024(x, warp_tot, total) - x;
        if (i < end) {
            rp[i] = excl;
            cursor[i] = excl;
        }
        carry += total;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) rp[n] = carry;
}

__global__ void scatter_cols_kernel(const int* edges, long long m, int n, int* cursor, int* col) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m; e += (long long)gridDim.x * blockDim.x) {
        const int x = edges[2 * e], y = edges[2 * e + 1];
        if (x < 0 || x >= n || y < 0 || y >= n) continue;
        const int pos = atomicAdd(&cursor[y], 1);
        col[pos] = x;
    }
}

// Sort each row's columns ascending.  Rows of up to 32 entries: one warp each, every
// entry stored at its rank (entries below it, ties by position); a 512-thread block
// per such row was 303 us at 65536 rows of mean length 16.
__global__ void __launch_bounds__(256) sort_short_rows_kernel(const int* rp, int n, int* col) {
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += warps) {
        const int s = rp[r], d = rp[r + 1] - s;
        if (d <= 1 || d > 32) continue;
        const int x = lane < d ? col[s + lane] : INT_MAX;
        int rank = 0;
        for (int k = 0; k < d; ++k) {
            const int y = __shfl_sync(0xffffffffu, x, k);
            rank += (y < x || (y == x && k < lane)) ? 1 : 0;
        }
        if (lane < d) col[s + rank] = x;
    }
}

// Longer rows: bitonic sort in shared memory, one block per row, rows up to
// kMaxSortRow entries (longer rows raise a flag).
constexpr int kMaxSortRow = 8192;

__global__ void __launch_bounds__(512) sort_rows_kernel(const int* rp, int n, int* col, int* bad) {
    __shared__ int buf[kMaxSortRow];
    __shared__ int found[512], nfound;
    // 512 rows at a time, strided over the blocks (hubs are often neighbours): the long ones
    for (long long base = blockIdx.x; base < n; base += 512ll * gridDim.x) {
      if (threadIdx.x == 0) nfound = 0;
      __syncthreads();
      const long long mine = base + static_cast<long long>(threadIdx.x) * gridDim.x;
      if (mine < n && rp[mine + 1] - rp[mine] > 32) found[atomicAdd(&nfound, 1)] = static_cast<int>(mine);
      __syncthreads();
      const int rows = nfound;
      for (int q = 0; q < rows; ++q) {
        const int r = found[q];
        const int s = rp[r], e = rp[r + 1], d = e - s;
        if (d > kMaxSortRow) {
            if (threadIdx.x == 0) atomicExch(bad, 2);
            continue;
        }
        int size = 1;
        while (size < d) size <<= 1;
        for (int i = threadIdx.x; i < size; i += blockDim.x) buf[i] = i < d ? col[s + i] : INT_MAX;
        __syncthreads();
        for (int k = 2; k <= size; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = threadIdx.x; i < size; i += blockDim.x) {
                    const int ij = i ^ j;
                    if (ij > i) {
                        const bool up = (i & k) == 0;
                        const int a = buf[i], b = buf[ij];
                        if ((a > b) == up) {
                            buf[i] = b;
                            buf[ij] = a;
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (int i = threadIdx.x; i < d; i += blockDim.x) col[s + i] = buf[i];
        __syncthreads();
      }
      __syncthreads();  // found is read
    }
}

}  // namespace fugal

using namespace fugal;

extern "C" fugal_status fugal_graph_features(const int32_t* col_indices, const int32_t* row_pointers, int64_t n,
                                             float* clustering, float* degrees, int32_t* degree_counts,
                                             int64_t* triangle_counts, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (row_pointers == nullptr || clustering == nullptr || degrees == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_graph_features: null argument");
    if (n <= 0 || n > INT_MAX - 1) return fail(FUGAL_BAD_SHAPE, "fugal_graph_features: bad n");
    const int threads = 256;
    const int ni = static_cast<int>(n);
    const int blocks = static_cast<int>(std::min<int64_t>((n * 32 + threads - 1) / threads, 32 * sm_count()));
    const int vec_blocks = static_cast<int>(std::min<int64_t>((n + threads - 1) / threads, 8 * sm_count()));
    const int chunk_blocks = static_cast<int>(std::min<int64_t>((n + 15) / 16 + 1, 16 * sm_count()));
    // Up to 65536 vertices a count is kept in 32 bits, in the vertex's clustering entry, until the
    // ratio is formed, and what does not fit them in its degree entry.
    if (triangle_counts != nullptr) {
        long long* tri = reinterpret_cast<long long*>(triangle_counts);
        FUGAL_TRY(cuda_check(cudaMemsetAsync(tri, 0, static_cast<size_t>(n) * 8, stream), "fugal_graph_features"));
        {
            LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
            triangle_kernel<unsigned long long><<<chunk_blocks, threads, 0, stream>>>(
                col_indices, row_pointers, ni, reinterpret_cast<unsigned long long*>(tri), nullptr);
            FUGAL_TRY(launch_check("fugal_graph_features: triangles"));
        }
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        clustering_kernel<long long><<<vec_blocks, threads, 0, stream>>>(row_pointers, ni, tri, clustering, degrees,
                                                                         degree_counts);
        return launch_check("fugal_graph_features");
    }
    if (n <= 65536) {
        unsigned* tri = reinterpret_cast<unsigned*>(clustering);
        unsigned* carry = reinterpret_cast<unsigned*>(degrees);
        {
            LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
            clear_counts_kernel<<<vec_blocks, threads, 0, stream>>>(ni, tri, carry);
            FUGAL_TRY(launch_check("fugal_graph_features: clear"));
        }
        {
            LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
            triangle_kernel<unsigned><<<chunk_blocks, threads, 0, stream>>>(col_indices, row_pointers, ni, tri, carry);
            FUGAL_TRY(launch_check("fugal_graph_features: triangles"));
        }
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        clustering_kernel<unsigned><<<vec_blocks, threads, 0, stream>>>(row_pointers, ni, tri, clustering, degrees,
                                                                        degree_counts);
        return launch_check("fugal_graph_features");
    }
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    graph_features_kernel<<<blocks, threads, 0, stream>>>(col_indices, row_pointers, ni, clustering, degrees,
                                                          degree_counts);
    return launch_check("fugal_graph_features");
}

extern "C" fugal_status fugal_average_neighbor_features(const int32_t* col_indices, const int32_t* row_pointers,
                                                        int64_t n, const float* features, float* averages,
                                                        fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (row_pointers == nullptr || features == nullptr || averages == nullptr)
        return fail(FUGAL_BAD_ARGUMENT, "fugal_average_neighbor_features: null argument");
    if (n <= 0 || n > INT_MAX - 1) return fail(FUGAL_BAD_SHAPE, "fugal_average_neighbor_features: bad n");
    const int blocks = static_cast<int>(std::min<int64_t>((n + 7) / 8, 16 * sm_count()));
    LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
    average_neighbor_kernel<<<blocks, 256, 0, stream>>>(col_indices, row_pointers, static_cast<int>(n), features,
                                                        averages);
    return launch_check("fugal_average_neighbor_features");
}

extern "C" fugal_status fugal_create_adjacency_workspace_size(int64_t edge_count, int64_t node_count,
                                                              size_t* bytes) {
    if (bytes == nullptr) return fail(FUGAL_BAD_ARGUMENT, "fugal_create_adjacency_workspace_size: null output");
    if (edge_count < 0 || node_count <= 0 || node_count > INT_MAX - 1)
        return fail(FUGAL_BAD_SHAPE, "fugal_create_adjacency_workspace_size: bad sizes");
    // counts [n+1], cursor [n+1], flag word
    *bytes = static_cast<size_t>(2 * (node_count + 1) + 4) * sizeof(int);
    return FUGAL_OK;
}

extern "C" fugal_status fugal_create_adjacency(const int32_t* edges, int64_t edge_count, int64_t node_count,
                                               int32_t* col_indices, int32_t* row_pointers, void* workspace,
                                               size_t workspace_bytes, fugal_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    size_t need = 0;
    FUGAL_TRY(fugal_create_adjacency_workspace_size(edge_count, node_count, &need));
    if (row_pointers == nullptr || workspace == nullptr || (edge_count > 0 && (edges == nullptr || col_indices == nullptr)))
        return fail(FUGAL_BAD_ARGUMENT, "fugal_create_adjacency: null argument");
    if (workspace_bytes < need)
        return fail(FUGAL_WORKSPACE_TOO_SMALL, "fugal_create_adjacency: workspace %zu < %zu", workspace_bytes, need);
    const int n = static_cast<int>(node_count);
    int* counts = static_cast<int*>(workspace);
    int* cursor = counts + (n + 1);
    int* bad = cursor + (n + 1);
    FUGAL_TRY(cuda_check(cudaMemsetAsync(counts, 0, need, stream), "fugal_create_adjacency: clear"));
    const int blocks = static_cast<int>(std::min<int64_t>((edge_count + 255) / 256 + 1, 8 * sm_count()));
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        count_rows_kernel<<<blocks, 256, 0, stream>>>(edges, edge_count, n, counts, bad);
        FUGAL_TRY(launch_check("fugal_create_adjacency: count"));
    }
    {
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        const int blocks1024 = std::min((n + 1023) / 1024, kScanBlocks);
        scan_rows_kernel<<<blocks1024, 1024, 0, stream>>>(counts, n, row_pointers, cursor);
        FUGAL_TRY(launch_check("fugal_create_adjacency: scan"));
    }
    if (edge_count > 0) {
        {
            LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
            scatter_cols_kernel<<<blocks, 256, 0, stream>>>(edges, edge_count, n, cursor, col_indices);
            FUGAL_TRY(launch_check("fugal_create_adjacency: scatter"));
        }
        {
            LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
            const int wblocks = static_cast<int>(std::min<int64_t>((node_count + 7) / 8, 16 * sm_count()));
            sort_short_rows_kernel<<<wblocks, 256, 0, stream>>>(row_pointers, n, col_indices);
            FUGAL_TRY(launch_check("fugal_create_adjacency: short rows"));
        }
        LaunchScope scope(FUGAL_KERNEL_OTHER, stream);
        const int sblocks = static_cast<int>(std::min<int64_t>(n, 8 * sm_count()));
        sort_rows_kernel<<<sblocks, 512, 0, stream>>>(row_pointers, n, col_indices, bad);
        FUGAL_TRY(launch_check("fugal_create_adjacency: sort"));
    }
    return FUGAL_OK;
}
