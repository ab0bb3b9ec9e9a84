// Shared helpers of the yitu_b200 CUDA library (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/yitu_b200.h"

namespace yitu {

void set_error(const char *fmt, ...);

#define YITU_REQUIRE(cond, code, ...)      \
    do {                                   \
        if (!(cond)) {                     \
            ::yitu::set_error(__VA_ARGS__); \
            return (code);                 \
        }                                  \
    } while (0)

#define YITU_CUDA(expr)                                                                              \
    do {                                                                                             \
        cudaError_t e_ = (expr);                                                                     \
        if (e_ != cudaSuccess) {                                                                     \
            ::yitu::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return YITU_ERR_CUDA;                                                                    \
        }                                                                                            \
    } while (0)

#define YITU_LAUNCH_CHECK()                                                                      \
    do {                                                                                         \
        cudaError_t e_ = cudaGetLastError();                                                     \
        if (e_ != cudaSuccess) {                                                                 \
            ::yitu::set_error("kernel launch failed: %s (%s:%d)", cudaGetErrorString(e_), __FILE__, __LINE__); \
            return YITU_ERR_CUDA;                                                                \
        }                                                                                        \
    } while (0)

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

__device__ __forceinline__ int64_t load_ptr(const void *indptr, int is64, int64_t i) {
    return is64 ? __ldg(reinterpret_cast<const int64_t *>(indptr) + i)
                : static_cast<int64_t>(__ldg(reinterpret_cast<const int32_t *>(indptr) + i));
}

__device__ __forceinline__ float leaky_relu(float v, float slope) {
    return fmaxf(0.0f, v) + slope * fminf(0.0f, v);
}

__device__ __forceinline__ float activate(float v, int act) {
    if (act == YITU_ACT_RELU) return fmaxf(v, 0.0f);
    if (act == YITU_ACT_ELU) return v > 0.0f ? v : expm1f(v);
    return v;
}

// Loads of data that is streamed once (indices, edge values): kept out of L1, and marked evict-first in L2 through
// a cache-hint policy, so that they do not push the gathered feature rows out of the 126 MB L2.
__device__ __forceinline__ uint64_t stream_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ int ld_stream(const int *p) {
    int v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(stream_policy()));
    return v;
}
__device__ __forceinline__ float ld_stream(const float *p) {
    float v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(stream_policy()));
    return v;
}

// Row slices of VEC floats: 128-bit or (new with sm_100) 256-bit global loads; streaming stores for outputs.
template <int VEC>
__device__ __forceinline__ void load_vec(float (&r)[VEC], const float *p) {
    if constexpr (VEC == 8) {
        // 256-bit global load (new with sm_100): one request moves 32 bytes per lane, 1 KiB per warp
        asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                     : "l"(p));
    } else if constexpr (VEC == 4) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
        r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
    } else if constexpr (VEC == 2) {
        const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
        r[0] = v.x; r[1] = v.y;
    } else {
        r[0] = __ldg(p);
    }
}

template <int VEC>
__device__ __forceinline__ void store_vec(float *p, const float (&r)[VEC]) {
    // output rows are written once and not read again by this kernel: streaming stores (evict-first)
    if constexpr (VEC == 8) {
        __stcs(reinterpret_cast<float4 *>(p), make_float4(r[0], r[1], r[2], r[3]));
        __stcs(reinterpret_cast<float4 *>(p) + 1, make_float4(r[4], r[5], r[6], r[7]));
    } else if constexpr (VEC == 4) {
        __stcs(reinterpret_cast<float4 *>(p), make_float4(r[0], r[1], r[2], r[3]));
    } else if constexpr (VEC == 2) {
        __stcs(reinterpret_cast<float2 *>(p), make_float2(r[0], r[1]));
    } else {
        __stcs(p, r[0]);
    }
}

// Sums of the hub rows' chunk partials (width W, chunk c at partial + c * stride), handed to finish(row, d, sum).  A CTA of
// 256 threads looks at eight consecutive chunks, one per warp: the warp that finds its row's first chunk adds a row of up to
// 16 chunks by itself, longer rows are shared by the whole CTA, every group of threads taking every groups-th chunk.  Added
// in a fixed order: run-to-run identical.  (One CTA per chunk, most of which leave at once, took 0.95 ms for the chunks of a
// graph of 520 M edges.)  Launch with (n_chunks + 7) / 8 CTAs.
struct HubRows {
    const void *indptr;
    int is64, chunk_edges;
    int64_t n_chunks;
    const int *chunk_row;
    const int64_t *chunk_begin;
};

// VEC = 4 takes W, stride and the partials' address as multiples of four floats.
template <int VEC, typename Finish>
__device__ __forceinline__ void reduce_hub_rows(const HubRows &h, const float *partial, int64_t stride, int64_t W, Finish finish) {
    __shared__ float s_part[256][VEC];
    __shared__ int s_nch[8];
    __shared__ int64_t s_row[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t first = static_cast<int64_t>(blockIdx.x) * 8, chunk = first + w;
    int nch = 0;
    int64_t row = 0;
    if (chunk < h.n_chunks) {
        row = __ldg(h.chunk_row + chunk);
        const int64_t rb = load_ptr(h.indptr, h.is64, row);
        if (__ldg(h.chunk_begin + chunk) == rb)
            nch = static_cast<int>((load_ptr(h.indptr, h.is64, row + 1) - rb + h.chunk_edges - 1) / h.chunk_edges);
    }
    const auto sum = [&](const float *part, int k0, int step, int n, float (&a)[VEC]) {
#pragma unroll
        for (int q = 0; q < VEC; ++q) a[q] = 0.0f;
        for (int k = k0; k < n; k += 8 * step) {
            float v[8][VEC];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (k + u * step < n) {
                    load_vec<VEC>(v[u], part + static_cast<int64_t>(k + u * step) * stride);
                } else {
#pragma unroll
                    for (int q = 0; q < VEC; ++q) v[u][q] = 0.0f;
                }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int q = 0; q < VEC; ++q) a[q] += v[u][q];
        }
    };
    const bool alone = nch <= 16;
    float a[VEC];
    if (alone && nch > 0)
        for (int64_t d = lane * VEC; d < W; d += 32 * VEC) {
            sum(partial + chunk * stride + d, 0, 1, nch, a);
            finish(row, d, a);
        }
    if (lane == 0) {
        s_nch[w] = alone ? 0 : nch;
        s_row[w] = row;
    }
    __syncthreads();
    int cols = 8;
    while (cols * VEC < W && cols < 256) cols <<= 1;
    const int tx = threadIdx.x & (cols - 1), grp = threadIdx.x / cols, groups = 256 / cols;
    for (int i = 0; i < 8; ++i) {
        if (s_nch[i] == 0) continue;
        for (int64_t d0 = 0; d0 < W; d0 += cols * VEC) {
            const int64_t d = d0 + tx * VEC;
#pragma unroll
            for (int q = 0; q < VEC; ++q) a[q] = 0.0f;
            if (d < W) sum(partial + (first + i) * stride + d, grp, groups, s_nch[i], a);
            if (groups > 1) {
#pragma unroll
                for (int q = 0; q < VEC; ++q) s_part[threadIdx.x][q] = a[q];
                __syncthreads();
                if (grp == 0)
                    for (int g = 1; g < groups; ++g)
#pragma unroll
                        for (int q = 0; q < VEC; ++q) a[q] += s_part[g * cols + tx][q];
                __syncthreads();
            }
            if (grp == 0 && d < W) finish(s_row[i], d, a);
        }
    }
}

inline int validate_csr(const yitu_csr_t *g) {
    YITU_REQUIRE(g != nullptr, YITU_ERR_INVALID_ARG, "graph is NULL");
    YITU_REQUIRE(g->n_rows >= 0 && g->n_cols >= 0 && g->nnz >= 0, YITU_ERR_INVALID_ARG,
                 "negative graph size (n_rows=%lld n_cols=%lld nnz=%lld)", (long long)g->n_rows,
                 (long long)g->n_cols, (long long)g->nnz);
    YITU_REQUIRE(g->indptr != nullptr, YITU_ERR_INVALID_ARG, "graph.indptr is NULL");
    YITU_REQUIRE(g->nnz == 0 || g->indices != nullptr, YITU_ERR_INVALID_ARG, "graph.indices is NULL");
    YITU_REQUIRE(g->n_rows < (1ll << 31) && g->n_cols < (1ll << 31), YITU_ERR_LIMIT,
                 "node ids must fit int32 (n_rows=%lld n_cols=%lld)", (long long)g->n_rows, (long long)g->n_cols);
    YITU_REQUIRE(g->indptr_is64 || g->nnz < (1ll << 31), YITU_ERR_LIMIT,
                 "nnz=%lld needs int64 row pointers", (long long)g->nnz);
    YITU_REQUIRE(g->index_mask == 0 || g->index_mask == 0xffffff, YITU_ERR_INVALID_ARG,
                 "index_mask must be 0 or 0xffffff");
    return YITU_OK;
}

}  // namespace yitu
