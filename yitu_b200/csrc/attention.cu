// GAT attention kernels for sm_100a.
//
//   edge_softmax_{fwd,bwd}  stand-alone "SDDMM" of the reference (u_add_v -> LeakyReLU -> per-segment edge
//                           softmax) with [nnz,H] attention in memory — the drop-in operator path;
//   edge_dot                grad of the per-edge values of a multi-head SpMM;
//   edge_gather_sum         per-source sum of per-edge gradients over the transposed graph (replaces the
//                           reference's atomicAdd scatter);
//   gat_fwd / gat_bwd       the fused layer core: one pass over a row's edges computes scores, an online
//                           max/sum softmax and the weighted aggregation; the backward is one pass over the
//                           transposed graph that reuses every gathered gradient row for grad_x and for d attn
//                           (attention rebuilt per edge from the forward's row statistics);
//   hub rows                every kernel takes the optional hub schedule: long rows are cut into chunks with an ordered
//                           merge, or handed to a whole CTA.
//
// All of them are bound by gather bandwidth (HBM/L2); none uses float atomics.
#include <math_constants.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace yitu {

__device__ __forceinline__ int pow2_shift(int v) { return 31 - __clz(v); }

// Loads that have to be issued where they stand: a plain __ldg may be sunk to its first use, behind the wait for the feature
// row that was requested with it, which puts its latency on top of the row's.
__device__ __forceinline__ float load_now(const float *p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
// base + row * bytes as one 32 x 32 + 64 bit multiply-add
template <typename T>
__device__ __forceinline__ const T *row_at(const T *base, int row, uint32_t bytes) {
    return reinterpret_cast<const T *>(reinterpret_cast<const char *>(base) + static_cast<uint64_t>(static_cast<uint32_t>(row)) * bytes);
}
__device__ __forceinline__ float4 load_now(const float4 *p) {
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// ---------------------------------------------------------------------------------------------------------
// Stand-alone edge softmax.  A lane is (edge slot, head): HB = pow2 >= min(H,32) lanes span the heads (coalesced key / attn
// accesses).  A warp owns a row; a row of more than HUB_EDGES edges gets a CTA of 512 threads.  A row of up to four edges per
// slot is held in registers: ids, segments and scores are read once, all in flight together, whatever the number of segments.
// Longer rows are walked four edges per slot at a time, for SEGS segments at once (1, 2 or 4, by their number: a plain graph
// does not compute the sums of three segments it has not).  (One edge at a time, once per segment and pass, a row was a chain
// of gathers: the hub rows of 2.4 M edges x 4 heads in 3 segments took 368 us forward and 416 us backward.)
//   NARROW: a step is no wider than the edges left ask for.  On a plain graph of even rows the empty positions of four-wide steps
// cost more than the gathers in flight gain (us, forward / backward, one edge at a time | always four | NARROW: 100 k rows x 33
// edges x 4 heads 86 / 117 | 134 / 185 | 85 / 123, 300 k x 16 166 / 246 | 173 / 315 | 157 / 219, R-MAT 500 k x 32 1148 / 1713 |
// 854 / 1374 | 604 / 977); with several segments the forward is better without (100 k x 100 in three: 371, NARROW 545).
// ---------------------------------------------------------------------------------------------------------
struct SoftmaxParams {
    int64_t n_rows;
    const void *indptr;
    const int *indices;
    int is64, mask, B, H, HB;
    float slope;
    const float *q, *k, *attn_in, *grad_attn;
    float *attn_out, *grad_q, *edge_grad;
    // optional hub schedule: rows longer than hub_edges are left to the CTA-per-row variants below, one CTA per cta_chunks
    // consecutive chunks
    int64_t n_chunks;
    int chunk_edges, hub_edges, cta_chunks;
    const int *chunk_row;
    const int64_t *chunk_begin;
};

constexpr int HUB_THREADS = 512;
// Rows from which on a CTA is taken: 256 edges, and twice the average row, so that a graph whose rows are all long keeps a
// warp for each.  (One B200, us, forward / backward with 4 heads, every row of the chunk schedule, 64 edges and more | 256 and
// more: uniform 10 k rows x 70 edges 102 / 166 | 34 / 65, R-MAT 100 k x 24 133 / 249 | 131 / 242, with 1024 157 / 314; uniform
// 4 k x 500 109 / 237 | 82 / 154, with 1024 78 / 127.)
constexpr int HUB_EDGES = 256;

// Row assignment shared by the stand-alone kernels.  CTA = false: one warp per row, hub rows skipped when a schedule
// is given.  CTA = true: one CTA per hub row, its edge slots advancing together; a CTA looks at cta_chunks consecutive chunks, and
// at most one hub row begins there: it is longer than hub_edges >= cta_chunks * chunk_edges.
template <bool CTA>
__device__ __forceinline__ bool softmax_row(const SoftmaxParams &p, int64_t &row, int64_t &eb, int64_t &ee) {
    if constexpr (CTA) {
        __shared__ int64_t s_chunk;
        if (threadIdx.x == 0) s_chunk = -1;
        __syncthreads();
        const int64_t first = static_cast<int64_t>(blockIdx.x) * p.cta_chunks, last = min(first + p.cta_chunks, p.n_chunks);
        for (int64_t c = first + threadIdx.x; c < last; c += blockDim.x) {
            const int64_t r = __ldg(p.chunk_row + c), b = load_ptr(p.indptr, p.is64, r);
            if (__ldg(p.chunk_begin + c) == b && load_ptr(p.indptr, p.is64, r + 1) - b > p.hub_edges) s_chunk = c;
        }
        __syncthreads();
        if (s_chunk < 0) return false;
        row = __ldg(p.chunk_row + s_chunk);
        eb = load_ptr(p.indptr, p.is64, row);
        ee = load_ptr(p.indptr, p.is64, row + 1);
        return true;
    } else {
        row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
        if (row >= p.n_rows) return false;
        eb = load_ptr(p.indptr, p.is64, row);
        ee = load_ptr(p.indptr, p.is64, row + 1);
        return !(p.n_chunks > 0 && ee - eb > p.hub_edges);
    }
}

// Sum (or maximum) over the edge slots that share a head lane: shuffles inside the warp, then (CTA) across the warps through
// shared memory, every thread combining the values in the same order.
template <bool CTA, bool MAX>
__device__ __forceinline__ float slot_reduce(float v, int HB, float *s_red) {
    const auto join = [](float a, float b) { return MAX ? fmaxf(a, b) : a + b; };
    for (int o = HB; o < 32; o <<= 1) v = join(v, __shfl_xor_sync(0xffffffffu, v, o));
    if constexpr (CTA) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, hs = lane & (HB - 1), warps = blockDim.x >> 5;
        __syncthreads();
        if (lane < HB) s_red[warp * 32 + hs] = v;
        __syncthreads();
        v = s_red[hs];
        for (int w = 1; w < warps; ++w) v = join(v, s_red[w * 32 + hs]);
    }
    return v;
}

// U edges of a slot (`left` of them and of the other slots' up to there are edges of the row): segment (-1: none) and column.
template <int U>
struct Edges {
    int seg[U], col[U];
    __device__ __forceinline__ void load(const SoftmaxParams &p, int64_t at, int left, int ES) {
        int raw[U];
#pragma unroll
        for (int u = 0; u < U; ++u) raw[u] = u * ES < left ? __ldg(p.indices + at + u * ES) : 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            seg[u] = u * ES < left ? (p.mask ? static_cast<int>(static_cast<unsigned>(raw[u]) >> 24) : 0) : -1;
            if (seg[u] >= p.B) seg[u] = -1;  // edges of segments without a query take no part
            col[u] = p.mask ? (raw[u] & p.mask) : raw[u];
        }
    }
};
template <int U>
using Width = std::integral_constant<int, U>;

// step(width, first edge of this slot, edges from there) over a row: four edges per slot at a time; NARROW: what is left of the
// row in one step that is no wider than it has to be
template <bool NARROW, typename Step>
__device__ __forceinline__ void walk_row(int64_t eb, int64_t ee, int slot, int ES, Step step) {
    if constexpr (NARROW) {
        int64_t b = eb;
        for (; ee - b >= 4 * ES; b += 4 * ES) step(Width<4>{}, b + slot, 4 * ES - slot);
        const int left = static_cast<int>(ee - b);
        if (left > 2 * ES) step(Width<4>{}, b + slot, left - slot);
        else if (left > ES) step(Width<2>{}, b + slot, left - slot);
        else if (left > 0) step(Width<1>{}, b + slot, left - slot);
    } else {
        for (int64_t b = eb; b < ee; b += 4 * ES) step(Width<4>{}, b + slot, static_cast<int>(min(ee - b, static_cast<int64_t>(4 * ES))) - slot);
    }
}
// held(width): a row that fits the registers, NARROW: as narrow as it allows
template <bool NARROW, typename Held>
__device__ __forceinline__ void hold_row(int len, int ES, Held held) {
    if (!NARROW || len > 2 * ES) {
        held(Width<4>{});
    } else if constexpr (NARROW) {
        if (len > ES) held(Width<2>{});
        else held(Width<1>{});
    }
}

template <bool CTA, int SEGS>
__global__ void __launch_bounds__(CTA ? HUB_THREADS : 256, CTA ? 2 : 5) edge_softmax_fwd_kernel(const __grid_constant__ SoftmaxParams p) {
    constexpr bool NARROW = !CTA && SEGS == 1;
    __shared__ float s_red[CTA ? HUB_THREADS : 1];
    int64_t row, eb, ee;
    if (!softmax_row<CTA>(p, row, eb, ee)) return;
    const int lane = threadIdx.x & 31;
    const int hs = lane & (p.HB - 1);
    const int slot = (CTA ? threadIdx.x : lane) >> pow2_shift(p.HB);
    const int ES = (CTA ? HUB_THREADS : 32) / p.HB;
    for (int hc = 0; hc < p.H; hc += p.HB) {
        const int h = hc + hs;
        const bool hv = h < p.H;
        const auto query = [&](int s) { return __ldg(p.q + (static_cast<int64_t>(s) * p.n_rows + row) * p.H + h); };
        const auto scores = [&](const auto &e, int first, int last, auto &z) {  // of the edges in segments [first, last)
            constexpr int U = std::extent<std::remove_reference_t<decltype(z)>>::value;
#pragma unroll
            for (int u = 0; u < U; ++u)
                z[u] = (hv && e.seg[u] >= first && e.seg[u] < last) ? __ldg(row_at(p.k + h, e.col[u], static_cast<uint32_t>(p.H) * 4u)) : -CUDART_INF_F;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (hv && e.seg[u] >= first && e.seg[u] < last) z[u] = leaky_relu(query(e.seg[u]) + z[u], p.slope);
        };
        if (ee - eb <= 4 * ES) {
            hold_row<NARROW>(static_cast<int>(ee - eb), ES, [&](auto width) {
                constexpr int U = decltype(width)::value;
                Edges<U> e;
                e.load(p, eb + slot, static_cast<int>(ee - eb) - slot, ES);
                float z[U];
                scores(e, 0, p.B, z);
                for (int s = 0; s < p.B; ++s) {
                    float m = -CUDART_INF_F, l = 0.0f;
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (e.seg[u] == s) m = fmaxf(m, z[u]);
                    m = slot_reduce<CTA, true>(m, p.HB, s_red);
                    float w[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        w[u] = e.seg[u] == s ? expf(z[u] - m) : 0.0f;
                        l += w[u];
                    }
                    l = slot_reduce<CTA, false>(l, p.HB, s_red);
                    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (hv && e.seg[u] == s) p.attn_out[(eb + slot) * p.H + h + u * ES * p.H] = w[u] * inv;
                }
            });
            continue;
        }
        for (int s0 = 0; s0 < p.B; s0 += SEGS) {
            float m[SEGS], l[SEGS];
#pragma unroll
            for (int s = 0; s < SEGS; ++s) {
                m[s] = -CUDART_INF_F;
                l[s] = 0.0f;
            }
            walk_row<NARROW>(eb, ee, slot, ES, [&](auto width, int64_t at, int left) {
                constexpr int U = decltype(width)::value;
                Edges<U> e;
                e.load(p, at, left, ES);
                float z[U];
                scores(e, s0, s0 + SEGS, z);
#pragma unroll
                for (int s = 0; s < SEGS; ++s) {
                    float top = m[s];
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (e.seg[u] == s0 + s) top = fmaxf(top, z[u]);
                    const float ref = top > -CUDART_INF_F ? top : 0.0f;
                    if (top > m[s]) l[s] *= expf(m[s] - ref);
                    m[s] = top;
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (e.seg[u] == s0 + s) l[s] += expf(z[u] - ref);
                }
            });
            float inv[SEGS];
#pragma unroll
            for (int s = 0; s < SEGS; ++s) {
                if (s0 + s >= p.B) break;
                const float top = slot_reduce<CTA, true>(m[s], p.HB, s_red);
                if (top > -CUDART_INF_F) l[s] *= expf(m[s] - top);
                l[s] = slot_reduce<CTA, false>(l[s], p.HB, s_red);
                m[s] = top;
                inv[s] = l[s] > 0.0f ? 1.0f / l[s] : 0.0f;
            }
            walk_row<NARROW>(eb, ee, slot, ES, [&](auto width, int64_t at, int left) {
                constexpr int U = decltype(width)::value;
                Edges<U> e;
                e.load(p, at, left, ES);
                float z[U];
                scores(e, s0, s0 + SEGS, z);
#pragma unroll
                for (int s = 0; s < SEGS; ++s)
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (hv && e.seg[u] == s0 + s) p.attn_out[at * p.H + h + u * ES * p.H] = expf(z[u] - m[s]) * inv[s];
            });
        }
    }
}

template <bool CTA, int SEGS>
__global__ void __launch_bounds__(CTA ? HUB_THREADS : 256, CTA ? 2 : SEGS == 1 ? 6 : 4) edge_softmax_bwd_kernel(const __grid_constant__ SoftmaxParams p) {
    constexpr bool NARROW = !CTA;
    __shared__ float s_red[CTA ? HUB_THREADS : 1];
    int64_t row, eb, ee;
    if (!softmax_row<CTA>(p, row, eb, ee)) return;
    const int lane = threadIdx.x & 31;
    const int hs = lane & (p.HB - 1);
    const int slot = (CTA ? threadIdx.x : lane) >> pow2_shift(p.HB);
    const int ES = (CTA ? HUB_THREADS : 32) / p.HB;
    for (int hc = 0; hc < p.H; hc += p.HB) {
        const int h = hc + hs;
        const bool hv = h < p.H;
        const auto query = [&](int s) { return __ldg(p.q + (static_cast<int64_t>(s) * p.n_rows + row) * p.H + h); };
        // attention and its gradient of the edges in segments [first, last)
        const auto weights = [&](const auto &e, int64_t at, int first, int last, auto &a, auto &g) {
            constexpr int U = std::extent<std::remove_reference_t<decltype(a)>>::value;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool on = hv && e.seg[u] >= first && e.seg[u] < last;
                a[u] = on ? __ldg(p.attn_in + at * p.H + h + u * ES * p.H) : 0.0f;
                g[u] = on ? __ldg(p.grad_attn + at * p.H + h + u * ES * p.H) : 0.0f;
            }
        };
        // whether their scores are negative
        const auto signs = [&](const auto &e, int first, int last, auto &neg) {
            constexpr int U = std::extent<std::remove_reference_t<decltype(neg)>>::value;
            float kv[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                kv[u] = hv && e.seg[u] >= first && e.seg[u] < last ? __ldg(row_at(p.k + h, e.col[u], static_cast<uint32_t>(p.H) * 4u)) : 0.0f;
#pragma unroll
            for (int u = 0; u < U; ++u)
                neg[u] = hv && e.seg[u] >= first && e.seg[u] < last && query(e.seg[u]) + kv[u] < 0.0f;
        };
        // per segment s0, s0 + 1, ...: t = sum of attn * grad, gq = sum of the score gradients
        const auto weigh = [&](const auto &e, int s0, const auto &a, const auto &g, float (&t)[SEGS]) {
            constexpr int U = std::extent<std::remove_reference_t<decltype(a)>>::value;
#pragma unroll
            for (int s = 0; s < SEGS; ++s)
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (e.seg[u] == s0 + s) t[s] = fmaf(a[u], g[u], t[s]);
        };
        const auto finish = [&](const auto &e, int64_t at, int s0, const auto &a, const auto &g, const auto &neg, const float (&t)[SEGS],
                                float (&gq)[SEGS]) {
            constexpr int U = std::extent<std::remove_reference_t<decltype(a)>>::value;
#pragma unroll
            for (int s = 0; s < SEGS; ++s)
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (hv && e.seg[u] == s0 + s) {
                        const float gs = a[u] * (g[u] - t[s]), gv = gs * (neg[u] ? p.slope : 1.0f);
                        p.edge_grad[at * p.H + h + u * ES * p.H] = gv;
                        gq[s] += gv;
                    }
        };
        const auto total = [&](int s0, float (&v)[SEGS]) {
#pragma unroll
            for (int s = 0; s < SEGS; ++s)
                if (s0 + s < p.B) v[s] = slot_reduce<CTA, false>(v[s], p.HB, s_red);
        };
        const auto store = [&](int s0, const float (&gq)[SEGS]) {
#pragma unroll
            for (int s = 0; s < SEGS; ++s)
                if (s0 + s < p.B && slot == 0 && hv) p.grad_q[(static_cast<int64_t>(s0 + s) * p.n_rows + row) * p.H + h] = gq[s];
        };
        if (ee - eb <= 4 * ES) {
            hold_row<NARROW>(static_cast<int>(ee - eb), ES, [&](auto width) {
                constexpr int U = decltype(width)::value;
                Edges<U> e;
                e.load(p, eb + slot, static_cast<int>(ee - eb) - slot, ES);
                float a[U], g[U];
                bool neg[U];
                weights(e, eb + slot, 0, p.B, a, g);
                signs(e, 0, p.B, neg);
                for (int s0 = 0; s0 < p.B; s0 += SEGS) {
                    float t[SEGS] = {}, gq[SEGS] = {};
                    weigh(e, s0, a, g, t);
                    total(s0, t);
                    finish(e, eb + slot, s0, a, g, neg, t, gq);
                    total(s0, gq);
                    store(s0, gq);
                }
            });
            continue;
        }
        for (int s0 = 0; s0 < p.B; s0 += SEGS) {
            float t[SEGS] = {}, gq[SEGS] = {};
            walk_row<NARROW>(eb, ee, slot, ES, [&](auto width, int64_t at, int left) {
                constexpr int U = decltype(width)::value;
                Edges<U> e;
                e.load(p, at, left, ES);
                float a[U], g[U];
                weights(e, at, s0, s0 + SEGS, a, g);
                weigh(e, s0, a, g, t);
            });
            total(s0, t);
            walk_row<NARROW>(eb, ee, slot, ES, [&](auto width, int64_t at, int left) {
                constexpr int U = decltype(width)::value;
                Edges<U> e;
                e.load(p, at, left, ES);
                float a[U], g[U];
                bool neg[U];
                weights(e, at, s0, s0 + SEGS, a, g);
                signs(e, s0, s0 + SEGS, neg);
                finish(e, at, s0, a, g, neg, t, gq);
            });
            total(s0, gq);
            store(s0, gq);
        }
    }
}

// out[c,h] = sum over column c of the transposed graph of vals[perm[j], h]
struct GatherSumParams {
    int64_t n_cols;
    const void *t_indptr;
    int is64;
    const int *perm;
    int H, HB;
    const float *vals;
    float *out;
    int64_t n_chunks;
    int chunk_edges;
    const int *chunk_row;
    const int64_t *chunk_begin;
};

// A group of RW = max(8, HB) lanes owns one column, or one chunk of a hub column whose sum goes to `partial`: RW / HB edges
// advance together, eight values per lane in flight.  (A warp per column left most lanes idle at the end of every row: 1 M
// rows x 16 edges x 4 heads 211 us.)  Without scratch for partial sums (n_parts = 0) hub columns get a CTA each, below.
template <int RW>
__global__ void __launch_bounds__(128) edge_gather_sum_kernel(const __grid_constant__ GatherSumParams p, int64_t n_parts, float *partial) {
    constexpr unsigned FULL = 0xffffffffu;
    const int gl = threadIdx.x & (RW - 1);
    const int64_t gid = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / RW;
    const int H = p.H, HB = p.HB, hs = gl & (HB - 1), slot = gl >> pow2_shift(HB), ES = RW / HB;
    int64_t b = 0, e = 0;
    float *dst = nullptr;
    if (gid < n_parts) {
        b = __ldg(p.chunk_begin + gid);
        e = min(b + static_cast<int64_t>(p.chunk_edges), load_ptr(p.t_indptr, p.is64, __ldg(p.chunk_row + gid) + 1));
        dst = partial + gid * H;
    } else if (gid - n_parts < p.n_cols) {
        const int64_t c = gid - n_parts;
        b = load_ptr(p.t_indptr, p.is64, c);
        e = load_ptr(p.t_indptr, p.is64, c + 1);
        if (p.n_chunks > 0 && e - b > p.chunk_edges) e = b;
        else dst = p.out + c * H;
    }
    for (int hc = 0; hc < H; hc += HB) {
        const int h = hc + hs;
        float a = 0.0f;
        for (int64_t j0 = b + slot; __any_sync(FULL, j0 < e); j0 += 8 * ES) {
            int64_t at[8];
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int64_t j = j0 + u * ES;
                at[u] = j < e ? (p.perm ? static_cast<int64_t>(__ldg(p.perm + j)) : j) : -1;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = (at[u] >= 0 && h < H) ? __ldg(p.vals + at[u] * H + h) : 0.0f;
            // in pairs: a column is no long chain of roundings (a bias gradient behind it may cancel to a thousandth)
            a += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        }
        for (int o = HB; o < RW; o <<= 1) a += __shfl_xor_sync(FULL, a, o, RW);
        if (dst && slot == 0 && h < H) dst[h] = a;
    }
}

__global__ void __launch_bounds__(256) edge_gather_sum_hub_kernel(const __grid_constant__ GatherSumParams p) {
    __shared__ float s_red[8 * 32];
    const int64_t c = __ldg(p.chunk_row + blockIdx.x);
    const int64_t b = load_ptr(p.t_indptr, p.is64, c);
    if (__ldg(p.chunk_begin + blockIdx.x) != b) return;
    const int64_t e = load_ptr(p.t_indptr, p.is64, c + 1);
    const int lane = threadIdx.x & 31;
    const int H = p.H, HB = p.HB;
    const int hs = lane & (HB - 1);
    const int slot = threadIdx.x >> pow2_shift(HB);
    const int ES = 256 / HB;
    const int *perm = p.perm;
    const float *vals = p.vals;
    for (int hc = 0; hc < H; hc += HB) {
        const int h = hc + hs;
        float a = 0.0f;
        if (h < H) {
            int64_t j = b + slot;
            // four permutation loads (none when perm is NULL: the identity), then four value loads, in flight together
            for (; j + 3 * ES < e; j += 4 * ES) {
                int64_t p0 = j, p1 = j + ES, p2 = j + 2 * ES, p3 = j + 3 * ES;
                if (perm != nullptr) {
                    p0 = __ldg(perm + j); p1 = __ldg(perm + j + ES); p2 = __ldg(perm + j + 2 * ES); p3 = __ldg(perm + j + 3 * ES);
                }
                const float v0 = __ldg(vals + p0 * H + h), v1 = __ldg(vals + p1 * H + h), v2 = __ldg(vals + p2 * H + h),
                            v3 = __ldg(vals + p3 * H + h);
                a += v0; a += v1; a += v2; a += v3;
            }
            for (; j < e; j += ES) a += __ldg(vals + (perm ? static_cast<int64_t>(__ldg(perm + j)) : j) * H + h);
        }
        a = slot_reduce<true, false>(a, HB, s_red);
        if (slot == 0 && h < H) p.out[c * H + h] = a;
    }
}

// grad_a[e,h] = <g[row,h,:], x[col,h,:]>.  A group of LP = pow2 >= min(F,32) lanes owns one (edge, head) pair.
__global__ void __launch_bounds__(256)
edge_dot_kernel(int64_t n_rows, const void *indptr, int is64, const int *indices, int mask, int H, int F, int LP,
                const float *g, int g_shared, float g_scale, const float *x, float *grad_a) {
    const int64_t row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (row >= n_rows) return;
    const int lane = threadIdx.x & 31;
    const int gl = lane & (LP - 1);
    const int grp = lane >> pow2_shift(LP);
    const int G = 32 / LP;
    const int64_t eb = load_ptr(indptr, is64, row), ee = load_ptr(indptr, is64, row + 1);
    const int64_t D = static_cast<int64_t>(H) * F;
    const int64_t pairs = (ee - eb) * H;
    const float *gr = g + row * (g_shared ? F : D);  // g_shared: one F-wide gradient row serves every head
    for (int64_t pb = 0; pb < pairs; pb += G) {  // uniform trip count: every lane joins the shuffles
        const int64_t pi = pb + grp;
        float a = 0.0f;
        int64_t e = 0;
        int h = 0;
        if (pi < pairs) {
            e = eb + pi / H;
            h = static_cast<int>(pi % H);
            const int raw = __ldg(indices + e);
            const int col = mask ? (raw & mask) : raw;
            const float *xr = x + static_cast<int64_t>(col) * D + static_cast<int64_t>(h) * F;
            const float *gh = g_shared ? gr : gr + static_cast<int64_t>(h) * F;
            for (int k = gl; k < F; k += LP) a = fmaf(__ldg(gh + k), __ldg(xr + k), a);
        }
        for (int o = LP >> 1; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (pi < pairs && gl == 0) grad_a[e * H + h] = a * g_scale;
    }
}

// Fast path of edge_dot for F a multiple of 4 with F/4 a power of two and H*F <= 512: one warp per row keeps the
// row of g in registers, gathers the source rows with 128-bit loads (two edges in flight), reduces each head's
// partial products with log2(F/4) shuffles, and writes the [32 edges, H] tile of results coalesced.
template <int NV>
__global__ void __launch_bounds__(256)
edge_dot_rows_kernel(int64_t n_rows, const void *indptr, int is64, const int *indices, int mask, int H, int F,
                     const float *g, int g_shared, float g_scale, const float *x, float *grad_a, int64_t n_chunks,
                     int chunk_edges, const int *chunk_row, const int64_t *chunk_begin) {
    extern __shared__ float smem[];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the first n_chunks warps take the chunks of the hub rows (every edge is independent: nothing to merge)
    const int64_t gid = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + wib;
    int64_t row, eb, ee;
    if (gid < n_chunks) {
        row = __ldg(chunk_row + gid);
        eb = __ldg(chunk_begin + gid);
        ee = min(eb + static_cast<int64_t>(chunk_edges), load_ptr(indptr, is64, row + 1));
    } else {
        row = gid - n_chunks;
        if (row >= n_rows) return;
        eb = load_ptr(indptr, is64, row);
        ee = load_ptr(indptr, is64, row + 1);
        if (n_chunks > 0 && ee - eb > chunk_edges) return;
    }
    float *base = smem + wib * (32 + 32 * H);
    int *s_col = reinterpret_cast<int *>(base);
    float *s_out = base + 32;
    const int64_t D = static_cast<int64_t>(H) * F;
    const int LPH = F >> 2;
    int hd[NV];
    bool valid[NV];
    int64_t off[NV];
    float4 gr[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        off[i] = static_cast<int64_t>(i * 32 + lane) * 4;
        valid[i] = off[i] < D;
        hd[i] = valid[i] ? static_cast<int>(off[i] / F) : 0;
        gr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid[i]) {
            const float *gp = g_shared ? g + row * F + (off[i] - static_cast<int64_t>(hd[i]) * F) : g + row * D + off[i];
            gr[i] = __ldg(reinterpret_cast<const float4 *>(gp));
            gr[i].x *= g_scale; gr[i].y *= g_scale; gr[i].z *= g_scale; gr[i].w *= g_scale;
        }
    }
    for (int64_t e0 = eb; e0 < ee; e0 += 32) {
        const int n = static_cast<int>(min(static_cast<int64_t>(32), ee - e0));
        int my_col = lane < n ? ld_stream(indices + e0 + lane) : 0;
        if (mask) my_col &= mask;
        const int c_first = __shfl_sync(0xffffffffu, my_col, 0);
        s_col[lane] = lane < n ? my_col : c_first;
        __syncwarp();
        const int n2 = (n + 1) & ~1;
        for (int j = 0; j < n2; j += 2) {
            float4 v[2][NV];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float *xr = x + static_cast<int64_t>(s_col[j + u]) * D;
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    v[u][i] = valid[i] ? __ldg(reinterpret_cast<const float4 *>(xr + off[i]))
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    float d = gr[i].x * v[u][i].x + gr[i].y * v[u][i].y + gr[i].z * v[u][i].z + gr[i].w * v[u][i].w;
                    for (int s = LPH >> 1; s > 0; s >>= 1) d += __shfl_xor_sync(0xffffffffu, d, s);
                    if (valid[i] && (lane & (LPH - 1)) == 0 && j + u < n) s_out[(j + u) * H + hd[i]] = d;
                }
        }
        __syncwarp();
        for (int idx = lane; idx < n * H; idx += 32) grad_a[e0 * H + idx] = s_out[idx];
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------------------------
// Fused GAT forward.  A group of RW lanes owns one destination row (or hub chunk); LPE of them cover a source row, NV slices
// of VEC floats each, and a slice lies inside one head.  A lane therefore computes the scores of its own head's edges itself
// (q in a register, one 4-byte key per edge, the same address for the lanes of a head) and keeps that head's running maximum
// and sum: no score ever goes through shared memory, and the key and feature gathers of EU edges are in flight together as
// soon as the ids are known.  The accumulators are rescaled once per step when the maximum moves (online softmax).  With
// RW > LPE the sub-groups take different edges and are merged at the end of the row like hub chunks.
//   Bound by gather bandwidth for wide rows; for narrow ones by the chain of three latencies per row, which is why the
// narrowest group that covers a row is taken (four rows of 64 floats per warp).  Against a warp per row with the scores of a
// tile in shared memory (us): uniform 1 M rows x 33 edges 8x32 6500 -> 5610 (6.3 TB/s gathered), 1 M x 17 8x8 2250 -> 756,
// 4x32 2150 -> 1360, R-MAT 1 M x 16 4x16 1920 -> 753, 131 k x 19 8x8 350 -> 119.
//   EU and the register bound: four edges per step at 80 registers for up to 128 floats (8x8 uniform: 752; at 64 registers
// 942, at 94 without a bound 981; two edges 807, eight 1006); wider rows run unbounded (5570; 5860 at 80 registers).
// ---------------------------------------------------------------------------------------------------------
struct GatParams {
    int64_t n_rows;
    const void *indptr;
    const int *indices;
    int is64, H, F;
    float slope;
    const float *q, *k, *x;
    float *out, *row_max, *row_sum;
    int head_mean, act;
    float *out_heads;           // head_mean: optional per-head result [n_rows,H,F]
    // hub rows: chunk c covers edges [chunk_begin[c], +chunk_edges) of row chunk_row[c]; its unnormalised sums, running
    // maxima and sums go to partial[c] = {H*F, H, H} floats and gat_fwd_merge_kernel finishes the row
    int64_t n_chunks;
    int chunk_edges;
    const int *chunk_row;
    const int64_t *chunk_begin;
    float *partial;
};

// floats of one hub chunk's partial result: H*F sums, then H maxima and H sums (padded so that chunks stay 32-byte aligned
// when the sums are whole 32-byte slices)
__host__ __device__ __forceinline__ int64_t fwd_partial_stride(int64_t H, int64_t F) { return H * F + ((2 * H + 7) & ~7ll); }

template <int RW, int LPE, int NV, int VEC, int EU, int MINB = 1>
__global__ void __launch_bounds__(128, MINB) gat_fwd_kernel(const __grid_constant__ GatParams p) {
    constexpr int EPI = RW / LPE, STEP = EPI * EU;
    static_assert(RW % STEP == 0, "a tile of RW ids is consumed in whole steps");
    extern __shared__ __align__(16) float smem[];  // head_mean: H*F floats per group
    const int lane = threadIdx.x & 31, gl = lane & (RW - 1), sub = gl / LPE, l_in = gl & (LPE - 1);
    constexpr unsigned FULL_WARP = 0xffffffffu;
    const int64_t gid = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / RW;
    int64_t row, eb, ee;
    const bool chunk = gid < p.n_chunks;
    bool store = true;  // a group without a row, or with a hub row (done by its chunks), keeps its warp company
    if (chunk) {
        row = __ldg(p.chunk_row + gid);
        eb = __ldg(p.chunk_begin + gid);
        ee = min(eb + static_cast<int64_t>(p.chunk_edges), load_ptr(p.indptr, p.is64, row + 1));
    } else {
        store = gid - p.n_chunks < p.n_rows;
        row = store ? gid - p.n_chunks : 0;
        eb = load_ptr(p.indptr, p.is64, row);
        ee = load_ptr(p.indptr, p.is64, row + 1);
        store = store && !(p.n_chunks > 0 && ee - eb > p.chunk_edges);
        if (!store) {
            if (RW == 32) return;
            ee = eb;
        }
    }
    const int H = p.H, F = p.F, D = H * F;
    int off[NV], hd[NV];
    bool valid[NV];  // lanes behind the row's end repeat its first slice and store nothing
    const float *kp[NV], *xp[NV];
    float q[NV], m[NV], l[NV], acc[NV][VEC];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        off[i] = (i * LPE + l_in) * VEC;
        valid[i] = off[i] < D;
        if (!valid[i]) off[i] = 0;
        hd[i] = off[i] / F;
        q[i] = __ldg(p.q + row * H + hd[i]);
        kp[i] = p.k + hd[i];
        xp[i] = p.x + off[i];
        m[i] = -CUDART_INF_F;
        l[i] = 0.0f;
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[i][v] = 0.0f;
    }
    const uint32_t k_bytes = static_cast<uint32_t>(H) * 4u, x_bytes = static_cast<uint32_t>(D) * 4u;
    int my_col = eb + gl < ee ? ld_stream(p.indices + eb + gl) : 0;
    // EU edges of this lane's sub-group, starting at position j of the tile; FULL: all STEP positions carry an edge
    auto step = [&](int j, int n, auto full) {
        constexpr bool FULL = decltype(full)::value;
        float s[EU][NV], x[EU][NV][VEC];
#pragma unroll
        for (int u = 0; u < EU; ++u) {
            const int at = j + u * EPI + sub;
            const int c = __shfl_sync(FULL_WARP, my_col, at, RW);
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                if (FULL || at < n) {
                    s[u][i] = load_now(row_at(kp[i], c, k_bytes));
                    load_vec<VEC>(x[u][i], row_at(xp[i], c, x_bytes));
                } else {
                    s[u][i] = -CUDART_INF_F;
#pragma unroll
                    for (int v = 0; v < VEC; ++v) x[u][i][v] = 0.0f;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            float top = m[i];
#pragma unroll
            for (int u = 0; u < EU; ++u) {
                if (FULL || j + u * EPI + sub < n) s[u][i] = leaky_relu(q[i] + s[u][i], p.slope);
                top = fmaxf(top, s[u][i]);
            }
            // a lane that has met no finite score yet subtracts 0: exp(-inf - 0) = 0 and not NaN
            const float ref = top > -CUDART_INF_F ? top : 0.0f;
            const float scale = expf(m[i] - ref);
            m[i] = top;
            l[i] *= scale;
#pragma unroll
            for (int v = 0; v < VEC; ++v) acc[i][v] *= scale;
#pragma unroll
            for (int u = 0; u < EU; ++u) {
                const float w = expf(s[u][i] - ref);
                l[i] += w;
#pragma unroll
                for (int v = 0; v < VEC; ++v) acc[i][v] = fmaf(w, x[u][i][v], acc[i][v]);
            }
        }
    };
    // a warp per row walks whole steps without predicates; with several rows per warp every group takes the predicated form
    // and the trips of the longest, because groups that leave each other execute one after the other
    for (int64_t e0 = eb; RW == 32 ? e0 < ee : __any_sync(FULL_WARP, e0 < ee); e0 += RW) {
        const int n = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(RW), ee - e0)));
        const int nx_col = e0 + RW + gl < ee ? ld_stream(p.indices + e0 + RW + gl) : 0;
        int j = 0;
        if constexpr (RW == 32) {
            for (; j + STEP <= n; j += STEP) step(j, n, std::true_type{});
            if (j < n) step(j, n, std::false_type{});
        } else {
            const int most = __reduce_max_sync(FULL_WARP, n);
            for (; j < most; j += STEP) step(j, n, std::false_type{});
        }
        my_col = nx_col;
    }
    // merge the sub-groups (fixed order: deterministic)
#pragma unroll
    for (int o = LPE; o < RW; o <<= 1)
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const float m2 = __shfl_xor_sync(FULL_WARP, m[i], o, RW), l2 = __shfl_xor_sync(FULL_WARP, l[i], o, RW);
            const float top = fmaxf(m[i], m2), ref = top > -CUDART_INF_F ? top : 0.0f;
            const float mine = expf(m[i] - ref), other = expf(m2 - ref);
            m[i] = top;
            l[i] = l[i] * mine + l2 * other;
#pragma unroll
            for (int v = 0; v < VEC; ++v)
                acc[i][v] = acc[i][v] * mine + __shfl_xor_sync(FULL_WARP, acc[i][v], o, RW) * other;
        }
    if (chunk) {
        float *part = p.partial + gid * fwd_partial_stride(H, F);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if (!valid[i] || sub != 0) continue;
            store_vec<VEC>(part + off[i], acc[i]);
            if (off[i] == hd[i] * F) {
                part[D + hd[i]] = m[i];
                part[D + H + hd[i]] = l[i];
            }
        }
    }
    store = store && !chunk;
    float *stage = smem + static_cast<int64_t>(threadIdx.x / RW) * D;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        if (sub != 0 || !valid[i] || !store) continue;
        // every score of the row is -inf: the softmax is not defined
        if (ee > eb && m[i] == -CUDART_INF_F) l[i] = CUDART_NAN_F;
        const float inv = l[i] > 0.0f ? 1.0f / l[i] : (ee > eb ? CUDART_NAN_F : 0.0f);
        float r[VEC];
#pragma unroll
        for (int v = 0; v < VEC; ++v) r[v] = acc[i][v] * inv;
        if (p.head_mean) {
#pragma unroll
            for (int v = 0; v < VEC; ++v) stage[off[i] + v] = r[v];
            if (p.out_heads) store_vec<VEC>(p.out_heads + row * D + off[i], r);
        } else {
#pragma unroll
            for (int v = 0; v < VEC; ++v) r[v] = activate(r[v], p.act);
            store_vec<VEC>(p.out + row * D + off[i], r);
        }
        if (off[i] == hd[i] * F) {
            p.row_max[row * H + hd[i]] = m[i];
            p.row_sum[row * H + hd[i]] = l[i];
        }
    }
    if (!p.head_mean) return;
    // the layer's mean over heads: the H values of a feature are added in head order (fixed order: deterministic)
    __syncwarp();
    if (!store) return;
    const float inv_h = 1.0f / static_cast<float>(H);
    for (int f = gl; f < F; f += RW) {
        float a = 0.0f;
        for (int h = 0; h < H; ++h) a += stage[h * F + f];
        p.out[row * F + f] = activate(a * inv_h, p.act);
    }
}

// Finishes the hub rows of the fused forward: combines the chunks' (maximum, sum, unnormalised aggregate).  One CTA per hub
// row (the CTAs of a row's later chunks leave at once).  The threads split the chunks: `groups` of them share a head (or a
// feature), each taking every groups-th chunk, and are added in order, so that a row of hundreds of chunks is no serial tail.
__global__ void __launch_bounds__(256) gat_fwd_merge_kernel(const __grid_constant__ GatParams p) {
    __shared__ float s_red[256], s_m[32], s_inv[32], s_o[512];
    const int64_t c0 = blockIdx.x;
    const int64_t row = __ldg(p.chunk_row + c0);
    const int64_t rb = load_ptr(p.indptr, p.is64, row);
    if (__ldg(p.chunk_begin + c0) != rb) return;
    const int64_t re = load_ptr(p.indptr, p.is64, row + 1);
    const int nch = static_cast<int>((re - rb + p.chunk_edges - 1) / p.chunk_edges);
    const int H = p.H, F = p.F, D = H * F, t = threadIdx.x;
    const int64_t stride = fwd_partial_stride(H, F);
    const float *part = p.partial + c0 * stride;
    {
        int hb = 1;
        while (hb < H) hb <<= 1;
        const int h = t & (hb - 1), g = t / hb, groups = 256 / hb;
        float m = -CUDART_INF_F;
        if (h < H)
            for (int c = g; c < nch; c += groups) m = fmaxf(m, part[c * stride + D + h]);
        s_red[t] = m;
        __syncthreads();
        if (g == 0 && h < H) {
            for (int k = 1; k < groups && k < nch; ++k) m = fmaxf(m, s_red[k * hb + h]);
            s_m[h] = m;
        }
        __syncthreads();
        float l = 0.0f;
        if (h < H)
            for (int c = g; c < nch; c += groups) l += part[c * stride + D + H + h] * expf(part[c * stride + D + h] - s_m[h]);
        s_red[t] = l;
        __syncthreads();
        if (g == 0 && h < H) {
            for (int k = 1; k < groups && k < nch; ++k) l += s_red[k * hb + h];
            s_inv[h] = l > 0.0f ? 1.0f / l : CUDART_NAN_F;
            p.row_max[row * H + h] = s_m[h];
            p.row_sum[row * H + h] = l;
        }
        __syncthreads();
    }
    int cols = 8;
    while (cols < D && cols < 256) cols <<= 1;
    const int tx = t & (cols - 1), g = t / cols, groups = 256 / cols;
    for (int d0 = 0; d0 < D; d0 += cols) {
        const int d = d0 + tx, h = d < D ? d / F : 0;
        float a = 0.0f;
        if (d < D) {
#pragma unroll 4
            for (int c = g; c < nch; c += groups) a = fmaf(part[c * stride + d], expf(part[c * stride + D + h] - s_m[h]), a);
        }
        if (groups > 1) {
            s_red[t] = a;
            __syncthreads();
            if (g == 0)
                for (int k = 1; k < groups && k < nch; ++k) a += s_red[k * cols + tx];
            __syncthreads();
        }
        if (g != 0 || d >= D) continue;
        const float v = a * s_inv[h];
        if (p.head_mean) {
            s_o[d] = v;
            if (p.out_heads) p.out_heads[row * D + d] = v;
        } else {
            p.out[row * D + d] = activate(v, p.act);
        }
    }
    if (!p.head_mean) return;
    __syncthreads();
    const float inv_h = 1.0f / static_cast<float>(H);
    for (int f = t; f < F; f += 256) {
        float a = 0.0f;
        for (int h = 0; h < H; ++h) a += s_o[h * F + f];
        p.out[row * F + f] = activate(a * inv_h, p.act);
    }
}

// ---------------------------------------------------------------------------------------------------------
// Fused GAT backward, destination side.  With the forward's row statistics (max M, sum L) the attention of an edge
// is p = exp(LeakyReLU(q+k) - M) / L on its own, and sum_e p_e * dp_e over a row equals Dv = <grad_out, out> of that
// row, so every edge is independent:
//   dp = <grad_out[row,h,:], x[col,h,:]>   (edge_dot_rows_kernel: the gather pass, at the DRAM roofline)
//   d score = p * (dp - Dv) * LeakyReLU'(q+k)   (gat_bwd_score_kernel: streams dp, writes attention and d score in
//                                                place, sums d score per row into grad_query)
// A single kernel doing both passes was measured slower (9.0 ms against 5.6 + 2.2 ms on the 8x32 layer): its register
// count costs the gather pass a fifth of its warps.  The score pass is latency bound (a short dependent chain per row),
// so it is held to 48 registers for five CTAs per SM (2.9 ms at 64 registers).  Hub rows are processed as chunks; chunk_sum_kernel adds the
// chunks' grad_query partials in order.
// ---------------------------------------------------------------------------------------------------------
struct GatBwdParams {
    int64_t n_rows;
    const void *indptr;
    const int *indices;
    int is64, H, F, hshift;
    int vec;  // out_heads is 16-byte aligned (the upstream gradient always is)
    float slope;
    const float *q, *k, *out_heads, *row_max, *row_sum;
    const float *g;  // upstream gradient: [n_rows,H,F], or [n_rows,F] shared by the heads (g_shared), times g_scale
    int g_shared;
    float g_scale;
    float *edge_attn, *edge_grad, *grad_q;  // edge_grad holds dp on entry, d score on exit
    int64_t n_chunks;
    int chunk_edges;
    const int *chunk_row;
    const int64_t *chunk_begin;
    float *q_partial;  // [n_chunks, H]
};

__global__ void __launch_bounds__(256, 5) gat_bwd_score_kernel(const __grid_constant__ GatBwdParams p) {
    extern __shared__ float smem[];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t gid = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + wib;
    int64_t row, eb, ee;
    const bool chunk = gid < p.n_chunks;
    if (chunk) {
        row = __ldg(p.chunk_row + gid);
        eb = __ldg(p.chunk_begin + gid);
        ee = min(eb + static_cast<int64_t>(p.chunk_edges), load_ptr(p.indptr, p.is64, row + 1));
    } else {
        row = gid - p.n_chunks;
        if (row >= p.n_rows) return;
        eb = load_ptr(p.indptr, p.is64, row);
        ee = load_ptr(p.indptr, p.is64, row + 1);
        if (p.n_chunks > 0 && ee - eb > p.chunk_edges) return;
    }
    const int H = p.H, F = p.F;
    const int64_t D = static_cast<int64_t>(H) * F;
    const bool pow2 = p.hshift >= 0;  // then a lane always meets the same head: idx % H == lane % H
    float *base = smem + wib * (32 + 32 * H + 4 * 32);
    int *s_col = reinterpret_cast<int *>(base);
    float *s_v = base + 32;
    float *s_q = s_v + 32 * H, *s_m = s_q + 32, *s_il = s_m + 32, *s_d = s_il + 32;
    if (lane < H) {
        s_q[lane] = __ldg(p.q + row * H + lane);
        s_m[lane] = __ldg(p.row_max + row * H + lane);
        const float l = __ldg(p.row_sum + row * H + lane);
        s_il[lane] = l > 0.0f ? 1.0f / l : 0.0f;
    }
    // Dv[h] = <grad_out[row,h,:], out[row,h,:]>
    const int LPH = F >> 2;
    if (p.vec && (F & 3) == 0 && LPH <= 32 && (LPH & (LPH - 1)) == 0 && D <= 512) {
        // 128-bit slices, all requested before the first use; a head's lanes are adjacent: butterfly inside the head
        float d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t off = static_cast<int64_t>(i * 32 + lane) * 4;
            d[i] = 0.0f;
            if (off < D) {
                const int64_t goff = p.g_shared ? off % F : off;
                const float4 gv = __ldg(reinterpret_cast<const float4 *>(p.g + row * (p.g_shared ? F : D) + goff));
                const float4 ov = __ldg(reinterpret_cast<const float4 *>(p.out_heads + row * D + off));
                d[i] = gv.x * ov.x + gv.y * ov.y + gv.z * ov.z + gv.w * ov.w;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t off = static_cast<int64_t>(i * 32 + lane) * 4;
            for (int o = LPH >> 1; o > 0; o >>= 1) d[i] += __shfl_xor_sync(0xffffffffu, d[i], o);
            if (off < D && (lane & (LPH - 1)) == 0) s_d[off / F] = d[i] * p.g_scale;
        }
    } else {
        for (int h = 0; h < H; ++h) {
            const float *gp = p.g_shared ? p.g + row * F : p.g + row * D + static_cast<int64_t>(h) * F;
            const float *op = p.out_heads + row * D + static_cast<int64_t>(h) * F;
            float d = 0.0f;
            for (int k = lane; k < F; k += 32) d = fmaf(__ldg(gp + k), __ldg(op + k), d);
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            if (lane == 0) s_d[h] = d * p.g_scale;
        }
    }
    __syncwarp();
    float gq = 0.0f;  // pow2: the lane's own pairs (head lane % H); otherwise lane h owns head h
    for (int64_t e0 = eb; e0 < ee; e0 += 32) {
        const int n = static_cast<int>(min(static_cast<int64_t>(32), ee - e0));
        s_col[lane] = lane < n ? ld_stream(p.indices + e0 + lane) : 0;
        __syncwarp();
        const int npairs = n * H;
        // eight (edge, head) pairs per lane and step: their dp and key loads are all issued before the first result is
        // stored (the stores go to the array the dp values come from, which would otherwise order every load behind them)
        for (int idx0 = lane; idx0 < npairs; idx0 += 256) {
            float dpv[8], kv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int idx = idx0 + 32 * u;
                dpv[u] = kv[u] = 0.0f;
                if (idx < npairs) {
                    const int e = pow2 ? (idx >> p.hshift) : (idx / H);
                    dpv[u] = p.edge_grad[e0 * H + idx];
                    kv[u] = __ldg(p.k + static_cast<int64_t>(s_col[e]) * H + (idx - e * H));
                }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int idx = idx0 + 32 * u;
                if (idx < npairs) {
                    const int e = pow2 ? (idx >> p.hshift) : (idx / H);
                    const int h = idx - e * H;
                    const float sc = s_q[h] + kv[u];
                    const float pr = expf(leaky_relu(sc, p.slope) - s_m[h]) * s_il[h];
                    const float ds = pr * (dpv[u] - s_d[h]) * (sc < 0.0f ? p.slope : 1.0f);
                    p.edge_attn[e0 * H + idx] = pr;
                    p.edge_grad[e0 * H + idx] = ds;
                    if (pow2) gq += ds;
                    else s_v[idx] = ds;
                }
            }
        }
        if (!pow2) {
            __syncwarp();
            if (lane < H)
                for (int e = 0; e < n; ++e) gq += s_v[e * H + lane];
        }
        __syncwarp();
    }
    if (pow2)  // lanes lane, lane + H, lane + 2H, ... hold partial sums of head lane % H
        for (int o = H; o < 32; o <<= 1) gq += __shfl_xor_sync(0xffffffffu, gq, o);
    if (lane < H) {
        if (chunk) p.q_partial[gid * H + lane] = gq;
        else p.grad_q[row * H + lane] = gq;
    }
}

// ---------------------------------------------------------------------------------------------------------
// Fused GAT backward, source side: the whole backward in ONE pass over the transposed graph.
// For source c and each of its out-edges e = (c -> r) the row of the upstream gradient g[r] has to be gathered anyway
// (grad_x[c] = sum_e p_e g[r_e]); with x[c] held in registers the same row gives dp_e = <g[r_e], x[c]>, and with the
// per-destination constants (query, log-sum statistics, D = <g[r], out[r]>) packed into one 16-byte record per
// (row, head) the edge's attention p_e and score gradient ds_e follow on the spot:
//     p = exp(LeakyReLU(q[r] + k[c]) - M[r]) / L[r],   ds = p (dp - D[r]) LeakyReLU'(q[r] + k[c]).
// grad_key[c] = sum_e ds_e is local to the warp; ds_e is scattered to the edge's CSR position so that grad_query
// is a plain row sum afterwards.  No pass over the forward graph gathers features, and no [nnz,H] attention array
// exists.  One warp per source row or hub chunk (chunks leave partial grad_x / grad_key rows); EU edges in flight.
// ---------------------------------------------------------------------------------------------------------
struct GatSrcParams {
    int64_t n_cols;      // rows of the transposed graph
    const void *t_indptr;
    int is64;
    const int *t_rows, *t_perm;
    int H, F;
    float slope;
    const float4 *rowpack;  // [n_rows, H]: (query, row max + log row sum, D, unused)
    const float *k, *x;
    const float *g;
    int g_shared;
    float g_scale;
    float *grad_x, *grad_k, *edge_grad;
    int64_t n_chunks;
    int chunk_edges;
    const int *chunk_row;
    const int64_t *chunk_begin;
    float *x_partial, *k_partial;  // [n_chunks, H*F], [n_chunks, H]
    const float *values;           // GIVEN: per-edge weights [nnz, H] in CSR order instead of attention
    float *grad_values;            // GIVEN: d weight [nnz, H] in CSR order
};

// rowpack[r,h] = (q, M + log L, <g[r,h,:], out[r,h,:]>, 0).  One thread per 128-bit slice, the rows end to end; the F / 4
// lanes of a head are added by a butterfly, or one after the other when their number is no power of two (then LPH divides
// the 32 / LPH * LPH lanes that are used of a warp).  Streams g and out once (1 M rows x 64 floats: 258 us with a warp per
// row, which left half of the lanes without a slice).
__global__ void __launch_bounds__(256)
gat_rowpack_kernel(int64_t n_rows, int H, int F, const float *q, const float *row_max, const float *row_sum,
                   const float *g, int g_shared, float g_scale, const float *out_heads, float4 *rowpack) {
    const int lane = threadIdx.x & 31, LPH = F >> 2;
    const int per_warp = 32 / LPH;  // heads per warp
    const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t rh = warp * per_warp + lane / LPH;  // row * H + head
    const int k = lane % LPH;
    const bool valid = lane < per_warp * LPH && rh < n_rows * H;
    float d = 0.0f;
    if (valid) {
        const float4 gv = __ldg(reinterpret_cast<const float4 *>(g + (g_shared ? rh / H : rh) * F) + k);
        const float4 ov = __ldg(reinterpret_cast<const float4 *>(out_heads + rh * F) + k);
        d = gv.x * ov.x + gv.y * ov.y + gv.z * ov.z + gv.w * ov.w;
    }
    if ((LPH & (LPH - 1)) == 0) {
        for (int o = LPH >> 1; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    } else {
        const float mine = d;
        for (int o = 1; o < LPH; ++o) d += __shfl_sync(0xffffffffu, mine, (lane + o) & 31);  // right in each head's first lane
    }
    if (valid && k == 0) {
        // p = exp(score - M) / L = exp(score - (M + log L)); rows without edges are never looked up
        const float l = __ldg(row_sum + rh);
        rowpack[rh] = make_float4(__ldg(q + rh), __ldg(row_max + rh) + logf(fmaxf(l, 1e-38f)), d * g_scale, 0.0f);
    }
}

// Lanes and groups as in the forward: a slice of a lane lies inside one head, so the lane that holds x[c], k[c] and g[r] for
// its head also reads that head's record of the destination and forms p and ds itself, after a butterfly of log2(F / VEC)
// steps for dp.  The record, weight and gradient gathers of EU edges are in flight together.
// GIVEN = true is the backward of a multi-head SpMM with stored edge values (graph_ext.spmm_backward): the weights are
// read instead of rebuilt, and the by-product is d value = <g[r], x[c]> per edge and head.
template <int RW, int LPE, int NV, int VEC, int EU, bool GIVEN, int LPH_T, int MINB = 1>
__global__ void __launch_bounds__(128, MINB) gat_bwd_src_kernel(const __grid_constant__ GatSrcParams p) {
    constexpr int EPI = RW / LPE, STEP = EPI * EU;
    static_assert(RW % STEP == 0, "a tile of RW ids is consumed in whole steps");
    const int lane = threadIdx.x & 31, gl = lane & (RW - 1), sub = gl / LPE, l_in = gl & (LPE - 1);
    constexpr unsigned FULL_WARP = 0xffffffffu;
    const int64_t gid = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / RW;
    int64_t c, eb, ee;
    const bool chunk = gid < p.n_chunks;
    bool store = true;
    if (chunk) {
        c = __ldg(p.chunk_row + gid);
        eb = __ldg(p.chunk_begin + gid);
        ee = min(eb + static_cast<int64_t>(p.chunk_edges), load_ptr(p.t_indptr, p.is64, c + 1));
    } else {
        store = gid - p.n_chunks < p.n_cols;
        c = store ? gid - p.n_chunks : 0;
        eb = load_ptr(p.t_indptr, p.is64, c);
        ee = load_ptr(p.t_indptr, p.is64, c + 1);
        store = store && !(p.n_chunks > 0 && ee - eb > p.chunk_edges);
        if (!store) {
            if (RW == 32) return;
            ee = eb;
        }
    }
    const int H = p.H, F = p.F, D = H * F;
    const int LPH = LPH_T ? LPH_T : F / VEC;  // lanes per head, at most 32; any number only with one slice per lane
    const bool pow2 = (LPH & (LPH - 1)) == 0;
    const int head_lane = sub * LPE + l_in / LPH * LPH;  // read only in the other case
    const uint32_t g_bytes = static_cast<uint32_t>(p.g_shared ? F : D) * 4u, rec_bytes = static_cast<uint32_t>(H) * 16u,
                   edge_bytes = static_cast<uint32_t>(H) * 4u;
    int hd[NV], off[NV];
    bool valid[NV], first[NV];  // lanes behind the row's end repeat its first slice and store nothing; first lane of a head
    const float *gp[NV];
    const float4 *rp[NV];
    float xr[NV][VEC], acc[NV][VEC], kk[NV], gk[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        off[i] = (i * LPE + l_in) * VEC;
        valid[i] = off[i] < D;
        if (!valid[i]) off[i] = 0;
        hd[i] = off[i] / F;
        first[i] = valid[i] && off[i] == hd[i] * F;
        gp[i] = p.g + (p.g_shared ? off[i] - hd[i] * F : off[i]);
        rp[i] = p.rowpack + hd[i];
        kk[i] = GIVEN ? 0.0f : __ldg(p.k + c * H + hd[i]);
        gk[i] = 0.0f;
        load_vec<VEC>(xr[i], p.x + c * D + off[i]);
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
            xr[i][v] *= p.g_scale;
            acc[i][v] = 0.0f;
        }
    }
    int my_r = 0, my_pos = 0;
    if (eb + gl < ee) {
        my_r = ld_stream(p.t_rows + eb + gl);
        my_pos = ld_stream(p.t_perm + eb + gl);
    }
    // EU edges of this lane's sub-group, starting at position j of the tile; FULL: all STEP positions carry an edge
    auto step = [&](int j, int n, auto full) {
        constexpr bool FULL = decltype(full)::value;
        float gv[EU][NV][VEC], w[EU][NV];
        float4 rec[EU][NV];
        int pos[EU];
#pragma unroll
        for (int u = 0; u < EU; ++u) {
            const int at = j + u * EPI + sub;
            const int r = __shfl_sync(FULL_WARP, my_r, at, RW);
            pos[u] = __shfl_sync(FULL_WARP, my_pos, at, RW);
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                if (FULL || at < n) {
                    if constexpr (GIVEN) w[u][i] = load_now(row_at(p.values + hd[i], pos[u], edge_bytes));
                    else rec[u][i] = load_now(row_at(rp[i], r, rec_bytes));
                    load_vec<VEC>(gv[u][i], row_at(gp[i], r, g_bytes));
                } else {
                    w[u][i] = 0.0f;
                    rec[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int v = 0; v < VEC; ++v) gv[u][i][v] = 0.0f;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < EU; ++u) {
            const bool live = FULL || j + u * EPI + sub < n;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                float part[VEC / 4];  // chains of four: fewer roundings (and waits) than one of eight
#pragma unroll
                for (int t = 0; t < VEC / 4; ++t) {
                    part[t] = 0.0f;
#pragma unroll
                    for (int v = 4 * t; v < 4 * t + 4; ++v) part[t] = fmaf(gv[u][i][v], xr[i][v], part[t]);
                }
                float dp = part[0];
                if constexpr (VEC == 8) dp += part[1];
                if (LPH_T || pow2) {
#pragma unroll
                    for (int o = LPE >> 1; o > 0; o >>= 1)
                        if (o < LPH) dp += __shfl_xor_sync(FULL_WARP, dp, o, RW);
                } else {  // every lane adds the head's lanes in the same order
                    const float mine = dp;
                    dp = 0.0f;
                    for (int o = 0; o < LPH; ++o) dp += __shfl_sync(FULL_WARP, mine, head_lane + o, RW);
                }
                float out = dp, pr = 0.0f;
                if constexpr (GIVEN) {
                    pr = w[u][i];
                } else {
                    const float sc = rec[u][i].x + kk[i];
                    pr = expf(leaky_relu(sc, p.slope) - rec[u][i].y);
                    if (!live) pr = 0.0f;
                    out = (sc < 0.0f ? pr * p.slope : pr) * (dp - rec[u][i].z);
                    if (live) gk[i] += out;  // without an edge dp is 0 * x[c]: NaN where x[c] is not finite
                }
#pragma unroll
                for (int v = 0; v < VEC; ++v) acc[i][v] = fmaf(pr, gv[u][i][v], acc[i][v]);
                // the head's first lane writes the score gradient (or d value) to the edge's CSR position
                if (live && first[i])
                    *const_cast<float *>(row_at((GIVEN ? p.grad_values : p.edge_grad) + hd[i], pos[u], edge_bytes)) = out;
            }
        }
    };
    for (int64_t e0 = eb; RW == 32 ? e0 < ee : __any_sync(FULL_WARP, e0 < ee); e0 += RW) {  // as in the forward
        const int n = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(RW), ee - e0)));
        int nx_r = 0, nx_pos = 0;
        if (e0 + RW + gl < ee) {
            nx_r = ld_stream(p.t_rows + e0 + RW + gl);
            nx_pos = ld_stream(p.t_perm + e0 + RW + gl);
        }
        int j = 0;
        if constexpr (RW == 32) {
            for (; j + STEP <= n; j += STEP) step(j, n, std::true_type{});
            if (j < n) step(j, n, std::false_type{});
        } else {
            const int most = __reduce_max_sync(FULL_WARP, n);
            for (; j < most; j += STEP) step(j, n, std::false_type{});
        }
        my_r = nx_r;
        my_pos = nx_pos;
    }
#pragma unroll
    for (int o = LPE; o < RW; o <<= 1)
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            gk[i] += __shfl_xor_sync(FULL_WARP, gk[i], o, RW);
#pragma unroll
            for (int v = 0; v < VEC; ++v) acc[i][v] += __shfl_xor_sync(FULL_WARP, acc[i][v], o, RW);
        }
    if (sub != 0 || !store) return;
    float *xdst = chunk ? p.x_partial + gid * D : p.grad_x + c * D;
    float *kdst = chunk ? p.k_partial + gid * H : p.grad_k + c * H;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        if (!valid[i]) continue;
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[i][v] *= p.g_scale;
        store_vec<VEC>(xdst + off[i], acc[i]);
        if (!GIVEN && first[i]) kdst[hd[i]] = gk[i];
    }
}

// out[row, :W] = sum of the row's chunk partials
template <int VEC>
__global__ void __launch_bounds__(256) chunk_sum_kernel(const __grid_constant__ HubRows h, int W, const float *partial, float *out) {
    reduce_hub_rows<VEC>(h, partial, W, W, [&](int64_t row, int64_t d, float (&a)[VEC]) { store_vec<VEC>(out + row * W + d, a); });
}

static int launch_chunk_sum(const HubRows &h, int64_t W, const float *partial, float *out, cudaStream_t st) {
    if (h.n_chunks == 0) return YITU_OK;
    const unsigned grid = static_cast<unsigned>((h.n_chunks + 7) / 8);
    if (W % 4 == 0 && aligned16(partial) && aligned16(out)) chunk_sum_kernel<4><<<grid, 256, 0, st>>>(h, static_cast<int>(W), partial, out);
    else chunk_sum_kernel<1><<<grid, 256, 0, st>>>(h, static_cast<int>(W), partial, out);
    YITU_LAUNCH_CHECK();
    return YITU_OK;
}

static int head_block(int64_t H) {
    int hb = 1;
    while (hb < H && hb < 32) hb <<= 1;
    return hb;
}

}  // namespace yitu

using namespace yitu;

static int fill_plan(const yitu_hub_plan_t *plan, int64_t *n_chunks, int *chunk_edges, const int **chunk_row,
                     const int64_t **chunk_begin) {
    *n_chunks = 0;
    *chunk_edges = 0;
    *chunk_row = nullptr;
    *chunk_begin = nullptr;
    if (plan == nullptr || plan->n_chunks == 0) return YITU_OK;
    YITU_REQUIRE(plan->chunk_edges >= 32 && plan->chunk_row && plan->chunk_begin, YITU_ERR_INVALID_ARG,
                 "hub plan needs chunk_edges >= 32 and its two tables");
    *n_chunks = plan->n_chunks;
    *chunk_edges = plan->chunk_edges;
    *chunk_row = plan->chunk_row;
    *chunk_begin = plan->chunk_begin;
    return YITU_OK;
}

static int check_softmax_args(const yitu_csr_t *g, int32_t n_segments, int64_t H) {
    if (int rc = validate_csr(g)) return rc;
    YITU_REQUIRE(n_segments >= 1 && n_segments <= 256, YITU_ERR_INVALID_ARG, "n_segments=%d", n_segments);
    YITU_REQUIRE(n_segments == 1 || g->index_mask != 0, YITU_ERR_INVALID_ARG,
                 "several segments need stitched indices (index_mask=0xffffff)");
    YITU_REQUIRE(H >= 1 && H < (1 << 20), YITU_ERR_INVALID_ARG, "n_heads=%lld", (long long)H);
    return YITU_OK;
}

template <bool BWD, int SEGS>
static int launch_softmax_segs(const SoftmaxParams &p, cudaStream_t st) {
    const unsigned grid = static_cast<unsigned>((p.n_rows + 7) / 8);
    if constexpr (BWD) edge_softmax_bwd_kernel<false, SEGS><<<grid, 256, 0, st>>>(p);
    else edge_softmax_fwd_kernel<false, SEGS><<<grid, 256, 0, st>>>(p);
    YITU_LAUNCH_CHECK();
    if (p.n_chunks == 0) return YITU_OK;
    const unsigned hubs = static_cast<unsigned>((p.n_chunks + p.cta_chunks - 1) / p.cta_chunks);
    if constexpr (BWD) edge_softmax_bwd_kernel<true, SEGS><<<hubs, HUB_THREADS, 0, st>>>(p);
    else edge_softmax_fwd_kernel<true, SEGS><<<hubs, HUB_THREADS, 0, st>>>(p);
    YITU_LAUNCH_CHECK();
    return YITU_OK;
}

template <bool BWD>
static int launch_softmax(SoftmaxParams &p, int64_t nnz, cudaStream_t st) {
    const int64_t twice = 2 * (nnz / p.n_rows);
    p.hub_edges = static_cast<int>(std::max<int64_t>({p.chunk_edges, HUB_EDGES, std::min<int64_t>(twice, INT32_MAX)}));
    p.cta_chunks = p.n_chunks > 0 ? p.hub_edges / p.chunk_edges : 1;
    if (p.B == 1) return launch_softmax_segs<BWD, 1>(p, st);
    if (p.B == 2) return launch_softmax_segs<BWD, 2>(p, st);
    return launch_softmax_segs<BWD, 4>(p, st);
}

extern "C" int yitu_edge_softmax_fwd_f32(const yitu_csr_t *g, int32_t n_segments, int64_t n_heads, float slope,
                                         const float *query, const float *key, float *attn,
                                         const yitu_hub_plan_t *plan, yitu_stream_t stream) {
    if (int rc = check_softmax_args(g, n_segments, n_heads)) return rc;
    if (g->n_rows == 0 || g->nnz == 0) return YITU_OK;
    YITU_REQUIRE(query && key && attn, YITU_ERR_INVALID_ARG, "NULL tensor");
    SoftmaxParams p{};
    p.n_rows = g->n_rows; p.indptr = g->indptr; p.indices = g->indices; p.is64 = g->indptr_is64;
    p.mask = g->index_mask; p.B = n_segments; p.H = static_cast<int>(n_heads); p.HB = head_block(n_heads);
    p.slope = slope; p.q = query; p.k = key; p.attn_out = attn;
    if (int rc = fill_plan(plan, &p.n_chunks, &p.chunk_edges, &p.chunk_row, &p.chunk_begin)) return rc;
    return launch_softmax<false>(p, g->nnz, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int yitu_edge_softmax_bwd_f32(const yitu_csr_t *g, int32_t n_segments, int64_t n_heads, float slope,
                                         const float *query, const float *key, const float *attn,
                                         const float *grad_attn, float *grad_query, float *edge_grad,
                                         const yitu_hub_plan_t *plan, yitu_stream_t stream) {
    if (int rc = check_softmax_args(g, n_segments, n_heads)) return rc;
    if (g->n_rows == 0) return YITU_OK;
    YITU_REQUIRE(query && grad_query, YITU_ERR_INVALID_ARG, "NULL tensor");
    YITU_REQUIRE(g->nnz == 0 || (key && attn && grad_attn && edge_grad), YITU_ERR_INVALID_ARG, "NULL tensor");
    SoftmaxParams p{};
    p.n_rows = g->n_rows; p.indptr = g->indptr; p.indices = g->indices; p.is64 = g->indptr_is64;
    p.mask = g->index_mask; p.B = n_segments; p.H = static_cast<int>(n_heads); p.HB = head_block(n_heads);
    p.slope = slope; p.q = query; p.k = key; p.attn_in = attn; p.grad_attn = grad_attn;
    p.grad_q = grad_query; p.edge_grad = edge_grad;
    if (int rc = fill_plan(plan, &p.n_chunks, &p.chunk_edges, &p.chunk_row, &p.chunk_begin)) return rc;
    return launch_softmax<true>(p, g->nnz, reinterpret_cast<cudaStream_t>(stream));
}

// partial: scratch of n_chunks * H floats for the hub columns' chunk sums, or NULL (a CTA per hub column)
static int gather_sum(int64_t n_cols, const void *t_indptr, int32_t indptr_is64, const int32_t *t_perm, int64_t n_heads,
                      const float *edge_vals, float *out, const yitu_hub_plan_t *t_plan, float *partial, cudaStream_t st) {
    if (n_cols == 0) return YITU_OK;
    GatherSumParams p{};
    p.n_cols = n_cols; p.t_indptr = t_indptr; p.is64 = indptr_is64; p.perm = t_perm;
    p.H = static_cast<int>(n_heads); p.HB = head_block(n_heads); p.vals = edge_vals; p.out = out;
    if (int rc = fill_plan(t_plan, &p.n_chunks, &p.chunk_edges, &p.chunk_row, &p.chunk_begin)) return rc;
    const int64_t n_parts = partial ? p.n_chunks : 0;
    // more lanes per column where the columns are too few to fill the chip (10 k columns x 70 edges, 8 heads, us: 16 with 8 lanes)
    int rw = p.HB < 8 ? 8 : p.HB;
    while (rw < 32 && n_cols * rw < 400000) rw *= 2;
    const unsigned grid = static_cast<unsigned>((n_cols + n_parts + 128 / rw - 1) / (128 / rw));
    if (rw == 8) edge_gather_sum_kernel<8><<<grid, 128, 0, st>>>(p, n_parts, partial);
    else if (rw == 16) edge_gather_sum_kernel<16><<<grid, 128, 0, st>>>(p, n_parts, partial);
    else edge_gather_sum_kernel<32><<<grid, 128, 0, st>>>(p, n_parts, partial);
    YITU_LAUNCH_CHECK();
    if (p.n_chunks == 0) return YITU_OK;
    if (partial) {
        const HubRows h{t_indptr, indptr_is64, p.chunk_edges, p.n_chunks, p.chunk_row, p.chunk_begin};
        return launch_chunk_sum(h, n_heads, partial, out, st);
    }
    edge_gather_sum_hub_kernel<<<static_cast<unsigned>(p.n_chunks), 256, 0, st>>>(p);
    YITU_LAUNCH_CHECK();
    return YITU_OK;
}

extern "C" int yitu_edge_gather_sum_f32(int64_t n_cols, const void *t_indptr, int32_t indptr_is64,
                                        const int32_t *t_perm, int64_t n_heads, const float *edge_vals, float *out,
                                        const yitu_hub_plan_t *t_plan, yitu_stream_t stream) {
    YITU_REQUIRE(n_cols >= 0 && n_heads >= 1 && t_indptr, YITU_ERR_INVALID_ARG, "bad argument");
    if (n_cols == 0) return YITU_OK;
    YITU_REQUIRE(out, YITU_ERR_INVALID_ARG, "out is NULL");
    return gather_sum(n_cols, t_indptr, indptr_is64, t_perm, n_heads, edge_vals, out, t_plan, nullptr,
                      reinterpret_cast<cudaStream_t>(stream));
}

// grad_shared: grad_out is [n_rows,F] and stands for every head (scaled by grad_scale) — the gradient of a mean
// over heads.
static int edge_dot_impl(const yitu_csr_t *g, int64_t n_heads, int64_t n_feats, const float *grad_out, int grad_shared,
                         float grad_scale, const float *x, float *grad_a, yitu_stream_t stream, int64_t n_chunks = 0,
                         int chunk_edges = 0, const int *chunk_row = nullptr, const int64_t *chunk_begin = nullptr) {
    if (int rc = validate_csr(g)) return rc;
    YITU_REQUIRE(n_heads >= 1 && n_feats >= 1, YITU_ERR_INVALID_ARG, "bad shape");
    if (g->n_rows == 0 || g->nnz == 0) return YITU_OK;
    YITU_REQUIRE(grad_out && x && grad_a, YITU_ERR_INVALID_ARG, "NULL tensor");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int64_t lph = n_feats / 4, D = n_heads * n_feats;
    const bool fast = n_feats % 4 == 0 && lph <= 32 && (lph & (lph - 1)) == 0 && D <= 512 && n_heads <= 128 &&
                      aligned16(grad_out) && aligned16(x);
    const unsigned blocks = static_cast<unsigned>((g->n_rows + 7) / 8);
    if (fast) {
        const int H = static_cast<int>(n_heads), F = static_cast<int>(n_feats);
        const size_t smem = 8 * (32 + 32 * static_cast<size_t>(H)) * sizeof(float);
        const unsigned blocks_plan = static_cast<unsigned>((g->n_rows + n_chunks + 7) / 8);
        auto run = [&](auto kernel) -> int {
            if (smem > 48 * 1024)
                YITU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
            kernel<<<blocks_plan, 256, smem, st>>>(g->n_rows, g->indptr, g->indptr_is64, g->indices, g->index_mask, H, F,
                                                   grad_out, grad_shared, grad_scale, x, grad_a, n_chunks, chunk_edges,
                                                   chunk_row, chunk_begin);
            YITU_LAUNCH_CHECK();
            return YITU_OK;
        };
        if (D <= 128) return run(edge_dot_rows_kernel<1>);
        if (D <= 256) return run(edge_dot_rows_kernel<2>);
        return run(edge_dot_rows_kernel<4>);
    }
    edge_dot_kernel<<<blocks, 256, 0, st>>>(g->n_rows, g->indptr, g->indptr_is64, g->indices, g->index_mask,
                                            static_cast<int>(n_heads), static_cast<int>(n_feats), head_block(n_feats),
                                            grad_out, grad_shared, grad_scale, x, grad_a);
    YITU_LAUNCH_CHECK();
    return YITU_OK;
}

extern "C" int yitu_edge_dot_f32(const yitu_csr_t *g, int64_t n_heads, int64_t n_feats, const float *grad_out,
                                 const float *x, float *grad_a, const yitu_hub_plan_t *plan, yitu_stream_t stream) {
    int64_t n_chunks;
    int chunk_edges;
    const int *chunk_row;
    const int64_t *chunk_begin;
    if (int rc = fill_plan(plan, &n_chunks, &chunk_edges, &chunk_row, &chunk_begin)) return rc;
    return edge_dot_impl(g, n_heads, n_feats, grad_out, 0, 1.0f, x, grad_a, stream, n_chunks, chunk_edges, chunk_row,
                         chunk_begin);
}

static int check_gat(const yitu_gat_args_t *a, bool backward) {
    YITU_REQUIRE(a != nullptr, YITU_ERR_INVALID_ARG, "args is NULL");
    if (int rc = validate_csr(&a->graph)) return rc;
    const int64_t H = a->n_heads, F = a->n_feats;
    YITU_REQUIRE(H >= 1 && F >= 1, YITU_ERR_INVALID_ARG, "bad shape");
    YITU_REQUIRE(a->graph.index_mask == 0, YITU_ERR_UNSUPPORTED, "fused GAT takes plain (unstitched) graphs");
    YITU_REQUIRE(H <= 32 && F % 4 == 0 && H * F <= 512, YITU_ERR_UNSUPPORTED,
                 "fused GAT needs H <= 32, F %% 4 == 0, H*F <= 512 (H=%lld F=%lld)", (long long)H, (long long)F);
    (void)backward;
    YITU_REQUIRE(a->activation >= YITU_ACT_NONE && a->activation <= YITU_ACT_ELU, YITU_ERR_INVALID_ARG,
                 "unknown activation %d", a->activation);
    YITU_REQUIRE(a->graph.n_rows == 0 || (a->query && a->out && a->row_max && a->row_sum), YITU_ERR_INVALID_ARG,
                 "NULL tensor");
    YITU_REQUIRE(a->graph.nnz == 0 || (a->key && a->x), YITU_ERR_INVALID_ARG, "NULL tensor");
    YITU_REQUIRE(aligned16(a->x) && aligned16(a->out), YITU_ERR_INVALID_ARG, "x / out must be 16-byte aligned");
    return YITU_OK;
}

static void fill_gat(GatParams &p, const yitu_gat_args_t *a) {
    p.n_rows = a->graph.n_rows; p.indptr = a->graph.indptr; p.indices = a->graph.indices;
    p.is64 = a->graph.indptr_is64; p.H = static_cast<int>(a->n_heads); p.F = static_cast<int>(a->n_feats);
    p.slope = a->slope; p.q = a->query; p.k = a->key; p.x = a->x;
    p.out = a->out; p.row_max = a->row_max; p.row_sum = a->row_sum;
    p.head_mean = a->head_mean ? 1 : 0; p.act = a->activation;
    p.out_heads = p.head_mean ? a->out_heads : nullptr;
}

template <int RW, int LPE, int NV, int VEC, int EU, int MINB = 1>
static int launch_gat_fwd(const GatParams &p, cudaStream_t st) {
    const int groups_per_cta = 128 / RW;
    const size_t smem = p.head_mean ? static_cast<size_t>(groups_per_cta) * p.H * p.F * sizeof(float) : 0;
    const int64_t groups = p.n_rows + p.n_chunks;
    const unsigned grid = static_cast<unsigned>((groups + groups_per_cta - 1) / groups_per_cta);
    gat_fwd_kernel<RW, LPE, NV, VEC, EU, MINB><<<grid, 128, smem, st>>>(p);
    YITU_LAUNCH_CHECK();
    return YITU_OK;
}

extern "C" int64_t yitu_gat_fwd_scratch_bytes(int64_t n_chunks, int64_t n_heads, int64_t n_feats) {
    if (n_chunks < 0 || n_heads < 1 || n_feats < 1) return -1;
    return n_chunks * fwd_partial_stride(n_heads, n_feats) * static_cast<int64_t>(sizeof(float));
}

static inline int64_t up256f(int64_t floats) { return (floats + 63) / 64 * 64; }  // 256-byte pieces, counted in floats

extern "C" int64_t yitu_gat_bwd_scratch_bytes(int64_t n_rows, int64_t n_chunks, int64_t t_n_chunks, int64_t n_heads,
                                              int64_t n_feats) {
    if (n_rows < 0 || n_chunks < 0 || t_n_chunks < 0 || n_heads < 1 || n_feats < 1) return -1;
    return (up256f(n_rows * n_heads * 4) + up256f(n_chunks * n_heads) + up256f(t_n_chunks * n_heads) +
            up256f(t_n_chunks * n_heads * n_feats)) *
           static_cast<int64_t>(sizeof(float));
}

extern "C" int yitu_gat_fwd_f32(const yitu_gat_args_t *a, yitu_stream_t stream) {
    if (int rc = check_gat(a, false)) return rc;
    if (a->graph.n_rows == 0) return YITU_OK;
    GatParams p{};
    fill_gat(p, a);
    YITU_REQUIRE(aligned16(p.out_heads), YITU_ERR_INVALID_ARG, "out_heads must be 16-byte aligned");
    if (int rc = fill_plan(a->plan, &p.n_chunks, &p.chunk_edges, &p.chunk_row, &p.chunk_begin)) return rc;
    const int64_t D = a->n_heads * a->n_feats;
    if (p.n_chunks > 0) {
        const int64_t need = yitu_gat_fwd_scratch_bytes(p.n_chunks, a->n_heads, a->n_feats);
        YITU_REQUIRE(a->scratch && a->scratch_bytes >= need && aligned16(a->scratch), YITU_ERR_WORKSPACE, "fused GAT forward with a hub plan needs %lld bytes of 16-byte aligned scratch",
                     (long long)need);
        p.partial = a->scratch;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // 256-bit gathers when a head spans whole 32-byte slices and every row starts on a 32-byte boundary
    const auto a32 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 31) == 0; };
    const bool wide = p.F % 8 == 0 && a32(a->x) && a32(a->out) && a32(p.out_heads) && a32(p.partial);
    int rc;
    if (wide) {
        if (D <= 8) rc = launch_gat_fwd<8, 1, 1, 8, 1>(p, st);
        else if (D <= 16) rc = launch_gat_fwd<8, 2, 1, 8, 2>(p, st);
        else if (D <= 32) rc = launch_gat_fwd<8, 4, 1, 8, 4>(p, st);
        else if (D <= 64) rc = launch_gat_fwd<8, 8, 1, 8, 4, 6>(p, st);
        else if (D <= 128) rc = launch_gat_fwd<16, 16, 1, 8, 4, 6>(p, st);
        else if (D <= 256) rc = launch_gat_fwd<32, 32, 1, 8, 4>(p, st);
        else rc = launch_gat_fwd<32, 32, 2, 8, 2>(p, st);
    } else {
        if (D <= 16) rc = launch_gat_fwd<8, 4, 1, 4, 4>(p, st);
        else if (D <= 32) rc = launch_gat_fwd<8, 8, 1, 4, 4>(p, st);
        else if (D <= 64) rc = launch_gat_fwd<16, 16, 1, 4, 8>(p, st);
        else if (D <= 128) rc = launch_gat_fwd<32, 32, 1, 4, 8>(p, st);
        else if (D <= 256) rc = launch_gat_fwd<32, 32, 2, 4, 4>(p, st);
        else rc = launch_gat_fwd<32, 32, 4, 4, 2>(p, st);
    }
    if (rc) return rc;
    if (p.n_chunks > 0) {
        gat_fwd_merge_kernel<<<static_cast<unsigned>(p.n_chunks), 256, 0, st>>>(p);
        YITU_LAUNCH_CHECK();
    }
    return YITU_OK;
}

// Launches the source-side pass (attention rebuilt, or GIVEN edge values); the caller merges hub chunks afterwards.
template <int RW, int LPE, int NV, int VEC, int EU, bool GIVEN, int MINB = 1>
static int launch_src_as(const GatSrcParams &p, cudaStream_t st) {
    const int groups_per_cta = 128 / RW;
    const unsigned grid = static_cast<unsigned>((p.n_cols + p.n_chunks + groups_per_cta - 1) / groups_per_cta);
    // the butterfly over the lanes of a head is unrolled for the wide loads; the others (heads of four floats, misaligned
    // tensors) branch over its steps.  A head is at most 128 floats wide, and its lanes fit those of a row; a number of them
    // that is no power of two comes with rows of 24 to 128 floats only, and not with GIVEN values.
    const auto run = [&](auto lph) { gat_bwd_src_kernel<RW, LPE, NV, VEC, EU, GIVEN, decltype(lph)::value, MINB><<<grid, 128, 0, st>>>(p); };
    if constexpr (VEC == 4) {
        run(std::integral_constant<int, 0>{});
    } else {
        switch (p.F / VEC) {
            case 1: run(std::integral_constant<int, 1>{}); break;
            case 2: if constexpr (LPE >= 2) run(std::integral_constant<int, 2>{}); break;
            case 4: if constexpr (LPE >= 4) run(std::integral_constant<int, 4>{}); break;
            case 8: if constexpr (LPE >= 8) run(std::integral_constant<int, 8>{}); break;
            case 16: if constexpr (LPE >= 16) run(std::integral_constant<int, 16>{}); break;
            default: if constexpr (!GIVEN && LPE >= 4 && LPE < 32) run(std::integral_constant<int, 0>{}); break;
        }
    }
    YITU_LAUNCH_CHECK();
    return YITU_OK;
}

template <bool GIVEN>
static int launch_src(const GatSrcParams &p, cudaStream_t st) {
    const int D = p.H * p.F;
    // 256-bit gathers when a head spans whole 32-byte slices and every row starts on a 32-byte boundary
    const auto a32 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 31) == 0; };
    if (p.F % 8 == 0 && a32(p.x) && a32(p.g) && a32(p.grad_x) && a32(p.x_partial)) {
        if (D <= 8) return launch_src_as<8, 1, 1, 8, 1, GIVEN>(p, st);
        if (D <= 16) return launch_src_as<8, 2, 1, 8, 2, GIVEN>(p, st);
        if (D <= 32) return launch_src_as<8, 4, 1, 8, 4, GIVEN>(p, st);
        if (D <= 64) return launch_src_as<8, 8, 1, 8, 2, GIVEN, 6>(p, st);
        if (D <= 128) return launch_src_as<16, 16, 1, 8, 4, GIVEN, 4>(p, st);
        if (D <= 256) return launch_src_as<32, 32, 1, 8, 4, GIVEN, 4>(p, st);
        return launch_src_as<32, 32, 2, 8, 2, GIVEN>(p, st);
    }
    if (D <= 16) return launch_src_as<8, 4, 1, 4, 4, GIVEN>(p, st);
    if (D <= 32) return launch_src_as<8, 8, 1, 4, 4, GIVEN>(p, st);
    if (D <= 64) return launch_src_as<16, 16, 1, 4, 4, GIVEN>(p, st);
    if (D <= 128) return launch_src_as<32, 32, 1, 4, 4, GIVEN>(p, st);
    if (D <= 256) return launch_src_as<32, 32, 2, 4, 4, GIVEN>(p, st);
    return launch_src_as<32, 32, 4, 4, 2, GIVEN>(p, st);
}

extern "C" int yitu_gat_bwd_f32(const yitu_gat_bwd_args_t *b, yitu_stream_t stream) {
    YITU_REQUIRE(b != nullptr, YITU_ERR_INVALID_ARG, "args is NULL");
    const yitu_gat_args_t *a = &b->fwd;
    if (int rc = check_gat(a, true)) return rc;
    const yitu_csr_t &g = a->graph;
    YITU_REQUIRE(g.nnz < (1ll << 31), YITU_ERR_LIMIT, "fused GAT backward needs nnz < 2^31");
    YITU_REQUIRE(b->grad_out && b->grad_query && b->grad_key && b->grad_x && b->t_indptr, YITU_ERR_INVALID_ARG,
                 "NULL tensor");
    YITU_REQUIRE(g.nnz == 0 || (b->t_rows && b->t_perm && b->edge_grad), YITU_ERR_INVALID_ARG,
                 "NULL transposed graph or scratch");
    YITU_REQUIRE(aligned16(b->grad_out) && aligned16(b->grad_x), YITU_ERR_INVALID_ARG,
                 "grad_out / grad_x must be 16-byte aligned");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int64_t H = a->n_heads, F = a->n_feats, D = H * F;
    const int shared = a->head_mean ? 1 : 0;
    const float gscale = shared ? 1.0f / static_cast<float>(H) : 1.0f;
    const float *out_heads = shared ? a->out_heads : a->out;
    YITU_REQUIRE(g.n_rows == 0 || out_heads, YITU_ERR_INVALID_ARG,
                 "the backward of a head-mean forward needs fwd.out_heads (the per-head result)");

    GatBwdParams p{};
    int64_t t_chunks = 0;
    int t_chunk_edges = 0;
    const int *t_chunk_row = nullptr;
    const int64_t *t_chunk_begin = nullptr;
    if (int rc = fill_plan(a->plan, &p.n_chunks, &p.chunk_edges, &p.chunk_row, &p.chunk_begin)) return rc;
    if (int rc = fill_plan(b->t_plan, &t_chunks, &t_chunk_edges, &t_chunk_row, &t_chunk_begin)) return rc;
    const int64_t need = yitu_gat_bwd_scratch_bytes(g.n_rows, p.n_chunks, t_chunks, H, F);
    YITU_REQUIRE(b->scratch && b->scratch_bytes >= need && aligned16(b->scratch), YITU_ERR_WORKSPACE,
                 "fused GAT backward needs %lld bytes of 16-byte aligned scratch", (long long)need);
    float *rowpack = b->scratch;
    float *q_partial = rowpack + up256f(g.n_rows * H * 4);
    float *k_partial = q_partial + up256f(p.n_chunks * H);
    float *x_partial = k_partial + up256f(t_chunks * H);
    if (g.nnz == 0) {  // x and key may be NULL then, which the kernels below read whether a source has edges or not
        if (g.n_rows > 0) YITU_CUDA(cudaMemsetAsync(b->grad_query, 0, g.n_rows * H * sizeof(float), st));
        if (g.n_cols > 0) {
            YITU_CUDA(cudaMemsetAsync(b->grad_key, 0, g.n_cols * H * sizeof(float), st));
            YITU_CUDA(cudaMemsetAsync(b->grad_x, 0, g.n_cols * D * sizeof(float), st));
        }
        return YITU_OK;
    }
    const int64_t lph = F / 4;
    // lanes per head: a power of two, or any number when a row is one slice per lane
    const bool one_pass = lph <= 32 && ((lph & (lph - 1)) == 0 || D <= 128) && aligned16(a->x) && aligned16(out_heads);

    if (one_pass) {
        // (1) per-destination constants, (2) everything else in one pass over the transposed graph, (3) grad_query as
        // the row sum of the scattered score gradients
        if (g.n_rows > 0) {
            const int64_t heads_per_cta = 8 * (32 / lph);
            gat_rowpack_kernel<<<static_cast<unsigned>((g.n_rows * H + heads_per_cta - 1) / heads_per_cta), 256, 0, st>>>(
                g.n_rows, static_cast<int>(H), static_cast<int>(F), a->query, a->row_max, a->row_sum, b->grad_out, shared,
                gscale, out_heads, reinterpret_cast<float4 *>(rowpack));
            YITU_LAUNCH_CHECK();
        }
        if (g.n_cols > 0) {
            GatSrcParams sp{};
            sp.n_cols = g.n_cols; sp.t_indptr = b->t_indptr; sp.is64 = g.indptr_is64;
            sp.t_rows = b->t_rows; sp.t_perm = b->t_perm; sp.H = static_cast<int>(H); sp.F = static_cast<int>(F);
            sp.slope = a->slope; sp.rowpack = reinterpret_cast<const float4 *>(rowpack); sp.k = a->key; sp.x = a->x;
            sp.g = b->grad_out; sp.g_shared = shared; sp.g_scale = gscale;
            sp.grad_x = b->grad_x; sp.grad_k = b->grad_key; sp.edge_grad = b->edge_grad;
            sp.n_chunks = t_chunks; sp.chunk_edges = t_chunk_edges; sp.chunk_row = t_chunk_row;
            sp.chunk_begin = t_chunk_begin; sp.x_partial = x_partial; sp.k_partial = k_partial;
            if (int rc = launch_src<false>(sp, st)) return rc;
            const HubRows h{b->t_indptr, g.indptr_is64, t_chunk_edges, t_chunks, t_chunk_row, t_chunk_begin};
            if (int rc = launch_chunk_sum(h, D, x_partial, b->grad_x, st)) return rc;
            if (int rc = launch_chunk_sum(h, H, k_partial, b->grad_key, st)) return rc;
        }
        return gather_sum(g.n_rows, g.indptr, g.indptr_is64, nullptr, H, b->edge_grad, b->grad_query,
                          p.n_chunks > 0 ? a->plan : nullptr, q_partial, st);
    }

    // Head widths whose lanes-per-head count is not a power of two (or exceeds a warp): destination side as a gather
    // pass (dp) and a score pass over the forward graph, source side as a per-head SpMM and a per-source sum.
    YITU_REQUIRE(g.nnz == 0 || b->edge_attn, YITU_ERR_INVALID_ARG,
                 "this head width takes the two-sided backward, which needs the edge_attn scratch");
    float *spmm_scratch = x_partial;
    if (g.n_rows > 0) {
        if (int rc = edge_dot_impl(&g, H, F, b->grad_out, shared, gscale, a->x, b->edge_grad, stream, p.n_chunks,
                                   p.chunk_edges, p.chunk_row, p.chunk_begin))
            return rc;
        p.n_rows = g.n_rows; p.indptr = g.indptr; p.indices = g.indices; p.is64 = g.indptr_is64;
        p.H = static_cast<int>(H); p.F = static_cast<int>(F);
        p.hshift = (p.H & (p.H - 1)) == 0 ? 31 - __builtin_clz(p.H) : -1;
        p.slope = a->slope; p.q = a->query; p.k = a->key; p.out_heads = out_heads; p.vec = aligned16(out_heads);
        p.row_max = a->row_max; p.row_sum = a->row_sum;
        p.g = b->grad_out; p.g_shared = shared; p.g_scale = gscale;
        p.edge_attn = b->edge_attn; p.edge_grad = b->edge_grad; p.grad_q = b->grad_query;
        p.q_partial = q_partial;
        const int warps = 8;
        const size_t smem = static_cast<size_t>(warps) * (32 + 32 * p.H + 4 * 32) * sizeof(float);
        if (smem > 48 * 1024)
            YITU_CUDA(cudaFuncSetAttribute(gat_bwd_score_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(smem)));
        gat_bwd_score_kernel<<<static_cast<unsigned>((g.n_rows + p.n_chunks + warps - 1) / warps), warps * 32, smem, st>>>(p);
        YITU_LAUNCH_CHECK();
        const HubRows h{g.indptr, g.indptr_is64, p.chunk_edges, p.n_chunks, p.chunk_row, p.chunk_begin};
        if (int rc = launch_chunk_sum(h, H, q_partial, b->grad_query, st)) return rc;
    }
    yitu_hub_plan_t tp{};
    yitu_spmm_args_t s{};
    s.graph.n_rows = g.n_cols; s.graph.n_cols = g.n_rows; s.graph.nnz = g.nnz;
    s.graph.indptr = b->t_indptr; s.graph.indptr_is64 = g.indptr_is64; s.graph.index_mask = 0;
    s.graph.indices = b->t_rows;
    s.n_heads = H; s.n_feats = F; s.weight_mode = YITU_W_EDGE_HEAD;
    s.edge_values = b->edge_attn; s.edge_perm = b->t_perm; s.alpha = gscale;
    s.x = b->grad_out; s.x_stride = shared ? F : D; s.x_shared_heads = shared; s.out = b->grad_x; s.out_stride = D;
    if (t_chunks > 0) {
        tp = *b->t_plan;
        s.plan = &tp;
        s.scratch = spmm_scratch;
        s.scratch_bytes = t_chunks * D * static_cast<int64_t>(sizeof(float));
    }
    if (int rc = yitu_spmm_csr_f32(&s, stream)) return rc;
    if (g.n_cols == 0) return YITU_OK;
    return gather_sum(g.n_cols, b->t_indptr, g.indptr_is64, b->t_perm, H, b->edge_grad, b->grad_key,
                      t_chunks > 0 ? b->t_plan : nullptr, k_partial, st);
}

extern "C" int yitu_spmm_bwd_f32(const yitu_spmm_bwd_args_t *a, yitu_stream_t stream) {
    YITU_REQUIRE(a != nullptr, YITU_ERR_INVALID_ARG, "args is NULL");
    if (int rc = validate_csr(&a->graph)) return rc;
    const yitu_csr_t &g = a->graph;
    const int64_t H = a->n_heads, F = a->n_feats, D = H * F, lph = F / 4;
    YITU_REQUIRE(H >= 1 && F >= 1, YITU_ERR_INVALID_ARG, "bad shape");
    YITU_REQUIRE(H <= 32 && F % 4 == 0 && D <= 512 && lph <= 32 && (lph & (lph - 1)) == 0, YITU_ERR_UNSUPPORTED,
                 "one-pass SpMM backward needs H <= 32, H*F <= 512 and F/4 a power of two <= 32 (H=%lld F=%lld)",
                 (long long)H, (long long)F);
    YITU_REQUIRE(g.nnz < (1ll << 31), YITU_ERR_LIMIT, "one-pass SpMM backward needs nnz < 2^31");
    YITU_REQUIRE(a->t_indptr && (g.n_cols == 0 || a->grad_x), YITU_ERR_INVALID_ARG, "NULL tensor");
    YITU_REQUIRE(g.nnz == 0 || (a->edge_values && a->x && a->grad_out && a->t_rows && a->t_perm && a->grad_values),
                 YITU_ERR_INVALID_ARG, "NULL tensor");
    YITU_REQUIRE(aligned16(a->x) && aligned16(a->grad_out) && aligned16(a->grad_x), YITU_ERR_INVALID_ARG,
                 "x / grad_out / grad_x must be 16-byte aligned");
    if (g.n_cols == 0) return YITU_OK;
    GatSrcParams sp{};
    int64_t t_chunks = 0;
    if (int rc = fill_plan(a->t_plan, &t_chunks, &sp.chunk_edges, &sp.chunk_row, &sp.chunk_begin)) return rc;
    if (t_chunks > 0)
        YITU_REQUIRE(a->scratch && aligned16(a->scratch) && a->scratch_bytes >= t_chunks * D * 4, YITU_ERR_WORKSPACE,
                     "one-pass SpMM backward with a hub plan needs %lld bytes of scratch", (long long)(t_chunks * D * 4));
    sp.n_cols = g.n_cols; sp.t_indptr = a->t_indptr; sp.is64 = g.indptr_is64; sp.t_rows = a->t_rows; sp.t_perm = a->t_perm;
    sp.H = static_cast<int>(H); sp.F = static_cast<int>(F); sp.x = a->x; sp.g = a->grad_out; sp.g_shared = 0;
    sp.g_scale = 1.0f; sp.grad_x = a->grad_x; sp.n_chunks = t_chunks; sp.x_partial = a->scratch;
    sp.values = a->edge_values; sp.grad_values = a->grad_values;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (g.nnz == 0) {  // x may be NULL then
        YITU_CUDA(cudaMemsetAsync(a->grad_x, 0, g.n_cols * D * sizeof(float), st));
        return YITU_OK;
    }
    if (int rc = launch_src<true>(sp, st)) return rc;
    const HubRows h{a->t_indptr, g.indptr_is64, sp.chunk_edges, t_chunks, sp.chunk_row, sp.chunk_begin};
    return launch_chunk_sum(h, D, a->scratch, a->grad_x, st);
}
