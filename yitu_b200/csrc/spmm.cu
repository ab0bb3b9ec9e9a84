// CSR pull SpMM for sm_100a:  out[r,:] = act(alpha*row_scale[r] * sum_{e in row r} w(e) * x[col_e,:] + bias)
//
// Work decomposition
//   * scalar weights: spmm_group_kernel, the narrowest group of lanes that covers a source row owns one destination row or
//     one chunk of a hub row; spmm_stream_kernel for wide rows of huge graphs (a warp walks 16 rows as one edge stream);
//     per-head weights: spmm_heads_kernel;
//   * column ids / edge weights are fetched one per lane (coalesced, streamed past L1) and broadcast with shuffles, so the
//     gather loop issues nothing but 128- or 256-bit loads and FMAs;
//   * rows longer than plan->chunk_edges are cut into chunks handled by the first n_chunks groups of the
//     grid (scheduled first: they are the longest tasks); partial sums land in scratch and a second small
//     kernel adds them in a fixed order.  No float atomics anywhere: results are run-to-run identical.
//
// Measured alternatives that lost on B200 and are not kept: staging rows in a shared-memory ring with
// cp.async.bulk + mbarrier (2.2x slower: 1 KiB per bulk copy is too fine a grain) or per-lane cp.async (equal
// at best, only at the same occupancy); a persistent
// grid with software-pipelined row pointers / index tiles (1.7x slower than letting the CTA scheduler
// balance short CTAs); the features in slices of 128 or 64 floats, one pass over the graph per slice, so that a larger
// share of the gathered table stays in L2 (uniform graph 1 M rows x 32 edges x 256 floats: 4.87 ms in one pass, 4.84 in
// two, 5.11 in four; R-MAT 2.1 M rows x 30 edges: 5.75-6.1 in one, 6.7 in two); for heads that share one source
// row (x_shared_heads), a lane-per-feature layout with the H edge weights broadcast by shuffle (5.4 ms against 3.7 ms
// for the per-head layout below on the 8x32 layer: ten shuffles per edge cost more than the replicated loads).
//
// The kernel is bound by HBM/L2 gather bandwidth; algorithmic bytes per edge = 4*D + 4 (+4 with edge
// values), per row = 4*D written + one row pointer.

#include <cstdlib>

#include "common.cuh"

namespace yitu {

struct SpmmParams {
    int64_t n_rows, n_cols, D, H, F;
    const void *indptr;
    const int *indices;
    int is64, mask, wmode, accumulate;
    const float *values;
    const int *perm;
    const float *norm_dst, *norm_src, *row_scale;
    float alpha;
    const float *x;
    int64_t xs;
    float *out;
    int64_t os;
    int64_t n_chunks;     // chunks of the hub schedule (> 0: rows longer than chunk_edges are not aggregated as rows)
    int64_t chunk_tasks;  // how many of them THIS launch aggregates (its first groups): n_chunks, or 0
    int64_t row_tasks;    // rows THIS launch aggregates: n_rows, or 0 for a launch that takes the chunks only
    int chunk_edges;
    const int *chunk_row;
    const int64_t *chunk_begin;
    float *scratch;
    const float *bias;
    int act, xshared;
    uint32_t piece;  // spmm_group_kernel without SMALL walks longer rows in pieces of this many edges
    int64_t nnz;
};

// Last step of every output row: bias, then activation (both optional).
template <int VEC>
__device__ __forceinline__ void finish_vec(float (&r)[VEC], const SpmmParams &p, int64_t d) {
    if (p.bias) {
#pragma unroll
        for (int q = 0; q < VEC; ++q) r[q] += __ldg(p.bias + d + q);
    }
    if (p.act) {
#pragma unroll
        for (int q = 0; q < VEC; ++q) r[q] = activate(r[q], p.act);
    }
}

// Per-head edge values (weight of an edge differs from head to head): LPR lanes per row, NV slices of VEC floats per lane.
template <int LPR, int NV, int VEC, int EU, bool IDX32>
__global__ void __launch_bounds__(256) spmm_heads_kernel(const __grid_constant__ SpmmParams p) {
    static_assert(EU <= LPR && (EU & (EU - 1)) == 0, "edge unroll must be a power of two <= lanes per row");
    const int lane = threadIdx.x & 31;
    const int l = lane & (LPR - 1);
    const unsigned gmask = (LPR == 32) ? 0xffffffffu : (((1u << LPR) - 1u) << (lane & ~(LPR - 1)));
    const int64_t gid = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / LPR;
    const int64_t d0 = static_cast<int64_t>(blockIdx.y) * (LPR * NV * VEC);

    int64_t row, eb, ee;
    float *dst;
    bool raw;
    if (gid < p.chunk_tasks) {
        row = __ldg(p.chunk_row + gid);
        eb = __ldg(p.chunk_begin + gid);
        const int64_t rend = load_ptr(p.indptr, p.is64, row + 1);
        ee = min(eb + static_cast<int64_t>(p.chunk_edges), rend);
        dst = p.scratch + gid * p.D;
        raw = true;
    } else {
        row = gid - p.chunk_tasks;
        if (row >= p.row_tasks) return;
        eb = load_ptr(p.indptr, p.is64, row);
        ee = load_ptr(p.indptr, p.is64, row + 1);
        if (p.n_chunks > 0 && ee - eb > p.chunk_edges) return;  // hub row: done by its chunks
        dst = p.out + row * p.os;
        raw = false;
    }

    int64_t off[NV];
    bool valid[NV];
    int hd[NV];
    int64_t xo[NV];  // offset of the lane's slice inside a source row (differs from off[] when heads share x)
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        off[i] = d0 + static_cast<int64_t>(i * LPR + l) * VEC;
        valid[i] = off[i] < p.D;
        hd[i] = static_cast<int>(off[i] / p.F);
        xo[i] = p.xshared ? off[i] - static_cast<int64_t>(hd[i]) * p.F : off[i];
    }

    float acc[NV][VEC];
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[i][v] = 0.0f;

    for (int64_t e0 = eb; e0 < ee; e0 += LPR) {
        const int n = static_cast<int>(min(static_cast<int64_t>(LPR), ee - e0));
        int my_col = 0, my_vi = 0;
        if (l < n) {
            const int64_t e = e0 + l;
            const int rawidx = ld_stream(p.indices + e);
            my_col = p.mask ? (rawidx & p.mask) : rawidx;
            my_vi = p.perm ? ld_stream(p.perm + e) : static_cast<int>(e);
        }
        // lanes past the end of the row repeat the tile's first edge with weight 0, so the gather loop
        // below runs in steps of EU edges without a remainder path (the repeated row is an L1 hit)
        const int c_first = __shfl_sync(gmask, my_col, 0, LPR);
        const int v_first = __shfl_sync(gmask, my_vi, 0, LPR);
        if (l >= n) {
            my_col = c_first;
            my_vi = v_first;
        }
        const int n_up = (n + EU - 1) & ~(EU - 1);
        for (int j = 0; j < n_up; j += EU) {
            int c[EU], vi[EU];
#pragma unroll
            for (int u = 0; u < EU; ++u) {
                c[u] = __shfl_sync(gmask, my_col, j + u, LPR);
                vi[u] = __shfl_sync(gmask, my_vi, j + u, LPR);
            }
            float v[EU][NV][VEC];
            float wh[EU][NV];
#pragma unroll
            for (int u = 0; u < EU; ++u) {
                const float *xr = p.x + static_cast<int64_t>(c[u]) * p.xs;
                // 32-bit element offsets when the feature matrix has fewer than 2^32 elements
                const uint32_t xr32 = static_cast<uint32_t>(c[u]) * static_cast<uint32_t>(p.xs);
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    if (valid[i]) {
                        if constexpr (IDX32) load_vec<VEC>(v[u][i], p.x + (xr32 + static_cast<uint32_t>(xo[i])));
                        else load_vec<VEC>(v[u][i], xr + xo[i]);
                        wh[u][i] = (j + u < n) ? __ldg(p.values + static_cast<int64_t>(vi[u]) * p.H + hd[i]) : 0.0f;
                    } else {
#pragma unroll
                        for (int q = 0; q < VEC; ++q) v[u][i][q] = 0.0f;
                        wh[u][i] = 0.0f;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < EU; ++u)
#pragma unroll
                for (int i = 0; i < NV; ++i)
#pragma unroll
                    for (int q = 0; q < VEC; ++q) acc[i][q] = fmaf(wh[u][i], v[u][i][q], acc[i][q]);
        }
    }

    if (raw) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (valid[i]) store_vec<VEC>(dst + off[i], acc[i]);
    } else {
        const float s = p.alpha * (p.row_scale ? __ldg(p.row_scale + row) : 1.0f);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if (!valid[i]) continue;
            float r[VEC];
            if (p.accumulate) {
                load_vec<VEC>(r, dst + off[i]);
#pragma unroll
                for (int q = 0; q < VEC; ++q) r[q] = fmaf(s, acc[i][q], r[q]);
            } else {
#pragma unroll
                for (int q = 0; q < VEC; ++q) r[q] = s * acc[i][q];
            }
            finish_vec<VEC>(r, p, off[i]);
            store_vec<VEC>(dst + off[i], r);
        }
    }
}

// Scalar weights.  A group of RW lanes owns one destination row (or hub chunk); LPE of them cover a source row (NV slices
// of VEC floats each), so one load instruction of the group fetches RW/LPE edges, and EU such instructions are in flight per
// step.  With RW > LPE every sub-group sums its own edges and a reduce-scatter over the sub-groups ends the row (half of the
// values change hands at every level, so 8 values over 8 sub-groups cost 7 shuffles instead of 24) and leaves each lane one
// contiguous piece of the result to store.
//   What bounds it: DRAM and L2 bandwidth for wide rows; for narrow ones the chain of three dependent latencies per row
// (row pointer, ids, gathers).  A row's edges are therefore gathered 8 to 16 at a time, and the next tile of ids is
// requested before the current one is consumed.
//   SMALL: element offsets into x and the edges of a row fit 32 bits.
template <int RW, int LPE, int NV, int VEC, int EU, bool SMALL, int CTAS>
__global__ void __launch_bounds__(128, SMALL || CTAS < 16 ? CTAS : 12) spmm_group_kernel(const __grid_constant__ SpmmParams p) {
    constexpr int EPI = RW / LPE;  // edges per load instruction
    constexpr int STEP = EPI * EU;
    static_assert(RW % LPE == 0 && RW % STEP == 0, "a tile of RW ids is consumed in whole steps");
    const int lane = threadIdx.x & 31;
    const int gl = lane & (RW - 1);
    const int sub = gl / LPE, l = gl & (LPE - 1);
    constexpr unsigned FULL = 0xffffffffu;
    const int64_t gid = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / RW;
    const int64_t d0 = static_cast<int64_t>(blockIdx.y) * (LPE * NV * VEC);
    const bool raw = gid < p.chunk_tasks;
    bool store = true;  // a group without a row, or with a hub row (done by its chunks), keeps its warp company
    int row;
    int64_t eb;
    uint32_t len;  // edges of the row or chunk, counted from eb, in 32 bits (registers are what limits the warps per SM here):
                   // without SMALL a longer row (int64 row pointers) is walked in pieces of 2^31
    if (raw) {
        row = __ldg(p.chunk_row + gid);
        eb = __ldg(p.chunk_begin + gid);
        len = static_cast<uint32_t>(min(static_cast<int64_t>(p.chunk_edges), load_ptr(p.indptr, p.is64, row + 1) - eb));
    } else {
        store = gid - p.chunk_tasks < p.row_tasks;
        row = store ? static_cast<int>(gid - p.chunk_tasks) : 0;
        eb = load_ptr(p.indptr, p.is64, row);
        const int64_t edges = load_ptr(p.indptr, p.is64, row + 1) - eb;
        len = static_cast<uint32_t>(SMALL ? edges : min(edges, static_cast<int64_t>(p.piece)));
        store = store && !(p.n_chunks > 0 && edges > p.chunk_edges);
        if (!store) {
            if (RW == 32) return;
            len = 0;
        }
    }
    const int *ids = p.indices + eb;
    int off[NV];
    bool valid[NV];
    float acc[NV][VEC];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        off[i] = static_cast<int>(d0) + (i * LPE + l) * VEC;
        valid[i] = off[i] < p.D;
#pragma unroll
        for (int q = 0; q < VEC; ++q) acc[i][q] = 0.0f;
    }

    auto load_tile = [&](uint32_t e, int &col, float &w) {  // e: this lane's edge of the tile
        col = 0;
        w = 0.0f;
        if (e < len) {
            const int rawidx = ld_stream(ids + e);
            col = p.mask ? (rawidx & p.mask) : rawidx;
            if (p.wmode == YITU_W_NONE) {
                w = 1.0f;
            } else if (p.wmode == YITU_W_NODE) {
                w = __ldg(p.norm_src + col);  // the destination's factor is applied once per row, at the end
            } else {
                w = ld_stream(p.values + (p.perm ? static_cast<int64_t>(ld_stream(p.perm + eb + e)) : eb + e));
            }
        }
    };
    const bool empty = len == 0;
    while (true) {
        int my_col;
        float my_w;
        load_tile(gl, my_col, my_w);
        // with several rows per warp every group takes the trips of the longest: groups that leave each other would execute one
        // after the other
        for (uint32_t e0 = 0; RW == 32 ? e0 < len : __any_sync(FULL, e0 < len); e0 += RW) {
            const int n = e0 < len ? static_cast<int>(min(static_cast<uint32_t>(RW), len - e0)) : 0;
            const int most = RW == 32 ? n : __reduce_max_sync(FULL, n);
            int nx_col = 0;
            float nx_w = 0.0f;
            load_tile(e0 + RW + gl, nx_col, nx_w);
            for (int j = 0; j < most; j += STEP) {
                int c[EU];
                float w[EU];
#pragma unroll
                for (int u = 0; u < EU; ++u) {
                    c[u] = __shfl_sync(FULL, my_col, j + u * EPI + sub, RW);
                    w[u] = __shfl_sync(FULL, my_w, j + u * EPI + sub, RW);  // 0 behind the last edge
                }
                float v[EU][NV][VEC];
#pragma unroll
                for (int u = 0; u < EU; ++u) {
                    const bool live = j + u * EPI + sub < n;
                    // one address per edge: the slices lie at constant distances from the lane's first
                    const float *xr = SMALL ? p.x + (static_cast<uint32_t>(c[u]) * static_cast<uint32_t>(p.xs) + static_cast<uint32_t>(off[0]))
                                            : p.x + static_cast<int64_t>(c[u]) * p.xs + off[0];
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
                        if (live && valid[i]) {
                            load_vec<VEC>(v[u][i], xr + i * LPE * VEC);
                        } else {
#pragma unroll
                            for (int q = 0; q < VEC; ++q) v[u][i][q] = 0.0f;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < EU; ++u)
#pragma unroll
                    for (int i = 0; i < NV; ++i)
#pragma unroll
                        for (int q = 0; q < VEC; ++q) acc[i][q] = fmaf(w[u], v[u][i][q], acc[i][q]);
            }
            my_col = nx_col;
            my_w = nx_w;
        }
        if constexpr (SMALL) break;
        const bool more = !raw && len == p.piece;
        if (RW == 32 ? !more : !__any_sync(FULL, more)) break;
        eb += len;
        ids += len;
        len = more ? static_cast<uint32_t>(min(load_ptr(p.indptr, p.is64, row + 1) - eb, static_cast<int64_t>(p.piece))) : 0;
    }
    // reduce-scatter over the sub-groups (fixed order: deterministic); piece = floats of a slice that this lane ends up with
    constexpr int PIECE = (VEC >= EPI) ? VEC / EPI : 1;
    int piece_at = 0;    // offset of the lane's piece inside its VEC-wide slice
    bool owner = true;   // with more sub-groups than values several lanes hold the same piece: the first one stores it
#pragma unroll
    for (int o = LPE, have = VEC; o < RW; o <<= 1) {
        const bool upper = (gl & o) != 0;
        if (have > 1) {
            const int half = have / 2;
#pragma unroll
            for (int i = 0; i < NV; ++i)
#pragma unroll
                for (int q = 0; q < VEC / 2; ++q)
                    if (q < half) {
                        const float send = upper ? acc[i][q] : acc[i][q + half];
                        const float keep = upper ? acc[i][q + half] : acc[i][q];
                        acc[i][q] = keep + __shfl_xor_sync(FULL, send, o, RW);
                    }
            if (upper) piece_at += half;
            have = half;
        } else {
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[i][0] += __shfl_xor_sync(FULL, acc[i][0], o, RW);
            owner = owner && !upper;
        }
    }
    if (!owner || !store) return;
    float *dst = raw ? p.scratch + gid * p.D : p.out + row * p.os;
    // a hub row's chunk is left unscaled, but fully weighted; a row without edges is 0 whatever its factor
    const bool node = p.wmode == YITU_W_NODE && !empty;
    float s = raw ? 1.0f : p.alpha * (p.row_scale ? __ldg(p.row_scale + row) : 1.0f);
    if (node) s *= __ldg(p.norm_dst + row);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        if (!valid[i]) continue;
        const int at = off[i] + piece_at;
        float r[PIECE];
#pragma unroll
        for (int q = 0; q < PIECE; ++q) r[q] = acc[i][q];
        if (raw) {
            if (node) {
#pragma unroll
                for (int q = 0; q < PIECE; ++q) r[q] *= s;
            }
        } else {
            if (p.accumulate) {
                float old[PIECE];
                load_vec<PIECE>(old, dst + at);
#pragma unroll
                for (int q = 0; q < PIECE; ++q) r[q] = fmaf(s, r[q], old[q]);
            } else {
#pragma unroll
                for (int q = 0; q < PIECE; ++q) r[q] = s * r[q];
            }
            finish_vec<PIECE>(r, p, at);
        }
        store_vec<PIECE>(dst + at, r);
    }
}

// Edge-stream variant for rows of 16*VEC < D <= 32*VEC floats with scalar weights: a warp owns R consecutive
// destination rows (or one hub chunk) and walks their edges - which are contiguous in the CSR - as ONE stream.
// Row pointers of the batch come from one coalesced load, column ids / weights from one coalesced load per 32
// edges (the next tile is requested before the current one is consumed), and the feature gathers are issued EU
// edges at a time without regard to row boundaries: when the stream crosses into the next row the accumulator is
// written out (a store, nothing waits for it) and cleared.  A short row therefore costs one store and a
// warp-uniform branch instead of its own chain of three dependent memory latencies (row pointer -> ids ->
// features) and its own warp, and no gather slot is spent on padding a row up to EU edges.  Rows that the hub
// schedule cuts into chunks are stepped over (their edges are neither loaded nor gathered).  Sums are formed in
// edge order, so results are run-to-run identical.
// Measured and not kept: a warp walking several batches in a row with the next batch's row pointers and first index tile
// requested ahead (7.0 / 7.3 / 7.8 / 8.6 ms for 1 / 2 / 4 / 8 batches against 5.64 ms on a 7.27 M-row, 65 M-edge shard: more
// state, spills at 80 registers, and fewer, longer-lived warps hide less latency); 16 edges per gather step (128 registers,
// 16 resident warps: 10.4 ms).
template <int VEC, int EU, int R, bool HUB, bool IDX32>
__global__ void __launch_bounds__(128, (VEC * EU <= 32) ? 6 : 4) spmm_stream_kernel(const __grid_constant__ SpmmParams p) {
    static_assert(R >= 1 && R <= 31 && EU >= 1 && EU <= 16 && 32 % EU == 0, "batch / unroll out of range");
    constexpr unsigned FULL = 0xffffffffu;
    constexpr unsigned GM = (1u << EU) - 1u;
    const int lane = threadIdx.x & 31;
    const int64_t gid = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;

    // rp: first edge of row `lane` of the batch, relative to the batch's first edge (positions inside a batch fit 32
    // bits: the launcher sends graphs of 2^31 or more edges to the group kernel)
    int64_t r0, E0;
    int nr, rp;
    bool raw;
    if (gid < p.chunk_tasks) {  // one chunk of a hub row: a one-row batch whose sum goes to scratch
        raw = true;
        nr = 1;
        r0 = __ldg(p.chunk_row + gid);
        E0 = __ldg(p.chunk_begin + gid);
        const int64_t rend = load_ptr(p.indptr, p.is64, r0 + 1);
        rp = lane == 0 ? 0 : static_cast<int>(min(static_cast<int64_t>(p.chunk_edges), rend - E0));
    } else {
        raw = false;
        r0 = (gid - p.chunk_tasks) * R;
        if (r0 >= p.row_tasks) return;
        nr = static_cast<int>(min(static_cast<int64_t>(R), p.n_rows - r0));
        const int64_t myptr = load_ptr(p.indptr, p.is64, r0 + min(lane, nr));
        E0 = __shfl_sync(FULL, myptr, 0);
        rp = static_cast<int>(myptr - E0);
    }
    const int len = __shfl_sync(FULL, rp, nr);  // edges of the batch
    const int rp_next = __shfl_down_sync(FULL, rp, 1);  // end of row `lane` (lanes < nr)
    const bool myhub = HUB && !raw && lane < nr && (rp_next - rp) > p.chunk_edges;
    const unsigned hub_rows = HUB ? __ballot_sync(FULL, myhub) : 0u;
    const int *idx = p.indices + E0;

    const int off = lane * VEC;
    const bool valid = off < p.D;
    float acc[VEC];
#pragma unroll
    for (int q = 0; q < VEC; ++q) acc[q] = 0.0f;

    auto load_tile = [&](int t, int &col, float &w) {
        col = 0;
        w = 0.0f;
        const int te = t + lane;
        if (te < len) {
            const int rawidx = ld_stream(idx + te);
            col = p.mask ? (rawidx & p.mask) : rawidx;
            if (p.wmode == YITU_W_NONE) {
                w = 1.0f;
            } else if (p.wmode == YITU_W_NODE) {
                w = __ldg(p.norm_src + col);  // the destination's factor is applied once per row, at the end
            } else {
                const int64_t ee = E0 + te;
                const int64_t vi = p.perm ? static_cast<int64_t>(ld_stream(p.perm + ee)) : ee;
                w = ld_stream(p.values + vi);
            }
        }
    };

    int cur = 0;  // row of the batch that the stream is in
    int cur_begin = 0, cur_end = __shfl_sync(FULL, rp, 1);
    // writes out every row that ends at or before position t (several when empty rows follow); warp-uniform
    auto flush = [&](int t) {
        while (cur < nr && cur_end <= t) {
            const int64_t row = r0 + cur;
            if (raw) {
                if (valid) {
                    if (p.wmode == YITU_W_NODE) {  // the reduction over chunks expects fully weighted partial sums
                        const float nd = __ldg(p.norm_dst + row);
#pragma unroll
                        for (int q = 0; q < VEC; ++q) acc[q] *= nd;
                    }
                    store_vec<VEC>(p.scratch + gid * p.D + off, acc);
                }
            } else if (!((hub_rows >> cur) & 1u)) {
                const bool had = cur_end > cur_begin;
                if (valid && (had || !p.accumulate || p.bias || p.act)) {
                    float s = p.alpha * (p.row_scale ? __ldg(p.row_scale + row) : 1.0f);
                    if (p.wmode == YITU_W_NODE) s *= __ldg(p.norm_dst + row);
                    float *dst = p.out + row * p.os + off;
                    float r[VEC];
                    if (p.accumulate) {
                        load_vec<VEC>(r, dst);
#pragma unroll
                        for (int q = 0; q < VEC; ++q) r[q] = fmaf(s, acc[q], r[q]);
                    } else {
#pragma unroll
                        for (int q = 0; q < VEC; ++q) r[q] = s * acc[q];
                    }
                    finish_vec<VEC>(r, p, off);
                    store_vec<VEC>(dst, r);
                }
            }
#pragma unroll
            for (int q = 0; q < VEC; ++q) acc[q] = 0.0f;
            ++cur;
            cur_begin = cur_end;
            cur_end = __shfl_sync(FULL, rp, min(cur + 1, 31));
        }
    };

    auto gather = [&](float (&v)[VEC], int c) {
        if (valid) {
            if constexpr (IDX32)
                load_vec<VEC>(v, p.x + (static_cast<uint32_t>(c) * static_cast<uint32_t>(p.xs) + static_cast<uint32_t>(off)));
            else
                load_vec<VEC>(v, p.x + static_cast<int64_t>(c) * p.xs + off);
        } else {
#pragma unroll
            for (int q = 0; q < VEC; ++q) v[q] = 0.0f;
        }
    };

    int t0 = 0;
    int my_col;
    float my_w;
    load_tile(t0, my_col, my_w);
    while (t0 < len) {
        const int n = min(32, len - t0);
        const int t_next = t0 + 32;
        int nx_col = 0;
        float nx_w = 0.0f;
        if (t_next < len) load_tile(t_next, nx_col, nx_w);
        // bm: positions of this tile where a row of the batch begins; hm: positions inside hub rows
        unsigned bm = 0u, hm = 0u;
        if (lane >= 1 && lane < nr) {
            const int d = rp - t0;
            if (d >= 0 && d < n) bm = 1u << d;
        }
        bm = __reduce_or_sync(FULL, bm);
        if constexpr (HUB) {
            if (myhub) {
                const int lo = max(rp - t0, 0), hi = min(rp_next - t0, n);
                if (hi > lo) hm = (hi - lo >= 32 ? FULL : ((1u << (hi - lo)) - 1u)) << lo;
            }
            hm = __reduce_or_sync(FULL, hm);
        }
        const unsigned vm = (n == 32 ? FULL : ((1u << n) - 1u)) & ~hm;
        if (HUB && vm == 0u) {
            // every edge of the tile belongs to hub rows: continue behind the hub row that holds the tile's last edge
            const int last = t0 + n - 1;
            const unsigned who = __ballot_sync(FULL, myhub && rp <= last && rp_next > last);
            t0 = __shfl_sync(FULL, rp_next, __ffs(who) - 1);
            if (t0 == t_next) {
                my_col = nx_col;
                my_w = nx_w;
            } else if (t0 < len) {
                load_tile(t0, my_col, my_w);
            }
            continue;
        }
        for (int j = 0; j < n; j += EU) {
            const unsigned gv = (vm >> j) & GM, gb = (bm >> j) & GM;
            if (HUB && gv == 0u && gb == 0u) continue;  // a group wholly inside a hub row
            int c[EU];
            float w[EU];
#pragma unroll
            for (int u = 0; u < EU; ++u) {
                c[u] = __shfl_sync(FULL, my_col, j + u);
                w[u] = __shfl_sync(FULL, my_w, j + u);
            }
            float v[EU][VEC];
            if (gv == GM && gb == 0u) {  // EU edges of one row: the common case
#pragma unroll
                for (int u = 0; u < EU; ++u) gather(v[u], c[u]);
#pragma unroll
                for (int u = 0; u < EU; ++u)
#pragma unroll
                    for (int q = 0; q < VEC; ++q) acc[q] = fmaf(w[u], v[u][q], acc[q]);
            } else {  // a row ends inside the group, or some positions carry no edge: same loads, uniform predicates
#pragma unroll
                for (int u = 0; u < EU; ++u)
                    if ((gv >> u) & 1u) gather(v[u], c[u]);
#pragma unroll
                for (int u = 0; u < EU; ++u) {
                    if ((gb >> u) & 1u) flush(t0 + j + u);
                    if ((gv >> u) & 1u) {
#pragma unroll
                        for (int q = 0; q < VEC; ++q) acc[q] = fmaf(w[u], v[u][q], acc[q]);
                    }
                }
            }
        }
        t0 = t_next;
        my_col = nx_col;
        my_w = nx_w;
    }
    flush(INT32_MAX);
}

// Adds the chunk partials of each hub row and applies the epilogue.
template <int VEC>
__global__ void __launch_bounds__(256) hub_reduce_kernel(const __grid_constant__ SpmmParams p) {
    const HubRows h{p.indptr, p.is64, p.chunk_edges, p.n_chunks, p.chunk_row, p.chunk_begin};
    reduce_hub_rows<VEC>(h, p.scratch, p.D, p.D, [&](int64_t row, int64_t d, float (&a)[VEC]) {
        const float s = p.alpha * (p.row_scale ? __ldg(p.row_scale + row) : 1.0f);
        float *o = p.out + row * p.os + d;
        float r[VEC];
        if (p.accumulate) {
            load_vec<VEC>(r, o);
#pragma unroll
            for (int q = 0; q < VEC; ++q) r[q] = fmaf(s, a[q], r[q]);
        } else {
#pragma unroll
            for (int q = 0; q < VEC; ++q) r[q] = s * a[q];
        }
        finish_vec<VEC>(r, p, d);
        store_vec<VEC>(o, r);
    });
}

static int launch_hub_reduce(const SpmmParams &p, cudaStream_t st) {
    if (p.n_chunks == 0) return YITU_OK;
    const unsigned grid = static_cast<unsigned>((p.n_chunks + 7) / 8);
    if (p.D % 4 == 0 && p.os % 4 == 0 && aligned16(p.out) && aligned16(p.scratch)) hub_reduce_kernel<4><<<grid, 256, 0, st>>>(p);
    else hub_reduce_kernel<1><<<grid, 256, 0, st>>>(p);
    YITU_LAUNCH_CHECK();
    return YITU_OK;
}

// 128-thread CTAs: with 256 a CTA waits for its longest row and occupancy drops (measured 7.57 -> 6.98 ms on the
// D=256 R-MAT workload; 32/64/128/256 gave 6.86/7.21/6.98/7.57 ms and 128 was best over all workloads).
static int block_threads() { return 128; }

template <int LPR, int NV, int VEC>
static int launch_heads(const SpmmParams &p, cudaStream_t st) {
    const int64_t groups = p.chunk_tasks + p.row_tasks;
    if (groups == 0) return YITU_OK;
    const int threads = block_threads();
    const int gpb = threads / LPR;
    const int64_t gx = (groups + gpb - 1) / gpb;
    const int64_t gy = (p.D + LPR * NV * VEC - 1) / (LPR * NV * VEC);
    YITU_REQUIRE(gx < (1ll << 31) && gy <= 65535, YITU_ERR_LIMIT, "spmm grid too large (%lld x %lld)",
                 (long long)gx, (long long)gy);
    dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy));
    // 32-bit element offsets into x when they fit; per-head weights cost registers per gathered slice: 4 edges per step
    if (VEC >= 4 && p.n_cols * p.xs < (1ll << 32)) spmm_heads_kernel<LPR, NV, VEC, 4, true><<<grid, threads, 0, st>>>(p);
    else spmm_heads_kernel<LPR, NV, VEC, 4, false><<<grid, threads, 0, st>>>(p);
    YITU_LAUNCH_CHECK();
    return launch_hub_reduce(p, st);
}

template <int VEC, int EU, int R>
static int launch_stream(const SpmmParams &p, cudaStream_t st) {  // always followed by the hub reduction, if any
    const int64_t groups = p.chunk_tasks + (p.row_tasks + R - 1) / R;
    if (groups == 0) return YITU_OK;
    const int threads = block_threads();
    const int64_t gx = (groups + threads / 32 - 1) / (threads / 32);
    YITU_REQUIRE(gx < (1ll << 31), YITU_ERR_LIMIT, "spmm grid too large (%lld)", (long long)gx);
    const unsigned grid = static_cast<unsigned>(gx);
    const bool idx32 = p.n_cols * p.xs < (1ll << 32);
    const bool hub = p.n_chunks > 0;
    if (hub) {
        if (idx32) spmm_stream_kernel<VEC, EU, R, true, true><<<grid, threads, 0, st>>>(p);
        else spmm_stream_kernel<VEC, EU, R, true, false><<<grid, threads, 0, st>>>(p);
    } else {
        if (idx32) spmm_stream_kernel<VEC, EU, R, false, true><<<grid, threads, 0, st>>>(p);
        else spmm_stream_kernel<VEC, EU, R, false, false><<<grid, threads, 0, st>>>(p);
    }
    YITU_LAUNCH_CHECK();
    return launch_hub_reduce(p, st);
}

// Development switches read from the environment at every call (measurement of one kernel form against another):
// YITU_SPMM_STREAM=0 keeps the group kernel for every graph, =2 takes the edge-stream kernel for every graph
// whose shape it covers, =3 the same with the hub rows' chunks on the group kernel (default 1: by the rule in
// yitu_spmm_csr_f32); YITU_SPMM_STREAM_ROWS=8|16|31 and
// YITU_SPMM_STREAM_EU pick an instantiation of the edge-stream kernel other than the default; YITU_SPMM_PIECE=<multiple of 32> is the
// length of the pieces in which the group kernel walks a row (default 2^31).
static int env_int(const char *name, int dflt) {
    const char *v = getenv(name);
    return (v && *v) ? atoi(v) : dflt;
}

template <int VEC, int EU_A, int EU_B>
static int dispatch_stream(const SpmmParams &p, cudaStream_t st, int rows_dflt, int eu_dflt) {
    const int rows = env_int("YITU_SPMM_STREAM_ROWS", rows_dflt);
    const int eu = env_int("YITU_SPMM_STREAM_EU", eu_dflt);
    if (eu == EU_B) {
        if (rows == 8) return launch_stream<VEC, EU_B, 8>(p, st);
        if (rows == 31) return launch_stream<VEC, EU_B, 31>(p, st);
        return launch_stream<VEC, EU_B, 16>(p, st);
    }
    if (rows == 8) return launch_stream<VEC, EU_A, 8>(p, st);
    if (rows == 31) return launch_stream<VEC, EU_A, 31>(p, st);
    return launch_stream<VEC, EU_A, 16>(p, st);
}

template <int RW, int LPE, int NV, int VEC, int EU, int CTAS = 1>
static int launch_group(const SpmmParams &p, cudaStream_t st, bool reduce = true) {
    const int64_t groups = p.chunk_tasks + p.row_tasks;
    if (groups == 0) return YITU_OK;
    const int threads = block_threads();
    const int64_t gx = (groups + threads / RW - 1) / (threads / RW);
    const int64_t gy = (p.D + LPE * NV * VEC - 1) / (LPE * NV * VEC);
    YITU_REQUIRE(gx < (1ll << 31) && gy <= 65535, YITU_ERR_LIMIT, "spmm grid too large (%lld x %lld)",
                 (long long)gx, (long long)gy);
    dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy));
    // a row's edges are bounded by the graph's, or by the schedule that cuts it
    const bool small = p.n_cols * p.xs < (1ll << 32) &&
                       (p.n_chunks > 0 ? p.chunk_edges < p.piece : p.nnz < p.piece);
    if (small) spmm_group_kernel<RW, LPE, NV, VEC, EU, true, CTAS><<<grid, threads, 0, st>>>(p);
    else spmm_group_kernel<RW, LPE, NV, VEC, EU, false, CTAS><<<grid, threads, 0, st>>>(p);
    YITU_LAUNCH_CHECK();
    return reduce ? launch_hub_reduce(p, st) : YITU_OK;
}

// Lanes per row (RW), lanes per edge, edges per step and resident CTAs of spmm_group_kernel by row width, from sweeps on B200
// over uniform and R-MAT graphs of 16 k to 2 M rows.  What decides below 256 floats is how many dependent chains are in flight:
// the narrowest group that covers a source row (four rows of 32 floats per warp), and few registers, so that 12 or 16 CTAs of
// 128 threads fit an SM - a register bound that leaves one or two gathers of a chain in flight beats deeper unrolling at half
// the warps (1 M rows x 16 edges, us: 32 floats 331 at 40 registers, 480 with two edges per step, 368 with eight and no bound;
// R-MAT 1 M x 15, 64 floats 560 at 32 registers, 677 without the bound; 128 floats 808 at 32 registers, 910 without).
// Rows of 33..64 floats are the exception to the narrow group: a warp per row, four edges per load, is as fast on uniform
// graphs (660 us against 671) and faster on power-law ones, where the longest of a warp's rows holds up the others (R-MAT
// 1 M x 15: 511 against 624).
// Rows of up to 16 floats run unbounded up to half a million rows (100 k rows x 16 edges 16.5 us at 16 CTAs, 15.1 without; R-MAT
// 16 k x 14 23 and 16; 1 M x 16 162 and 168).  Where all rows are long and too few to fill the chip twelve CTAs deep, a chain of one
// or two gathers is what counts, and the deeper forms win (128 floats, us: 1 k rows x 100 edges in chunks of 64 18.1 and 10.3,
// 10 k x 70 43.2 and 36.6, whole rows of 30 k x 400 406 and 341; but 100 k x 100 284 and 293.  64 floats, whole rows: 30 k x 400
// 199 and 180; in chunks the shallow form is as good: 3 k x 100 13.1 and 14.6).
// The edges of a row that is not cut into chunks are summed in the order the CSR stores them; 33..64 floats by 256-bit loads in
// four interleaved sums.
static bool few_long_rows(const SpmmParams &p) { return p.n_rows <= 65536 && p.nnz >= 64 * p.n_rows; }
static int dispatch_group4(const SpmmParams &p, cudaStream_t st, bool reduce = true) {
    if (p.D <= 16) return p.n_rows <= 524288 ? launch_group<4, 4, 1, 4, 4>(p, st, reduce) : launch_group<4, 4, 1, 4, 4, 16>(p, st, reduce);
    if (p.D <= 32) return launch_group<8, 8, 1, 4, 4, 12>(p, st, reduce);
    if (p.D <= 64) return launch_group<16, 16, 1, 4, 8>(p, st, reduce);
    if (p.D <= 128 && few_long_rows(p)) return launch_group<32, 32, 1, 4, 8>(p, st, reduce);
    if (p.D <= 128) return launch_group<32, 32, 1, 4, 2, 12>(p, st, reduce);
    if (p.D <= 256) return launch_group<32, 32, 2, 4, 8>(p, st, reduce);
    return launch_group<32, 32, 4, 4, 4>(p, st, reduce);
}
static int dispatch_group8(const SpmmParams &p, cudaStream_t st, bool reduce = true) {
    if (p.D <= 32 || (p.D > 64 && p.D <= 128 && few_long_rows(p))) return dispatch_group4(p, st, reduce);
    if (p.D <= 64 && p.n_chunks == 0 && few_long_rows(p)) return launch_group<32, 8, 1, 8, 2>(p, st, reduce);
    if (p.D <= 64) return launch_group<32, 8, 1, 8, 1, 16>(p, st, reduce);
    if (p.D <= 128) return launch_group<16, 16, 1, 8, 2, 12>(p, st, reduce);
    if (p.D <= 256) return launch_group<32, 32, 1, 8, 2>(p, st, reduce);
    return launch_group<32, 32, 2, 8, 4>(p, st, reduce);
}
// Widths that are no multiple of four, or rows that are not 16-byte aligned: scalar loads, NV of them per lane and edge
// (41 floats, 170 k rows x 13 edges: 200 us with one warp and four masked slices per row, 120 us with 16 lanes x 3).  From 49
// floats on four edges per step without a bound (us, two edges at 12 CTAs | four: 50 floats, 30 k x 100 79 | 66, 1 M x 16 733 |
// 662; 101 floats 114 | 98 and 1323 | 1294); 33..48 up to half a million rows (41 floats, 100 k x 100 185 | 170, 1 M x 16 507 |
// 555).  With an address per load instead of one per edge, 101 floats took 202 (30 k x 100).
static int dispatch_group1(const SpmmParams &p, cudaStream_t st) {
    if (p.D <= 4) return launch_group<4, 4, 1, 1, 4, 16>(p, st);
    if (p.D <= 8) return launch_group<8, 8, 1, 1, 8, 16>(p, st);
    if (p.D <= 16) return launch_group<16, 16, 1, 1, 8, 12>(p, st);
    if (p.D <= 32) return launch_group<16, 16, 2, 1, 4, 12>(p, st);
    if (p.D <= 48) return p.n_rows <= 524288 ? launch_group<16, 16, 3, 1, 4>(p, st) : launch_group<16, 16, 3, 1, 2, 16>(p, st);
    if (p.D <= 64) return launch_group<16, 16, 4, 1, 4>(p, st);
    if (p.D <= 96) return launch_group<32, 32, 3, 1, 4>(p, st);
    return launch_group<32, 32, 4, 1, 4>(p, st);
}

}  // namespace yitu

using namespace yitu;

extern "C" int yitu_spmm_csr_f32(const yitu_spmm_args_t *a, yitu_stream_t stream) {
    YITU_REQUIRE(a != nullptr, YITU_ERR_INVALID_ARG, "args is NULL");
    if (int rc = validate_csr(&a->graph)) return rc;
    const yitu_csr_t &g = a->graph;
    YITU_REQUIRE(a->n_heads >= 1 && a->n_feats >= 1, YITU_ERR_INVALID_ARG, "n_heads=%lld n_feats=%lld",
                 (long long)a->n_heads, (long long)a->n_feats);
    const int64_t D = a->n_heads * a->n_feats;
    YITU_REQUIRE(a->x_shared_heads == 0 || a->weight_mode == YITU_W_EDGE_HEAD, YITU_ERR_INVALID_ARG,
                 "x_shared_heads needs per-head edge values (YITU_W_EDGE_HEAD)");
    const int64_t x_width = a->x_shared_heads ? a->n_feats : D;
    YITU_REQUIRE(a->x_stride >= x_width && a->out_stride >= D, YITU_ERR_INVALID_ARG,
                 "row strides (%lld, %lld) smaller than the rows (%lld, %lld)", (long long)a->x_stride,
                 (long long)a->out_stride, (long long)x_width, (long long)D);
    YITU_REQUIRE(a->activation >= YITU_ACT_NONE && a->activation <= YITU_ACT_ELU, YITU_ERR_INVALID_ARG,
                 "unknown activation %d", a->activation);
    YITU_REQUIRE(g.n_rows == 0 || a->out != nullptr, YITU_ERR_INVALID_ARG, "out is NULL");
    YITU_REQUIRE(g.nnz == 0 || a->x != nullptr, YITU_ERR_INVALID_ARG, "x is NULL");
    YITU_REQUIRE(a->weight_mode >= YITU_W_NONE && a->weight_mode <= YITU_W_EDGE_HEAD, YITU_ERR_INVALID_ARG,
                 "unknown weight_mode %d", a->weight_mode);
    if (a->weight_mode == YITU_W_NODE)
        YITU_REQUIRE(a->norm_dst && a->norm_src, YITU_ERR_INVALID_ARG, "W_NODE needs norm_dst and norm_src");
    if (a->weight_mode == YITU_W_EDGE || a->weight_mode == YITU_W_EDGE_HEAD)
        YITU_REQUIRE(g.nnz == 0 || a->edge_values, YITU_ERR_INVALID_ARG, "edge_values is NULL");
    const bool per_head = a->weight_mode == YITU_W_EDGE_HEAD;
    if (per_head)
        YITU_REQUIRE(g.nnz < (1ll << 31), YITU_ERR_LIMIT, "per-head edge values need nnz < 2^31");

    SpmmParams p{};
    p.n_rows = g.n_rows; p.n_cols = g.n_cols; p.nnz = g.nnz; p.D = D; p.H = a->n_heads; p.F = a->n_feats;
    p.indptr = g.indptr; p.indices = g.indices; p.is64 = g.indptr_is64; p.mask = g.index_mask;
    p.wmode = a->weight_mode; p.accumulate = a->accumulate;
    p.values = a->edge_values; p.perm = a->edge_perm;
    p.norm_dst = a->norm_dst; p.norm_src = a->norm_src; p.row_scale = a->row_scale; p.alpha = a->alpha;
    p.x = a->x; p.xs = a->x_stride; p.out = a->out; p.os = a->out_stride;
    p.bias = a->bias; p.act = a->activation; p.xshared = a->x_shared_heads ? 1 : 0;
    p.row_tasks = g.n_rows;
    p.piece = static_cast<uint32_t>(env_int("YITU_SPMM_PIECE", 0));
    if (p.piece == 0) p.piece = 1u << 31;
    if (a->plan && a->plan->n_chunks > 0) {
        YITU_REQUIRE(a->plan->chunk_edges >= 32, YITU_ERR_INVALID_ARG, "plan.chunk_edges must be >= 32");
        YITU_REQUIRE(a->plan->chunk_row && a->plan->chunk_begin, YITU_ERR_INVALID_ARG, "plan tables are NULL");
        YITU_REQUIRE(a->scratch != nullptr && a->scratch_bytes >= a->plan->n_chunks * D * 4, YITU_ERR_WORKSPACE,
                     "scratch needs %lld bytes, got %lld", (long long)(a->plan->n_chunks * D * 4),
                     (long long)a->scratch_bytes);
        p.n_chunks = a->plan->n_chunks; p.chunk_tasks = p.n_chunks; p.chunk_edges = a->plan->chunk_edges;
        p.chunk_row = a->plan->chunk_row; p.chunk_begin = a->plan->chunk_begin; p.scratch = a->scratch;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);

    const bool vec_ok = (D % 4 == 0) && (a->x_stride % 4 == 0) && (a->out_stride % 4 == 0) && aligned16(a->x) &&
                        aligned16(a->out) && (p.scratch == nullptr || aligned16(p.scratch)) &&
                        (!per_head || a->n_feats % 4 == 0);
    // 256-bit loads when every row starts on a 32-byte boundary
    const auto aligned32 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 31) == 0; };
    const bool vec8_ok = vec_ok && D % 8 == 0 && a->x_stride % 8 == 0 && a->out_stride % 8 == 0 && aligned32(a->x) &&
                         aligned32(a->out) && (p.scratch == nullptr || aligned32(p.scratch)) &&
                         (!per_head || a->n_feats % 8 == 0);
    if (per_head) {
        if (!vec_ok) return launch_heads<32, 4, 1>(p, st);
        if (vec8_ok && D > 128 && D <= 512) return D <= 256 ? launch_heads<32, 1, 8>(p, st) : launch_heads<32, 2, 8>(p, st);
        if (D <= 16) return launch_heads<4, 1, 4>(p, st);
        if (D <= 32) return launch_heads<8, 1, 4>(p, st);
        if (D <= 64) return launch_heads<16, 1, 4>(p, st);
        if (D <= 128) return launch_heads<32, 1, 4>(p, st);
        if (D <= 256) return launch_heads<32, 2, 4>(p, st);
        return launch_heads<32, 4, 4>(p, st);
    }
    if (!vec_ok) return dispatch_group1(p, st);

    // Edge-stream kernel, for rows of 65..256 floats.  It spares a short row its own chain of latencies, but a warp walks
    // 16 consecutive rows, so it needs a graph of so many rows that the heavy batches of a power-law graph do not become
    // the tail (50 k rows x 18 edges, 128 floats: 386 us against 69 us with the group kernel) and rows of few edges.
    // Measured on B200 (us, group / stream), 128 floats: uniform 1 M rows x 16 edges 1246 / 1220, 2 M x 4 edges 908 / 969;
    // 100 floats 1275 / 1196, 1085 / 991; 256 floats 2458 / 2396, 1640 / 1499.  With hub rows (a chunk schedule) the
    // chunks go to the group kernel (a whole warp per chunk, two edges per load) and only the other rows are streamed: R-MAT
    // with 128 floats (ms, group alone / stream alone / both) 16.8 M rows x 31 edges 35.7 / 36.6 / 34.3, 8 M x 8 5.52 / - /
    // 5.23, 4 M x 15 3.93 / 4.16 / 3.87; below 2 M rows the group kernel alone.
    // YITU_SPMM_STREAM (development switch): 0 never, 2 for everything the kernel covers, chunks included, 3 for all rows that
    // are not cut into chunks, 1 (default) by this rule.
    const int stream_mode = env_int("YITU_SPMM_STREAM", 1);
    const bool stream_shape = g.nnz < (1ll << 31) && D > 64 && (D <= 128 || (D <= 256 && vec8_ok));
    const bool use_stream = stream_shape && (stream_mode >= 2 || (stream_mode == 1 && (p.n_chunks > 0
                            ? D <= 128 && g.n_rows >= (2 << 20) && g.nnz < 64 * g.n_rows
                            : g.n_rows >= 150000 && g.nnz < 24 * g.n_rows && !(vec8_ok && D <= 128 && g.nnz < 8 * g.n_rows))));
    if (use_stream) {
        SpmmParams r = p;
        if (p.n_chunks > 0 && stream_mode != 2) {
            SpmmParams c = p;
            c.row_tasks = 0;  // the chunks only; the reduction follows the second launch
            if (int rc = vec8_ok ? launch_group<32, 16, 1, 8, 8>(c, st, false) : dispatch_group4(c, st, false)) return rc;
            r.chunk_tasks = 0;  // the rows that are not cut into chunks (those are stepped over), then the reduction
        }
        return D > 128 ? dispatch_stream<8, 4, 8>(r, st, 16, 4) : dispatch_stream<4, 8, 16>(r, st, 16, 8);
    }
    if (vec8_ok) return dispatch_group8(p, st);
    return dispatch_group4(p, st);
}
