// Dense float32 products of the layers around the aggregation, for matrices of many rows (nodes) and few columns (features):
//   yitu_linear_f32  C[n,N] = A[n,K] B (+ bias): the layer's x W^T + b, x W, and the input gradient g W
//   yitu_gram_f32    C[M,N] = A[n,M]^T B[n,N] and, from the same pass, the column sums of A: weight and bias gradient
// Plain float32 multiply-adds throughout: no operand or partial sum is held in fewer bits.
#include <math_constants.h>

#include "common.cuh"

namespace yitu {

template <int V>
__device__ __forceinline__ void cp_async(float *smem, const float *g, bool ok) {
    const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    if constexpr (V == 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(g), "r"(ok ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s), "l"(g), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two multiply-adds per instruction (new with sm_100): one instruction slot where two plain ones would leave none for
// the shared-memory loads.  Each half rounds like fmaf.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

constexpr int STAGES = 3;

// ---------------------------------------------------------------------------------------------------------
// C = A B + bias.  TX*TY threads hold MT x NT results each: a tile of TY*MT rows and TX*NT columns, K taken in steps of
// KC through a ring of three cp.async stages.  A is staged as it lies ([row][k], rows padded by four floats so that the
// four rows a warp reads at once fall on different banks) and read four k at a time; B is staged as [k][column], with
// four-byte copies when it has to be turned (B_T: B is stored [N,K]).
//   Bound by the fp32 units for N of 64 and more (1 M x 64 x 64: 8.4 GFLOP, 115 us at 74 TFLOP/s, against 512 MB, 78 us),
// by memory below.  The bias is added in the epilogue: the library's SGEMM adds it in a second pass over the result.
// ---------------------------------------------------------------------------------------------------------
struct LinearParams {
    int64_t n;
    int K, N;
    const float *a;
    int64_t lda;
    const float *b;
    int64_t ldb;
    const float *bias;
    float *c;
    int64_t ldc;
    int vec_c;
};

constexpr int KC = 16;

template <int MT, int NT, int TX, int TY>
constexpr int linear_smem_bytes() { return STAGES * (TY * MT * (KC + 4) + KC * (TX * NT + 4)) * 4; }

template <int MT, int NT, int TX, int TY, int VA, int VB, bool B_T>
__global__ void __launch_bounds__(TX *TY, MT *NT == 64 ? 512 / (TX * TY) : 1) linear_kernel(const __grid_constant__ LinearParams p) {
    constexpr int T = TX * TY, TR = TY * MT, TN = TX * NT, AS = KC + 4, BS = TN + 4;
    extern __shared__ __align__(16) float smem[];
    float *sa = smem, *sb = smem + STAGES * TR * AS;
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int n0 = blockIdx.x * TN;
    const int64_t r0 = static_cast<int64_t>(blockIdx.y) * TR;
    const int rows = static_cast<int>(min(static_cast<int64_t>(TR), p.n - r0));

    // a thread copies the same columns of every RA-th (RB-th) row in every step: addresses advance by constants
    constexpr int CA = KC / VA, RA = T / CA, LA = (TR + RA - 1) / RA;
    const int ka = (tid % CA) * VA, ra = tid / CA;
    const float *pa = p.a + (r0 + ra) * p.lda + ka;
    const int64_t step_a = static_cast<int64_t>(RA) * p.lda;
    constexpr int CB = B_T ? KC : TN / VB, RB = T / CB, LB = ((B_T ? TN : KC) + RB - 1) / RB;
    static_assert(T % CA == 0 && T % CB == 0, "threads split into whole rows of a stage");
    const int ib = (tid % CB) * (B_T ? 1 : VB), rb = tid / CB;  // B_T: ib = k, rb = column; else ib = column, rb = k
    const float *pb = B_T ? p.b + static_cast<int64_t>(n0 + rb) * p.ldb + ib : p.b + static_cast<int64_t>(rb) * p.ldb + n0 + ib;
    const int64_t step_b = static_cast<int64_t>(RB) * p.ldb;

    auto load = [&](int k0, int st) {
        float *da = sa + st * TR * AS + ra * AS + ka;
        const bool ka_ok = k0 + ka < p.K;
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int r = ra + i * RA;
            if (TR % RA != 0 && r >= TR) break;
            const bool ok = ka_ok && r < rows;
            cp_async<VA>(da + i * RA * AS, ok ? pa + i * step_a + k0 : p.a, ok);
        }
        float *db = sb + st * KC * BS;
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int r = rb + i * RB;
            if ((B_T ? TN : KC) % RB != 0 && r >= (B_T ? TN : KC)) break;
            if constexpr (B_T) {
                const bool ok = k0 + ib < p.K && n0 + r < p.N;
                cp_async<1>(db + ib * BS + r, ok ? pb + i * step_b + k0 : p.b, ok);
            } else {
                const bool ok = k0 + r < p.K && n0 + ib < p.N;
                cp_async<VB>(db + r * BS + ib, ok ? pb + i * step_b + static_cast<int64_t>(k0) * p.ldb : p.b, ok);
            }
        }
    };

    uint64_t acc[MT][NT / 2];  // pairs of neighbouring columns
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT / 2; ++j) acc[i][j] = 0;

    const int steps = (p.K + KC - 1) / KC;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load(s * KC, s);
        cp_async_commit();
    }
    for (int s = 0; s < steps; ++s) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        if (s + STAGES - 1 < steps) load((s + STAGES - 1) * KC, (s + STAGES - 1) % STAGES);
        cp_async_commit();
        const float *ca = sa + (s % STAGES) * TR * AS, *cb = sb + (s % STAGES) * KC * BS;
#pragma unroll
        for (int k = 0; k < KC; k += 4) {
            float4 av[MT];
#pragma unroll
            for (int i = 0; i < MT; ++i) av[i] = *reinterpret_cast<const float4 *>(ca + (ty + TY * i) * AS + k);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                uint64_t bv[NT / 2];
#pragma unroll
                for (int j = 0; j < NT / 2; j += 2) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(cb + (k + kk) * BS + tx * 4 + (j / 2) * (TX * 4));
                    bv[j] = v.x; bv[j + 1] = v.y;
                }
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    const float x = kk == 0 ? av[i].x : kk == 1 ? av[i].y : kk == 2 ? av[i].z : av[i].w;
                    const uint64_t xx = pack2(x, x);
#pragma unroll
                    for (int j = 0; j < NT / 2; ++j) fma2(acc[i][j], xx, bv[j]);
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NT; j += 4) {
        const int c0 = n0 + tx * 4 + (j / 4) * (TX * 4);
        float bias[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (p.bias) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (c0 + q < p.N) bias[q] = __ldg(p.bias + c0 + q);
        }
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int r = ty + TY * i;
            if (r >= rows) continue;
            float *dst = p.c + (r0 + r) * p.ldc + c0;
            float v[4];
            unpack2(acc[i][j / 2], v[0], v[1]);
            unpack2(acc[i][j / 2 + 1], v[2], v[3]);
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] += bias[q];
            if (p.vec_c) {
                if (c0 < p.N) *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (c0 + q < p.N) dst[q] = v[q];
            }
        }
    }
}

template <int MT, int NT, int TX, int TY>
static int launch_linear(const LinearParams &p, bool b_t, bool vec_a, bool vec_b, cudaStream_t st) {
    const int64_t gy = (p.n + TY * MT - 1) / (TY * MT);
    const unsigned gx = static_cast<unsigned>((p.N + TX * NT - 1) / (TX * NT));
    YITU_REQUIRE(gy <= 65535ll * 1024, YITU_ERR_LIMIT, "too many rows (%lld)", (long long)p.n);
    constexpr int smem = linear_smem_bytes<MT, NT, TX, TY>();
    auto run = [&](auto kernel) -> int {
        if (smem > 48 * 1024) YITU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        // grid.y holds 65535 row tiles: more rows than that take further launches
        LinearParams q = p;
        for (int64_t done = 0; done < gy; done += 65535) {
            const int64_t now = gy - done < 65535 ? gy - done : 65535;
            q.n = p.n - done * (TY * MT);
            q.a = p.a + done * (TY * MT) * p.lda;
            q.c = p.c + done * (TY * MT) * p.ldc;
            kernel<<<dim3(gx, static_cast<unsigned>(now)), TX * TY, smem, st>>>(q);
            YITU_LAUNCH_CHECK();
        }
        return YITU_OK;
    };
    if (b_t) return vec_a ? run(linear_kernel<MT, NT, TX, TY, 4, 1, true>) : run(linear_kernel<MT, NT, TX, TY, 1, 1, true>);
    if (vec_a) return vec_b ? run(linear_kernel<MT, NT, TX, TY, 4, 4, false>) : run(linear_kernel<MT, NT, TX, TY, 4, 1, false>);
    return vec_b ? run(linear_kernel<MT, NT, TX, TY, 1, 4, false>) : run(linear_kernel<MT, NT, TX, TY, 1, 1, false>);
}

// ---------------------------------------------------------------------------------------------------------
// C[M,N] = A^T B over n rows.  The rows are split over the grid; a CTA stages BK rows of its TA columns of A and TB columns
// of B at a time (three cp.async stages) and holds the TA x TB tile of the result in registers, 8 x 8 per thread.  A tile
// needs fewer than 256 threads, so KG groups of threads take every KG-th row and are added up through shared memory at the
// end; the splits leave partial results that gram_reduce_kernel adds in order (run-to-run identical).  The column sums of A
// (or B) are taken from the staged rows: a bias gradient costs no pass of its own.
//   Bound by the fp32 units (64 x 64: 4096 multiply-adds per 512 bytes read).
// ---------------------------------------------------------------------------------------------------------
struct GramParams {
    int64_t n;
    int M, N;
    const float *a;
    int64_t lda;
    const float *b;
    int64_t ldb;
    int64_t rows_per_split;
    float *partial;  // [splits][M*N + sums]
    int64_t pstride;
    int sum_of;      // 0: no column sums, 1: of A (M values), 2: of B (N values)
    int tiles_b;
};

template <int TA, int TB, int BK>
constexpr int gram_smem_bytes() {
    return (STAGES * BK * (TA + TB) > 128 * 64 ? STAGES * BK * (TA + TB) : 128 * 64) * 4;
}

template <int TA, int TB, int BK, int VA, int VB>
__global__ void __launch_bounds__(256, 2) gram_kernel(const __grid_constant__ GramParams p) {
    constexpr int TX = TB / 8, TY = TA / 8, GT = TX * TY, KG = 256 / GT;
    static_assert(BK % KG == 0, "every group takes the same number of a stage's rows");
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, g = tid / GT, t = tid % GT, tx = t % TX, ty = t / TX;
    const int ta = blockIdx.y / p.tiles_b, tb = blockIdx.y % p.tiles_b;
    const int a0 = ta * TA, b0 = tb * TB;
    const int64_t r0 = static_cast<int64_t>(blockIdx.x) * p.rows_per_split;
    const int rows = static_cast<int>(min(p.rows_per_split, p.n - r0));

    // a thread copies the same columns of every RA-th (RB-th) row of a stage: addresses advance by constants
    constexpr int CA = TA / VA, RA = 256 / CA, LA = (BK + RA - 1) / RA;
    constexpr int CB = TB / VB, RB = 256 / CB, LB = (BK + RB - 1) / RB;
    const int ca_at = (tid % CA) * VA, ra = tid / CA, cb_at = (tid % CB) * VB, rb = tid / CB;
    const bool a_ok = a0 + ca_at < p.M, b_ok = b0 + cb_at < p.N;
    const float *pa = p.a + (r0 + ra) * p.lda + a0 + ca_at, *pb = p.b + (r0 + rb) * p.ldb + b0 + cb_at;
    const int64_t step_a = static_cast<int64_t>(RA) * p.lda, step_b = static_cast<int64_t>(RB) * p.ldb;

    auto load = [&](int k0, int st) {
        float *da = smem + st * BK * (TA + TB) + ra * TA + ca_at, *db = smem + st * BK * (TA + TB) + BK * TA + rb * TB + cb_at;
        const float *ga = pa + k0 * p.lda, *gb = pb + k0 * p.ldb;
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int k = ra + i * RA;
            if (BK % RA != 0 && k >= BK) break;
            const bool ok = a_ok && k0 + k < rows;
            cp_async<VA>(da + i * RA * TA, ok ? ga + i * step_a : p.a, ok);
        }
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int k = rb + i * RB;
            if (BK % RB != 0 && k >= BK) break;
            const bool ok = b_ok && k0 + k < rows;
            cp_async<VB>(db + i * RB * TB, ok ? gb + i * step_b : p.b, ok);
        }
    };
    uint64_t acc2[8][4];  // pairs of neighbouring columns of B
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc2[i][j] = 0;
    // column sums: four columns per thread, the threads left over take every sum_step-th row
    const bool sums = (p.sum_of == 1 && tb == 0) || (p.sum_of == 2 && ta == 0);
    const int sw = p.sum_of == 2 ? TB : TA, sum_off = p.sum_of == 2 ? BK * TA : 0;
    const int sum_c = (tid % (sw / 4)) * 4, sum_r = tid / (sw / 4), sum_step = 256 / (sw / 4);
    // compensated: a split's column is a chain of thousands of additions, and the library's sums are trees.  A sum that has
    // become infinite (an infinite value, or overflow) goes on without: the compensation would be inf - inf
    float4 cs = make_float4(0.f, 0.f, 0.f, 0.f), cc = cs;
    const auto add = [](float v, float &sum, float &comp) {
        const float y = __fsub_rn(v, comp), t = __fadd_rn(sum, y);
        comp = fabsf(t) < CUDART_INF_F ? __fsub_rn(__fsub_rn(t, sum), y) : 0.0f;
        sum = t;
    };

    const int steps = (rows + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load(s * BK, s);
        cp_async_commit();
    }
    for (int s = 0; s < steps; ++s) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        if (s + STAGES - 1 < steps) load((s + STAGES - 1) * BK, (s + STAGES - 1) % STAGES);
        cp_async_commit();
        const float *ca = smem + (s % STAGES) * BK * (TA + TB), *cb = ca + BK * TA;
#pragma unroll 4
        for (int k = g; k < BK; k += KG) {
            float av[8];
            uint64_t bv[4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float4 v = *reinterpret_cast<const float4 *>(ca + k * TA + ty * 4 + j * (TA / 2));
                av[4 * j] = v.x; av[4 * j + 1] = v.y; av[4 * j + 2] = v.z; av[4 * j + 3] = v.w;
                const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(cb + k * TB + tx * 4 + j * (TB / 2));
                bv[2 * j] = w.x; bv[2 * j + 1] = w.y;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t aa = pack2(av[i], av[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) fma2(acc2[i][j], aa, bv[j]);
            }
        }
        if (sums)
            for (int k = sum_r; k < BK; k += sum_step) {
                const float4 v = *reinterpret_cast<const float4 *>(ca + sum_off + k * sw + sum_c);
                add(v.x, cs.x, cc.x); add(v.y, cs.y, cc.y); add(v.z, cs.z, cc.z); add(v.w, cs.w, cc.w);
            }
    }
    cp_async_wait<0>();
    __syncthreads();
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) unpack2(acc2[i][j], acc[i][2 * j], acc[i][2 * j + 1]);
    float *part = p.partial + blockIdx.x * p.pstride;
    if (sums) {
        *reinterpret_cast<float4 *>(smem + sum_r * sw + sum_c) = cs;
        __syncthreads();
        const int at = (p.sum_of == 2 ? b0 : a0) + tid, width = p.sum_of == 2 ? p.N : p.M;
        if (tid < sw && at < width) {
            // up to 128 threads' sums: a plain chain over them would give away what the compensation has kept
            double v = 0.0;
            for (int r = 0; r < sum_step; ++r) v += smem[r * sw + tid];
            part[static_cast<int64_t>(p.M) * p.N + at] = static_cast<float>(v);
        }
        __syncthreads();
    }
#pragma unroll
    for (int h = KG / 2; h >= 1; h >>= 1) {
        if (g >= h && g < 2 * h) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) smem[(i * 8 + j) * (h * GT) + tid - h * GT] = acc[i][j];
        }
        __syncthreads();
        if (g < h) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] += smem[(i * 8 + j) * (h * GT) + tid];
        }
        __syncthreads();
    }
    if (g != 0) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int ra = a0 + ty * 4 + (i / 4) * (TA / 2) + (i & 3);
        if (ra >= p.M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int rb = b0 + tx * 4 + (j / 4) * (TB / 2) + (j & 3);
            if (rb < p.N) part[static_cast<int64_t>(ra) * p.N + rb] = acc[i][j];
        }
    }
}

// out = sum of the splits' partial results, in order and in 64 bits (up to 296 of them, which may nearly cancel: a bias
// gradient): 32 results per CTA, eight threads share a result's splits
__global__ void __launch_bounds__(256)
gram_reduce_kernel(const float *partial, int64_t pstride, int splits, int M, int N, int sums, float *out, int64_t sa,
                   int64_t sb, float *colsum) {
    __shared__ double s[8][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t e = static_cast<int64_t>(blockIdx.x) * 32 + lane, total = static_cast<int64_t>(M) * N + sums;
    double v = 0.0;
    if (e < total) {
#pragma unroll 8
        for (int k = w; k < splits; k += 8) v += partial[k * pstride + e];
    }
    s[w][lane] = v;
    __syncthreads();
    if (w != 0 || e >= total) return;
#pragma unroll
    for (int k = 1; k < 8; ++k) v += s[k][lane];
    if (e < static_cast<int64_t>(M) * N) out[(e / N) * sa + (e % N) * sb] = static_cast<float>(v);
    else colsum[e - static_cast<int64_t>(M) * N] = static_cast<float>(v);
}

struct GramTile {
    int ta, tb, bk;
};
static GramTile gram_tile(int64_t M, int64_t N) {  // M <= N
    if (M <= 8) return {8, 64, 64};
    if (M <= 16) return {16, 64, 64};
    if (M <= 32) return {32, 64, 32};
    if (N <= 64) return {64, 64, 32};
    if (M <= 64) return {64, 128, 16};
    return {128, 128, 16};
}
static int64_t gram_splits(int64_t n, int64_t M, int64_t N) {
    const GramTile t = gram_tile(M, N);
    const int64_t tiles = ((M + t.ta - 1) / t.ta) * ((N + t.tb - 1) / t.tb);
    // two CTAs per SM over all tiles, but no split of fewer than four stages of rows
    int64_t s = (2 * 148 + tiles - 1) / tiles;
    const int64_t most = (n + 4 * t.bk - 1) / (4 * t.bk);
    s = s < most ? s : most;
    return s < 1 ? 1 : s;
}

template <int TA, int TB, int BK>
static int launch_gram(GramParams p, int64_t splits, bool vec_a, bool vec_b, cudaStream_t st) {
    p.tiles_b = (p.N + TB - 1) / TB;
    const int tiles_a = (p.M + TA - 1) / TA;
    p.rows_per_split = ((p.n + splits - 1) / splits + BK - 1) / BK * BK;
    constexpr int smem = gram_smem_bytes<TA, TB, BK>();
    YITU_REQUIRE(static_cast<int64_t>(tiles_a) * p.tiles_b <= 65535 && p.rows_per_split < (1ll << 31), YITU_ERR_LIMIT,
                 "gram product too large");
    auto run = [&](auto kernel) -> int {
        if (smem > 48 * 1024) YITU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kernel<<<dim3(static_cast<unsigned>(splits), static_cast<unsigned>(tiles_a * p.tiles_b)), 256, smem, st>>>(p);
        YITU_LAUNCH_CHECK();
        return YITU_OK;
    };
    if (vec_a) return vec_b ? run(gram_kernel<TA, TB, BK, 4, 4>) : run(gram_kernel<TA, TB, BK, 4, 1>);
    return vec_b ? run(gram_kernel<TA, TB, BK, 1, 4>) : run(gram_kernel<TA, TB, BK, 1, 1>);
}

}  // namespace yitu

using namespace yitu;

extern "C" int yitu_linear_f32(int64_t n, int64_t K, int64_t N, const float *a, int64_t lda, const float *b, int64_t ldb,
                               int32_t b_transposed, const float *bias, float *c, int64_t ldc, yitu_stream_t stream) {
    YITU_REQUIRE(n >= 0 && K >= 1 && N >= 1 && K < (1ll << 30) && N < (1ll << 30), YITU_ERR_INVALID_ARG,
                 "bad shape (%lld x %lld x %lld)", (long long)n, (long long)K, (long long)N);
    YITU_REQUIRE(lda >= K && ldc >= N && ldb >= (b_transposed ? K : N), YITU_ERR_INVALID_ARG, "row strides smaller than the rows");
    if (n == 0) return YITU_OK;
    YITU_REQUIRE(a && b && c, YITU_ERR_INVALID_ARG, "NULL tensor");
    LinearParams p{};
    p.n = n; p.K = static_cast<int>(K); p.N = static_cast<int>(N);
    p.a = a; p.lda = lda; p.b = b; p.ldb = ldb; p.bias = bias; p.c = c; p.ldc = ldc;
    p.vec_c = N % 4 == 0 && ldc % 4 == 0 && aligned16(c);
    const bool vec_a = K % 4 == 0 && lda % 4 == 0 && aligned16(a);
    const bool vec_b = !b_transposed && N % 4 == 0 && ldb % 4 == 0 && aligned16(b);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // tile by the result's width; below two CTAs per SM a quarter of the rows per CTA
    if (N <= 8) return n < 148 * 2 * 256 ? launch_linear<1, 4, 2, 64>(p, b_transposed, vec_a, vec_b, st) : launch_linear<4, 4, 2, 64>(p, b_transposed, vec_a, vec_b, st);
    if (N <= 16) return n < 148 * 2 * 256 ? launch_linear<2, 4, 4, 32>(p, b_transposed, vec_a, vec_b, st) : launch_linear<8, 4, 4, 32>(p, b_transposed, vec_a, vec_b, st);
    if (N <= 32) return n < 148 * 2 * 128 ? launch_linear<2, 4, 8, 16>(p, b_transposed, vec_a, vec_b, st) : launch_linear<8, 4, 8, 16>(p, b_transposed, vec_a, vec_b, st);
    const int64_t tiles64 = (N + 63) / 64;
    if ((n + 127) / 128 * tiles64 < 148 * 2) return launch_linear<4, 4, 16, 8>(p, b_transposed, vec_a, vec_b, st);
    if (N <= 64 || (n + 127) / 128 * ((N + 127) / 128) < 148 * 2) return launch_linear<8, 8, 8, 16>(p, b_transposed, vec_a, vec_b, st);
    return launch_linear<8, 8, 16, 16>(p, b_transposed, vec_a, vec_b, st);
}

extern "C" int64_t yitu_gram_scratch_bytes(int64_t n, int64_t M, int64_t N, int32_t column_sums) {
    if (n < 0 || M < 1 || N < 1) return -1;
    const int64_t lo = M < N ? M : N, hi = M < N ? N : M;
    return gram_splits(n, lo, hi) * (M * N + (column_sums ? M : 0)) * static_cast<int64_t>(sizeof(float));
}

extern "C" int yitu_gram_f32(int64_t n, int64_t M, int64_t N, const float *a, int64_t lda, const float *b, int64_t ldb,
                             float *c, float *a_sums, float *scratch, int64_t scratch_bytes, yitu_stream_t stream) {
    YITU_REQUIRE(n >= 0 && M >= 1 && N >= 1 && M < (1ll << 24) && N < (1ll << 24), YITU_ERR_INVALID_ARG,
                 "bad shape (%lld x %lld x %lld)", (long long)n, (long long)M, (long long)N);
    YITU_REQUIRE(lda >= M && ldb >= N && c, YITU_ERR_INVALID_ARG, "row strides smaller than the rows, or no output");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (n == 0) {
        YITU_CUDA(cudaMemsetAsync(c, 0, M * N * sizeof(float), st));
        if (a_sums) YITU_CUDA(cudaMemsetAsync(a_sums, 0, M * sizeof(float), st));
        return YITU_OK;
    }
    YITU_REQUIRE(a && b, YITU_ERR_INVALID_ARG, "NULL tensor");
    const int64_t need = yitu_gram_scratch_bytes(n, M, N, a_sums != nullptr);
    YITU_REQUIRE(scratch && scratch_bytes >= need, YITU_ERR_WORKSPACE, "gram product needs %lld bytes of scratch",
                 (long long)need);
    const bool vec_a = M % 4 == 0 && lda % 4 == 0 && aligned16(a), vec_b = N % 4 == 0 && ldb % 4 == 0 && aligned16(b);
    GramParams p{};
    p.n = n;
    p.partial = scratch;
    p.pstride = M * N + (a_sums ? M : 0);
    const bool swap = M > N;  // the kernel's first operand is the narrower one
    if (!swap) {
        p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.a = a; p.lda = lda; p.b = b; p.ldb = ldb;
        p.sum_of = a_sums ? 1 : 0;
    } else {
        p.M = static_cast<int>(N); p.N = static_cast<int>(M); p.a = b; p.lda = ldb; p.b = a; p.ldb = lda;
        p.sum_of = a_sums ? 2 : 0;
    }
    const bool va = swap ? vec_b : vec_a, vb = swap ? vec_a : vec_b;
    const GramTile t = gram_tile(p.M, p.N);
    int64_t splits = gram_splits(n, p.M, p.N);
    {   // rows are handed out in whole stages: no split may be left without any
        const int64_t rps = ((n + splits - 1) / splits + t.bk - 1) / t.bk * t.bk;
        splits = (n + rps - 1) / rps;
    }
    int rc;
    if (t.ta == 8) rc = launch_gram<8, 64, 64>(p, splits, va, vb, st);
    else if (t.ta == 16) rc = launch_gram<16, 64, 64>(p, splits, va, vb, st);
    else if (t.ta == 32) rc = launch_gram<32, 64, 32>(p, splits, va, vb, st);
    else if (t.tb == 64) rc = launch_gram<64, 64, 32>(p, splits, va, vb, st);
    else if (t.ta == 64) rc = launch_gram<64, 128, 16>(p, splits, va, vb, st);
    else rc = launch_gram<128, 128, 16>(p, splits, va, vb, st);
    if (rc) return rc;
    const int64_t total = p.pstride;
    gram_reduce_kernel<<<static_cast<unsigned>((total + 31) / 32), 256, 0, st>>>(
        scratch, p.pstride, static_cast<int>(splits), p.M, p.N, a_sums ? static_cast<int>(M) : 0, c, swap ? 1 : N, swap ? N : 1,
        a_sums);
    YITU_LAUNCH_CHECK();
    return YITU_OK;
}
