// SDDMM on CUDA cores: out[e] = s_e * <X[row(e), :], Y[col(e), :]> (sm_103a), fp32 or bf16
// operands, fp32 products and sums.
//
// A group of G lanes takes one edge at a time (G = about one lane per four 4-element blocks of
// K, a power of two up to a warp), so each Y row is read by neighbouring lanes in 16-byte (fp32) or
// 8-byte (bf16) pieces -- coalesced -- and the X row, shared by the consecutive edges of one
// row, comes from L1. A group walks a chunk of consecutive edges in CSR order: one binary
// search over rowptr for its first edge (the reference searches per edge, findRow in
// gcn/pytorch-custom/computeUtil.h:11-28), then the row pointer steps forward; the COO form
// reads each edge's row from the row array (the reference's sddmm_cuda_coo, sddmm.cu:427-457).
//
// Summation order (the oracle's or_sddmm_csr_f32_group): lane l runs one fused-FMA chain over
// the blocks l, l + G, l + 2G, ... of K in order; the lanes are summed by a butterfly
// (acc += shfl_xor(acc, off), off = G/2 .. 1); lane 0 writes s_e * sum. bf16 operands use the
// mixed-precision FMA of sm_100+ (a bf16 x bf16 product is exact in fp32), so the bf16 kernel
// gives bit for bit the fp32 kernel's result on the widened values.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace as {
namespace {

constexpr int kThreads = 256;
constexpr int kWalkRows = 64;  // rows walked (from L1) before the next one is searched for (from L2)
constexpr int kFarRows = 16;   // rows an edge past which a chunk of sddmm_rows searches

// acc = fma(x0, y0, acc); acc = fma(x1, y1, acc) for the bf16 halves of x and y, in order.
__device__ __forceinline__ void fma_bf16_seq2(unsigned x, unsigned y, float &acc) {
    asm("{\n .reg .b16 xl, xh, yl, yh;\n mov.b32 {xl, xh}, %1;\n mov.b32 {yl, yh}, %2;\n"
        " fma.rn.f32.bf16 %0, xl, yl, %0;\n fma.rn.f32.bf16 %0, xh, yh, %0;\n}\n"
        : "+f"(acc) : "r"(x), "r"(y));
}

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(uint16_t v) { return bf16_to_f32(v); }

// One 4-element block of the dot product, elements in order.
template <typename T>
struct Block;
template <>
struct Block<float> {
    using Raw = float4;
    __device__ static Raw load(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
    __device__ static Raw load_here(const float *p) {
        Raw v;
        asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "l"(p));
        return v;
    }
    __device__ static void chain(const Raw &x, const Raw &y, float &acc) {
        acc = fmaf(x.x, y.x, acc);
        acc = fmaf(x.y, y.y, acc);
        acc = fmaf(x.z, y.z, acc);
        acc = fmaf(x.w, y.w, acc);
    }
};
template <>
struct Block<uint16_t> {
    using Raw = uint2;
    __device__ static Raw load(const uint16_t *p) { return __ldg(reinterpret_cast<const uint2 *>(p)); }
    __device__ static Raw load_here(const uint16_t *p) {
        Raw v;
        asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
        return v;
    }
    __device__ static void chain(const Raw &x, const Raw &y, float &acc) {
        fma_bf16_seq2(x.x, y.x, acc);
        fma_bf16_seq2(x.y, y.y, acc);
    }
};

// Lane's chain over the blocks g, g + G, ... of one edge, four blocks at a time with all
// their loads issued before the FMAs. VEC: K % 4 == 0 and 4-element aligned rows, one vector
// load per block; else element loads (elements past K contribute nothing).
template <typename T, bool VEC, int G>
__device__ __forceinline__ float lane_chain(const T *xr, const T *yr, int K, int g) {
    using B = Block<T>;
    const int nq = (K + 3) >> 2;
    float acc = 0.0f;
    for (int q = g; q < nq; q += 4 * G) {
        if (VEC) {
            typename B::Raw x[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int qq = q + u * G;
                if (qq < nq) {
                    x[u] = B::load(xr + 4 * qq);
                    y[u] = B::load(yr + 4 * qq);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (q + u * G < nq) B::chain(x[u], y[u], acc);
        } else {
            float x[4][4], y[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int k = 4 * (q + u * G) + i;
                    x[u][i] = k < K ? to_f32(xr[k]) : 0.0f;
                    y[u][i] = k < K ? to_f32(yr[k]) : 0.0f;
                }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (4 * (q + u * G) + i < K) acc = fmaf(x[u][i], y[u][i], acc);
        }
    }
    return acc;
}

// Moves a group on to the row of entry e (r, its start and end): row by row, then (a long run of
// empty rows) by a search. Uniform over the group. (2M rows, 100,000
// entries, the last after 1.9M empty rows: 110 ms row by row, 0.10 with the search.)
template <int G>
__device__ __forceinline__ void next_row(const int *__restrict__ rowptr, int M, int e, int g,
                                         unsigned gmask, int &r, int &rs, int &re) {
    if (e < re) return;
    const int stop = r < M - kWalkRows ? r + kWalkRows : M - 1;
#pragma unroll 1
    while (e >= re && r < stop) {
        ++r;
        rs = re;
        re = __ldg(rowptr + r + 1);
    }
    if (e >= re && r + 1 < M) {
        r = find_row<G>(rowptr, M, e, g, gmask);
        rs = __ldg(rowptr + r);
        re = __ldg(rowptr + r + 1);
    }
}

// One group's edges e0 .. e1 - 1, one at a time. COO: rows come per edge from `rows` (any order);
// CSR: `rows` is the row pointer and r the row of edge e0.
template <typename T, bool VEC, int G, bool COO>
__device__ __forceinline__ void group_edges(int M, int N, int K, long e0, long e1, int r,
                                            const int *__restrict__ rows,
                                            const int *__restrict__ colind,
                                            const float *__restrict__ aval,
                                            const T *__restrict__ X, long ldx,
                                            const T *__restrict__ Y, long ldy,
                                            float *__restrict__ out, int g, unsigned gmask,
                                            unsigned *status) {
    int rs = 0, re = 0;
    if (!COO) {
        rs = __ldg(rows + r);
        re = __ldg(rows + r + 1);
    }
    for (long e = e0; e < e1; ++e) {  // every branch below is the same for the whole group
        int row;
        if (COO) {
            row = ld_stream(rows + e);
            if (static_cast<unsigned>(row) >= static_cast<unsigned>(M)) {
                if (g == 0) {
                    flag(status, kFlagBadRowptr);
                    out[e] = 0.0f;
                }
                continue;
            }
        } else {
            next_row<G>(rows, M, static_cast<int>(e), g, gmask, r, rs, re);
            if (rs > e || re <= e) {
                if (g == 0) {
                    flag(status, kFlagBadRowptr);
                    out[e] = 0.0f;
                }
                continue;
            }
            row = r;
        }
        const int c = ld_stream(colind + e);
        if (static_cast<unsigned>(c) >= static_cast<unsigned>(N)) {
            if (g == 0) {
                flag(status, kFlagBadColind);
                out[e] = 0.0f;
            }
            continue;
        }
        float acc = lane_chain<T, VEC, G>(X + static_cast<long>(row) * ldx,
                                          Y + static_cast<long>(c) * ldy, K, g);
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(gmask, acc, off, G);
        if (g == 0) out[e] = aval ? __ldg(aval + e) * acc : acc;
    }
}

template <typename T, bool VEC, int G, bool COO>
__global__ void __launch_bounds__(kThreads)
sddmm_group(int M, int N, int K, int nnz, int CH, const int *__restrict__ rows,
            const int *__restrict__ colind, const float *__restrict__ aval,
            const T *__restrict__ X, long ldx, const T *__restrict__ Y, long ldy,
            float *__restrict__ out, unsigned *status) {
    const long grp = (static_cast<long>(blockIdx.x) * kThreads + threadIdx.x) / G;
    const int g = threadIdx.x % G;
    const unsigned gmask =
        G == 32 ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    const long e0 = grp * CH;
    if (e0 >= nnz) return;  // the whole group leaves together
    const long e1 = e0 + CH < nnz ? e0 + CH : nnz;
    const int r = COO ? 0 : find_row<G>(rows, M, e0, g, gmask);
    group_edges<T, VEC, G, COO>(M, N, K, e0, e1, r, rows, colind, aval, X, ldx, Y, ldy, out, g,
                                gmask, status);
}

// The CSR form where a lane's part of a row is at most four blocks (K <= 16 G) and rows are
// aligned: X's row stays in registers while the row lasts, the next edge's Y row is loaded (and
// the column of the one after it read) while the present edge is summed. The sums are
// sddmm_group's, in the same order. What bounds it is Y's gathers, so warps in flight count: on a
// graph of 6M entries with K = 128 it takes 350 us with four CTAs per SM (64 registers), 425 with
// three, 655 with five (spills); two edges per turn, 488; sddmm_group 461; with the search in the
// walk 423. bf16 rows leave room for five. (K = 512: 1.24 and 2.23
// ms; K = 16: 0.21 and 0.31.) The loads are volatile because left to the compiler they move down
// to their uses.
template <typename T, int G>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 4 ? 4 : 5)
sddmm_rows(int M, int N, int K, int nnz, int CH, const int *__restrict__ rowptr,
           const int *__restrict__ colind, const float *__restrict__ aval,
           const T *__restrict__ X, long ldx, const T *__restrict__ Y, long ldy,
           float *__restrict__ out, unsigned *status) {
    using B = Block<T>;
    const long grp = (static_cast<long>(blockIdx.x) * kThreads + threadIdx.x) / G;
    const int g = threadIdx.x % G;
    const unsigned gmask =
        G == 32 ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    if (grp * CH >= nnz) return;  // the whole group leaves together
    const int e0 = static_cast<int>(grp * CH);
    const int e1 = CH < nnz - e0 ? e0 + CH : nnz;
    const int nq = K >> 2;
    int r = find_row<G>(rowptr, M, e0, g, gmask);
    const long far = static_cast<long>(r) + kFarRows * CH;
    const int far_start = far < M ? __ldg(rowptr + far) : e1;  // (read early, looked at late)
    const int rs = __ldg(rowptr + r);
    int re = __ldg(rowptr + r + 1);
    auto load = [&](const T *row, typename B::Raw (&v)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (g + u * G < nq) v[u] = B::load_here(row + 4 * (g + u * G));
    };
    // (unsigned: an entry ahead of 2^31 - 1 of them is past e1, not below zero)
    auto column = [&](unsigned e) {
        return e < static_cast<unsigned>(e1) ? ld_stream(colind + e) : -1;
    };
    auto in_range = [&](int c) { return static_cast<unsigned>(c) < static_cast<unsigned>(N); };
    typename B::Raw x[4], y[4], yn[4];
    int held = -1;  // the row that x holds
    int c = column(e0), cn = column(e0 + 1u);
    if (in_range(c)) load(Y + c * ldy, y);
    // a chunk over more than kFarRows rows an edge (a long run of empty ones) goes the way that
    // searches: the walk below is row by row, and a search in it costs it registers (so does one
    // whose first row starts past its first edge: a malformed pointer)
    if (far_start < e1 || rs > e0) {
        group_edges<T, true, G, false>(M, N, K, e0, e1, r, rowptr, colind, aval, X, ldx, Y, ldy, out,
                                       g, gmask, status);
        return;
    }
    for (int e = e0; e < e1; ++e) {  // every branch below is the same for the whole group
        while (e >= re && r + 1 < M) {
            ++r;
            re = __ldg(rowptr + r + 1);
        }
        if (in_range(cn)) load(Y + cn * ldy, yn);
        const int cnn = column(e + 2u);
        const bool row_ok = re > e;
        if (row_ok && in_range(c)) {
            if (held != r) {
                load(X + r * ldx, x);
                held = r;
            }
            float acc = 0.0f;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (g + u * G < nq) B::chain(x[u], y[u], acc);
#pragma unroll
            for (int off = G / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(gmask, acc, off, G);
            if (g == 0) out[e] = aval ? __ldg(aval + e) * acc : acc;
        } else if (g == 0) {
            flag(status, row_ok ? kFlagBadColind : kFlagBadRowptr);
            out[e] = 0.0f;
        }
        c = cn;
        cn = cnn;
#pragma unroll
        for (int u = 0; u < 4; ++u) y[u] = yn[u];
    }
}

int group_size(int K) {  // the oracle's or_sddmm_group_size: about four blocks per lane
    const int q = (K + 15) / 16;
    int g = 1;
    while (g < q && g < 32) g <<= 1;
    return g;
}

template <typename T, bool COO>
as_status launch_group(as_ctx *ctx, int M, int N, int K, int nnz, const int *rows,
                       const int *colind, const float *aval, const T *X, long ldx, const T *Y,
                       long ldy, float *out, cudaStream_t s, const char *what) {
    if (M == 0) return fail(AS_ERR_INVALID_CSR, "sddmm: nnz > 0 with zero rows");
    const int esz = static_cast<int>(sizeof(T));
    const bool vec = K % 4 == 0 && ldx % 4 == 0 && ldy % 4 == 0 &&
                     reinterpret_cast<uintptr_t>(X) % (4 * esz) == 0 &&
                     reinterpret_cast<uintptr_t>(Y) % (4 * esz) == 0;
    const int G = group_size(K);
    // K in (0, 16 G]: every lane's blocks fit its registers
    // (and rows are not mostly empty: most of its chunks would leave for the loop that searches)
    const bool resident = !COO && vec && K > 0 && K <= 16 * G && N > 0 && M <= 4L * nnz;
    int CH = G >= 32 ? 4 : 128 / G;  // edges per group: more for short dot products
    if (resident) {
        // Edges per group: as many as leave four waves of the CTAs that an SM holds (four of fp32, five
        // of bf16), up to 64; where that is under 16, as many as leave two whole waves, up to 16: a
        // chunk's first row is searched for, which a few short edges do not pay for (2.4M entries, K =
        // 20: 99 us with chunks of 7, 72 with 16; 600,000, K = 128: 41 and 35), but a chunk is walked
        // in order (20,000 entries, K = 132: 8 us with chunks of 4, 12 with 16).
        const long lanes = static_cast<long>(nnz) * G;
        const long wave = (sizeof(T) == 4 ? 4L : 5L) * kThreads * ctx->sms;
        long n = lanes / (4L * 4 * kThreads * ctx->sms);
        if (n < 16) n = std::min(16L, static_cast<long>(ceil_div(lanes, 2 * wave)));
        CH = static_cast<int>(n < 4 ? 4 : n > 64 ? 64 : n);
    }
    const long groups = ceil_div(nnz, CH);
    const unsigned grid = static_cast<unsigned>(ceil_div(groups * G, kThreads));
#define AS_SDDMM_G(GV)                                                                      \
    case GV:                                                                                \
        if (resident) {                                                                     \
            if constexpr (!COO)                                                             \
                sddmm_rows<T, GV><<<grid, kThreads, 0, s>>>(M, N, K, nnz, CH, rows, colind, \
                                                            aval, X, ldx, Y, ldy, out,      \
                                                            ctx->d_status);                 \
        } else if (vec)                                                                            \
            sddmm_group<T, true, GV, COO><<<grid, kThreads, 0, s>>>(                        \
                M, N, K, nnz, CH, rows, colind, aval, X, ldx, Y, ldy, out, ctx->d_status);  \
        else                                                                                \
            sddmm_group<T, false, GV, COO><<<grid, kThreads, 0, s>>>(                       \
                M, N, K, nnz, CH, rows, colind, aval, X, ldx, Y, ldy, out, ctx->d_status);  \
        break;
    switch (G) {
        AS_SDDMM_G(1) AS_SDDMM_G(2) AS_SDDMM_G(4) AS_SDDMM_G(8) AS_SDDMM_G(16) AS_SDDMM_G(32)
        default: return fail(AS_ERR_UNSUPPORTED, "sddmm: group size");
    }
#undef AS_SDDMM_G
    ctx->launches++;
    return check_cuda(cudaGetLastError(), what);
}

}  // namespace

as_status sddmm_f32_launch(as_ctx *ctx, int M, int N, int K, int nnz, const int *rowptr,
                           const int *colind, const float *aval, const float *X, long ldx,
                           const float *Y, long ldy, float *out, cudaStream_t s) {
    return launch_group<float, false>(ctx, M, N, K, nnz, rowptr, colind, aval, X, ldx, Y, ldy,
                                      out, s, "sddmm_f32 launch");
}

as_status sddmm_bf16_launch(as_ctx *ctx, int M, int N, int K, int nnz, const int *rowptr,
                            const int *colind, const float *aval, const uint16_t *X, long ldx,
                            const uint16_t *Y, long ldy, float *out, cudaStream_t s) {
    return launch_group<uint16_t, false>(ctx, M, N, K, nnz, rowptr, colind, aval, X, ldx, Y,
                                         ldy, out, s, "sddmm_bf16 launch");
}

as_status sddmm_coo_f32_launch(as_ctx *ctx, int M, int N, int K, int nnz, const int *rowind,
                               const int *colind, const float *aval, const float *X, long ldx,
                               const float *Y, long ldy, float *out, cudaStream_t s) {
    return launch_group<float, true>(ctx, M, N, K, nnz, rowind, colind, aval, X, ldx, Y, ldy,
                                     out, s, "sddmm_coo_f32 launch");
}

}  // namespace as
