// Sparse x sparse -> dense (sm_103a): C = beta*C + A*B with A (M x K) and B (K x N) in CSR and
// C dense row-major, bit-identical to the reference's sparse_matrix_mul3 (SpMM.cpp:309-327,
// built with FMA contraction): every output element is one fused-FMA chain over the entries
// of A's row in CSR order, each entry k contributing B[k, j] when B's row k holds column j.
//
// One warp per (row of A, tile of output columns). The tile's accumulators live in shared
// memory, start as beta*C, and take A's entries in order: for each, the lanes walk B's row k
// (one B entry per lane) and update acc[j] = fmaf(a, b, acc[j]) for the j in the tile. The
// columns of one B row are distinct, so no two lanes touch one accumulator in a step, and
// __syncwarp orders the steps.
//
// A warp reads B's rows whole for every tile, so the tile is as wide as leaves a warp for every
// scheduler: 4096 columns (16 KB, 14 warps per SM) when A has rows enough, down to 1024 for few
// rows. What bounds it then is the chain of steps (a shared-memory read, the FMA and the write, 50
// cycles or so) and B's latency: the (row start, row end) of B for 32 entries of A come with one
// load per lane, and the first 64 entries of the next kBatch rows of B are loaded while the
// present ones are applied. Measured on 4096 x 4096 operands of density 0.01 (C from zero): 47 us with
// one warp per CTA, 53 with two, 58 with 2048-column tiles; 96 with 1024-column tiles and the second
// 32 entries of each row of B loaded when their turn came.
#include "common.cuh"
#include "internal.h"

namespace as {
namespace {

constexpr int kWarps = 1;      // per CTA: rows are taken as single warps finish
constexpr int kThreads = 32 * kWarps;
constexpr int kMaxTile = 4096;  // output columns per warp (16 KB of accumulators)
constexpr int kMinTile = 1024;
constexpr int kBatch = 4;       // rows of B loaded together

// The first 64 entries of kBatch rows of B, two per lane.
struct Batch {
    float a[kBatch];
    unsigned s[kBatch], e[kBatch];   // the rows' extents (empty past the end)
    int j[kBatch][2];
    float b[kBatch][2];
};

__global__ void __launch_bounds__(kThreads)
spgemm_dense(int M, int K, int N, int tile, int nnz_a, int nnz_b, const int *__restrict__ rp1,
             const int *__restrict__ ci1, const float *__restrict__ v1,
             const int *__restrict__ rp2, const int *__restrict__ ci2,
             const float *__restrict__ v2, float *__restrict__ C, long ldc, float beta,
             bool vec, unsigned *status) {
    extern __shared__ __align__(16) float acc_s[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long row = static_cast<long>(blockIdx.x) * kWarps + warp;
    if (row >= M) return;  // warps are independent: no CTA-wide barrier below
    const int tile0 = blockIdx.y * tile;
    const int tw = min(tile, N - tile0);
    float *acc = acc_s + warp * tile;
    float *crow = C + row * ldc + tile0;
    const int tv = vec ? tw & ~3 : 0;  // columns in whole aligned vectors
    for (int j = 4 * lane; j < tv; j += 128) {
        float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (beta != 0.0f) {
            c = *reinterpret_cast<const float4 *>(crow + j);
            c.x *= beta; c.y *= beta; c.z *= beta; c.w *= beta;
        }
        *reinterpret_cast<float4 *>(acc + j) = c;
    }
    for (int j = tv + lane; j < tw; j += 32) acc[j] = beta != 0.0f ? crow[j] * beta : 0.0f;
    __syncwarp();

    int lo, hi;
    row_range(rp1, static_cast<int>(row), nnz_a, status, lo, hi);
    // entries are counted unsigned: one read ahead of 2^31 - 1 of them is past the end, not below zero
    const unsigned a_end = hi;
    for (unsigned base = lo; base < a_end; base += 32) {
        // this lane's A entry: its value and the extent of B's row
        const unsigned e = base + lane;
        float a = 0.0f;
        unsigned bs = 0, be = 0;
        if (e < a_end) {
            const int k = ld_stream(ci1 + e);
            a = ld_stream(v1 + e);
            if (static_cast<unsigned>(k) >= static_cast<unsigned>(K)) {
                flag(status, kFlagBadColind);
            } else {
                const int s = __ldg(rp2 + k), t = __ldg(rp2 + k + 1);
                if (s < 0 || t < s || t > nnz_b) {
                    flag(status, kFlagBadRowptr);
                } else {
                    bs = s;
                    be = t;
                }
            }
        }
        const int cnt = static_cast<int>(min(32u, a_end - base));
        auto load = [&](int u0, Batch &x) {
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int u = min(u0 + q, 31);
                x.a[q] = __shfl_sync(0xffffffffu, a, u);
                x.s[q] = __shfl_sync(0xffffffffu, bs, u);
                x.e[q] = __shfl_sync(0xffffffffu, be, u);
                if (u0 + q >= cnt) x.e[q] = x.s[q];  // past A's entries: nothing to apply
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const unsigned t = x.s[q] + 32 * h + lane;
                    x.j[q][h] = -1;
                    x.b[q][h] = 0.0f;
                    if (t < x.e[q]) {
                        x.j[q][h] = __ldg(ci2 + t);
                        x.b[q][h] = __ldg(v2 + t);
                    }
                }
            }
        };
        // one step: this lane's entry (column j, where it has one) of one row of B
        auto apply = [&](float av, bool has, int j, float b) {
            if (has) {
                if (static_cast<unsigned>(j) >= static_cast<unsigned>(N))
                    flag(status, kFlagBadColind);
                else if (j >= tile0 && j < tile0 + tw)
                    acc[j - tile0] = fmaf(av, b, acc[j - tile0]);
            }
            __syncwarp();
        };
        Batch x;
        load(0, x);
        for (int u0 = 0; u0 < cnt; u0 += kBatch) {
            Batch next;
            load(u0 + kBatch, next);
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int n = static_cast<int>(x.e[q] - x.s[q]);
                apply(x.a[q], lane < n, x.j[q][0], x.b[q][0]);
                if (n > 32) apply(x.a[q], 32 + lane < n, x.j[q][1], x.b[q][1]);
                for (unsigned t0 = x.s[q] + 64; t0 < x.e[q]; t0 += 32) {  // longer rows of B
                    const unsigned t = t0 + lane;
                    const bool has = t < x.e[q];
                    apply(x.a[q], has, has ? __ldg(ci2 + t) : 0, has ? __ldg(v2 + t) : 0.0f);
                }
            }
            x = next;
        }
    }
    __syncwarp();
    for (int j = 4 * lane; j < tv; j += 128)
        __stcs(reinterpret_cast<float4 *>(crow + j), *reinterpret_cast<const float4 *>(acc + j));
    for (int j = tv + lane; j < tw; j += 32) crow[j] = acc[j];
}

}  // namespace

as_status spgemm_dense_launch(as_ctx *ctx, int M, int K, int N, int nnz_a, const int *rp1,
                              const int *ci1, const float *v1, int nnz_b, const int *rp2,
                              const int *ci2, const float *v2, float *C, long ldc, float beta,
                              cudaStream_t s) {
    // the widest tile that still gives 12 warps per SM
    int tile = kMaxTile;
    while (tile > kMinTile && static_cast<long>(M) * ceil_div(N, tile) < 12L * ctx->sms) tile /= 2;
    const long tiles = ceil_div(N, tile);
    if (ceil_div(N, kMinTile) > 65535) return fail(AS_ERR_UNSUPPORTED, "spgemm_dense: N too large");
    const int held = static_cast<int>(min(static_cast<long long>(tile), ceil_div(N, 4) * 4));
    const bool vec = ldc % 4 == 0 && reinterpret_cast<uintptr_t>(C) % 16 == 0;
    dim3 grid(static_cast<unsigned>(ceil_div(M, kWarps)), static_cast<unsigned>(tiles));
    spgemm_dense<<<grid, kThreads, kWarps * held * sizeof(float), s>>>(
        M, K, N, held, nnz_a, nnz_b, rp1, ci1, v1, rp2, ci2, v2, C, ldc, beta, vec, ctx->d_status);
    ctx->launches++;
    return check_cuda(cudaGetLastError(), "spgemm_dense launch");
}

}  // namespace as
