// Softmax cross-entropy over rows of class scores in bf16 storage (sm_103a): the GCN's loss,
// log_softmax followed by the mean negative log-likelihood (gcn/pytorch-custom/gcn_custom.py,
// model output :90, loss :122-126), as one pass over the scores each way instead of torch's
// chain of slice, widen, log_softmax, gather, mean and their backward kernels.
//
// Forward: one thread per row streams the row in 8-score vectors with the running maximum and
// rescaled sum of the online softmax, so nothing is held per class: lse = m + log(s),
// loss_i = lse - x[label], and lse is kept for the backward. Rows are summed per CTA by a fixed
// tree, the CTA sums by one more fixed tree, then divided by n: deterministic.
// Backward: G[i, j] = (exp(x_j - lse_i) - [j == label]) * gscale / n in bf16 (round to nearest
// even), zero in the padding columns C .. width-1; gscale is read from device memory (the
// upstream gradient), so nothing synchronises. A thread works on its own row; its 16-byte loads
// and stores each touch 32 rows per instruction of its warp. Where scores and gradients pass through
// the caches without staying (park_rows), lines are evicted before they are used whole; there a CTA
// moves its rows as one run between memory and shared memory, neighbouring threads neighbouring
// pieces (a piece of padding per row keeps the accesses free of bank conflicts), and the gradients
// take the scores' place there: 2.4M rows of 48 in 138 us, 253 without; with only the gradients
// parked 278. (The forward, with nothing to store, lost by it: 106 us in place of 82.)
#include "common.cuh"
#include "internal.h"
#include "spmm_vec.cuh"

namespace as {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxC = 64;  // classes per row (bounds the unrolled vector loops)

__device__ __forceinline__ void unpack8(const uint4 &w, float (&x)[8]) {
    const unsigned u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        x[2 * q] = __uint_as_float(u[q] << 16);
        x[2 * q + 1] = __uint_as_float(u[q] & 0xffff0000u);
    }
}

// Scores [8v, 8v + 8) of a row as fp32: one 16-byte load when VEC, else element loads (with
// elements at or past `lim` left at -inf).
template <bool VEC>
__device__ __forceinline__ void load8(const uint16_t *row, int v, int lim, float (&x)[8]) {
    if (VEC) {
        unpack8(__ldcs(reinterpret_cast<const uint4 *>(row) + v), x);
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = 8 * v + q < lim ? bf16_to_f32(row[8 * v + q]) : -INFINITY;
    }
}

// Fixed-order sum over the CTA: butterfly within warps, then warp totals in warp order.
__device__ __forceinline__ float block_sum(float v, float *sm) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    float t = 0.0f;
    if (threadIdx.x == 0)
        for (int w = 0; w < kThreads / 32; ++w) t += sm[w];
    return t;  // meaningful in thread 0
}

template <bool VEC>
__global__ void __launch_bounds__(kThreads)
xent_fwd(int n, int C, const uint16_t *__restrict__ S, long lds,
         const int64_t *__restrict__ labels, float *__restrict__ lse_out,
         float *__restrict__ partial, unsigned *status) {
    __shared__ float sm[kThreads / 32];
    const long i = static_cast<long>(blockIdx.x) * kThreads + threadIdx.x;
    float li = 0.0f;
    if (i < n) {
        const uint16_t *row = S + i * lds;
        const int64_t t = labels[i];
        float m = -INFINITY, sum = 0.0f, xt = 0.0f;
#pragma unroll
        for (int v = 0; v < kMaxC / 8; ++v) {
            if (8 * v >= C) break;
            float x[8];
            load8<VEC>(row, v, C, x);
            float mv = m;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (8 * v + q < C) mv = fmaxf(mv, x[q]);
            float sv = 0.0f;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (8 * v + q < C) sv += expf(x[q] - mv);
                if (8 * v + q == t) xt = x[q];
            }
            sum = sum * expf(m - mv) + sv;  // exp(-inf) = 0 on the first vector
            m = mv;
        }
        const float lse = m + logf(sum);
        lse_out[i] = lse;
        if (t < 0 || t >= C)
            flag(status, kFlagBadLabel);
        else
            li = lse - xt;
    }
    const float tot = block_sum(li, sm);
    if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

// One CTA: the partials in a fixed order (each thread a strided run, then block_sum), / n.
__global__ void __launch_bounds__(kThreads)
xent_finish(int nparts, const float *__restrict__ partial, float inv_n, float *__restrict__ loss) {
    __shared__ float sm[kThreads / 32];
    float v = 0.0f;
    for (int p = threadIdx.x; p < nparts; p += kThreads) v += partial[p];
    const float t = block_sum(v, sm);
    if (threadIdx.x == 0) *loss = t * inv_n;
}

// VEC: 16-byte score loads and 16-byte gradient stores (width a multiple of 8, rows aligned). PARK
// (with VEC): by way of shared memory.
template <bool VEC, bool PARK>
__global__ void __launch_bounds__(kThreads)
xent_bwd(int n, int C, const uint16_t *__restrict__ S, long lds,
         const int64_t *__restrict__ labels, const float *__restrict__ lse_in,
         const float *__restrict__ gscale, float inv_n, uint16_t *__restrict__ G, long ldg,
         int width) {
    constexpr int kPitch = kMaxC / 8 + 1;  // 16-byte pieces per parked row
    __shared__ uint4 parked[PARK ? kThreads * kPitch : 1];
    const long row0 = static_cast<long>(blockIdx.x) * kThreads;
    const int rows = static_cast<int>(min(static_cast<long>(kThreads), n - row0));
    if (PARK) {
        const int pieces = (C + 7) / 8;
        for (int j = threadIdx.x; j < rows * pieces; j += kThreads) {
            const int r = j / pieces, p = j - r * pieces;
            parked[r * kPitch + p] =
                __ldcs(reinterpret_cast<const uint4 *>(S + (row0 + r) * lds) + p);
        }
        __syncthreads();
    } else if (threadIdx.x >= rows) {
        return;
    }
    uint4 *mine = parked + (PARK ? threadIdx.x * kPitch : 0);
    const long i = row0 + min(static_cast<int>(threadIdx.x), rows - 1);  // past the end: not stored
    const uint16_t *row = S + i * lds;
    const int64_t t = labels[i];
    const float lse = lse_in[i];
    const float scale = __ldg(gscale) * inv_n;
    const bool ok = t >= 0 && t < C;  // a bad label was flagged by the forward: zero gradient
    uint16_t *grow = G + i * ldg;
#pragma unroll
    for (int v = 0; v < kMaxC / 8; ++v) {
        if (8 * v >= width) break;
        float x[8], g[8];
        if (8 * v < C) {
            if constexpr (PARK)
                unpack8(mine[v], x);
            else
                load8<VEC>(row, v, C, x);
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) x[q] = -INFINITY;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int j = 8 * v + q;
            g[q] = (ok && j < C) ? (expf(x[q] - lse) - (j == t ? 1.0f : 0.0f)) * scale : 0.0f;
        }
        if (VEC) {
            uint4 *dst = PARK ? mine + v : reinterpret_cast<uint4 *>(grow) + v;
            *dst = make_uint4(pack_bf16x2(g[0], g[1]), pack_bf16x2(g[2], g[3]),
                              pack_bf16x2(g[4], g[5]), pack_bf16x2(g[6], g[7]));
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (8 * v + q < width) grow[8 * v + q] = f32_to_bf16(g[q]);
        }
    }
    if (PARK) {
        __syncthreads();
        const int pieces = width / 8;
        for (int j = threadIdx.x; j < rows * pieces; j += kThreads) {
            const int r = j / pieces, p = j - r * pieces;
            *(reinterpret_cast<uint4 *>(G + (row0 + r) * ldg) + p) = parked[r * kPitch + p];
        }
    }
}

// Whole 8-score vectors can be loaded (and, with G, stored) for every row.
bool vec_rows(int C, long lds, const void *S, int width, long ldg, const void *G) {
    const int Cv = (C + 7) / 8 * 8;
    const bool s_ok = lds % 8 == 0 && lds >= Cv && reinterpret_cast<uintptr_t>(S) % 16 == 0;
    if (!G) return s_ok;
    return s_ok && width % 8 == 0 && ldg % 8 == 0 && reinterpret_cast<uintptr_t>(G) % 16 == 0;
}

// Whether the backward's rows go by way of shared memory, from 8 to 64 classes and up to 2.4M rows
// timed both ways: rows of 32 classes or more whose scores and gradients together are past what L2
// keeps (40 wide: 1M rows, 160 MB, 49 us and 53 parked, 2.4M rows 210 and 118; 48 wide: 400,000 rows
// 25 and 27, 1M rows, 192 MB, 84 and 63; 32 wide: 2.4M rows 110 and 95), and for rows of a whole
// line (over 56 classes) from 50 MB (64 wide: 200,000 rows 22.6 and 20.6, 400,000 rows 46 and 33).
// Narrower rows use their lines whole soon enough (2.4M rows: 24 wide 75 and 88, 16 wide 43 and 64).
bool park_rows(long n, int width, long lds, long ldg) {
    const long bytes = 2 * n * (lds + ldg);
    return width > 56 ? bytes > 50'000'000 : width >= 32 && bytes > 170'000'000;
}

}  // namespace

as_status xent_fwd_launch(as_ctx *ctx, int n, int C, const uint16_t *S, long lds,
                          const int64_t *labels, float *lse, float *loss, cudaStream_t s) {
    if (C < 1 || C > kMaxC) return fail(AS_ERR_UNSUPPORTED, "softmax xent: 1 <= C <= 64 classes");
    const int blocks = static_cast<int>(ceil_div(n, kThreads));
    void *w = nullptr;
    as_status st = scratch(ctx, sizeof(float) * static_cast<size_t>(blocks > 0 ? blocks : 1), &w);
    if (st != AS_OK) return st;
    float *partial = static_cast<float *>(w);
    if (blocks > 0) {
        if (vec_rows(C, lds, S, 0, 0, nullptr))
            xent_fwd<true><<<blocks, kThreads, 0, s>>>(n, C, S, lds, labels, lse, partial,
                                                       ctx->d_status);
        else
            xent_fwd<false><<<blocks, kThreads, 0, s>>>(n, C, S, lds, labels, lse, partial,
                                                        ctx->d_status);
        ctx->launches++;
    }
    xent_finish<<<1, kThreads, 0, s>>>(blocks, partial, n > 0 ? 1.0f / static_cast<float>(n) : 0.0f,
                                       loss);
    ctx->launches++;
    return check_cuda(cudaGetLastError(), "softmax xent launch");
}

as_status xent_bwd_launch(as_ctx *ctx, int n, int C, const uint16_t *S, long lds,
                          const int64_t *labels, const float *lse, const float *gscale,
                          uint16_t *G, long ldg, int width, cudaStream_t s) {
    if (C < 1 || C > kMaxC || width < C || width > kMaxC)
        return fail(AS_ERR_UNSUPPORTED, "softmax xent: 1 <= C <= width <= 64 classes");
    if (n == 0) return AS_OK;
    const unsigned blocks = static_cast<unsigned>(ceil_div(n, kThreads));
    const float inv_n = 1.0f / static_cast<float>(n);
    const auto kernel = !vec_rows(C, lds, S, width, ldg, G) ? xent_bwd<false, false>
                        : park_rows(n, width, lds, ldg)     ? xent_bwd<true, true>
                                                            : xent_bwd<true, false>;
    kernel<<<blocks, kThreads, 0, s>>>(n, C, S, lds, labels, lse, gscale, inv_n, G, ldg, width);
    ctx->launches++;
    return check_cuda(cudaGetLastError(), "softmax xent backward launch");
}

}  // namespace as
