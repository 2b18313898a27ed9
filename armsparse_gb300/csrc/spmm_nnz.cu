// CSR SpMM balanced by entries (sm_103a): C = A*B + beta*C for matrices whose row lengths are
// skewed (power-law graphs), where one long row would serialise a row-per-group kernel.
//
// Pass 1 (spmm_nnzsplit): the entries are cut into chunks of CH consecutive entries; a group
//   of GROUP lanes takes one chunk and one column tile, and walks its entries in CSR order in
//   steps of U, whatever rows they belong to: a batch of GROUP entries (one per lane), the ends
//   of the next GROUP rows (one per lane) and from them a mask of the batch's row-ending
//   entries are at hand before the batch starts, so the U rows of B of a step are loaded
//   together across row ends, and the next batch's entries and row ends are loaded meanwhile.
//   (Row by row, each row cost its pointer's, its entries' and its last 1-3 entries' memory
//   latencies in turn: 57,442 rows of mean 10 at width 48 took 64 us and take 44; 1M rows, 15M
//   entries, fp32 width 128: 1.04 and 0.92 ms.) Each row's segment is accumulated with fmaf like
//   the row-split kernels. A row that lies entirely inside the chunk is written to C directly
//   (bit-identical to rowBaseSpmm3, SDMM.cpp:90-114). A row that crosses a chunk boundary leaves
//   its segment's partial sum in a carry slot: slot 0 when the segment starts the chunk, slot 1
//   otherwise.
// Pass 2 (spmm_nnz_fixup): for every row that ends inside chunk c after starting in an earlier
//   chunk, chunk c's warp (a whole CTA for a long span) adds that row's partial sums (in chunk
//   order when the row spans at most 8 chunks, else runs of chunks and then the runs in order;
//   then beta * C): a fixed order, so the result is deterministic run to run (not
//   bit-identical to a single chain for those rows).
// Pass 3 (spmm_empty_rows): rows without entries get beta * C (zeros when beta == 0).
//
// Fused form (FUSE): pass 1 also computes, for every entry e (row r, column k), the dot product
// dA[perm[e]] = <B[k, :], F[r, :]> from the B row it has just loaded for the SpMM and F's row r
// (loaded once per row segment): the SDDMM that the backward of a product with trainable
// values needs, without a second gather of B. Each lane chains over its own
// columns of the row (its E-element slices j = 0..CPL-1, in order), then the GROUP lanes are
// summed by a butterfly (lane l adds lane l ^ off, off = GROUP/2 .. 1) -- for a step of U
// entries the butterflies of all U run interleaved (each lane hands half of its values to its
// partner at the first log2(U) steps), which pairs the same lanes in the same order, so each
// dot product is the single-entry butterfly's bit for bit. One column tile only (TILE >= N).
#include <limits.h>

#include "common.cuh"
#include "internal.h"
#include "spmm_vec.cuh"

namespace as {
namespace {

constexpr int kThreads = 256;

// A row segment's E sums at p, in whole vectors where the caller found them aligned.
template <int E>
__device__ __forceinline__ void store_f32(float *p, const float *v, bool vec) {
    if constexpr (E % 4 == 0) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < E; i += 4)
                *reinterpret_cast<float4 *>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            return;
        }
    }
#pragma unroll
    for (int i = 0; i < E; ++i) p[i] = v[i];
}

// Sum of each of the U values d[0..U) over the GROUP lanes of a group (U <= GROUP, both powers
// of two). While a lane holds more than one value, it keeps one half and sends the other to its
// partner lane ^ off; then plain butterfly steps. Lane g ends with the total of value
// g / (GROUP / U); the pairing tree is the single-value butterfly's.
template <int U, int GROUP>
__device__ __forceinline__ float reduce_entries(float (&d)[U], unsigned gmask, int g) {
    static_assert(U <= GROUP && (U & (U - 1)) == 0 && (GROUP & (GROUP - 1)) == 0, "shape");
#pragma unroll
    for (int h = U / 2, off = GROUP / 2; h >= 1; h >>= 1, off >>= 1) {
        const bool up = (g & off) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float send = up ? d[i] : d[i + h];
            const float keep = up ? d[i + h] : d[i];
            d[i] = keep + __shfl_xor_sync(gmask, send, off, GROUP);
        }
    }
#pragma unroll
    for (int off = GROUP / (2 * U); off >= 1; off >>= 1)
        d[0] += __shfl_xor_sync(gmask, d[0], off, GROUP);
    return d[0];
}

// dA[perm[e]] (dA[e] without perm) = v, skipping and flagging a position outside [0, nnz).
__device__ __forceinline__ void store_dot(int e, float v, int nnz, const int *__restrict__ perm,
                                          float *__restrict__ dA, unsigned *status) {
    const int p = perm ? __ldg(perm + e) : e;
    if (static_cast<unsigned>(p) < static_cast<unsigned>(nnz))
        dA[p] = v;
    else
        flag(status, kFlagBadPerm);
}

// The U dot products of a step (entries e0 .. e0 + U - 1) reduced over the group and stored
// at their CSR positions; an entry with an out-of-range column (kk < 0, already flagged) is
// left unwritten.
template <int U, int GROUP>
__device__ __forceinline__ void write_dots(float (&d)[U], const int (&kk)[U], unsigned gmask,
                                           int g, int e0, int nnz, const int *__restrict__ perm,
                                           float *__restrict__ dA, unsigned *status) {
    unsigned ok = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) ok |= (kk[u] >= 0 ? 1u : 0u) << u;
    const float sum = reduce_entries<U, GROUP>(d, gmask, g);
    constexpr int SUB = GROUP / U;
    const int u = g / SUB;
    if (g % SUB == 0 && ((ok >> u) & 1u)) store_dot(e0 + u, sum, nnz, perm, dA, status);
}

// kk * ldb_bytes on top of p: one wide multiply-add for rows of B under 4 GB, two
// more instructions past that.
__device__ __forceinline__ const char *row_at(const char *p, int kk, unsigned ldb_lo, unsigned ldb_hi) {
    unsigned long long a;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(a) : "r"(kk), "r"(ldb_lo),
        "l"(reinterpret_cast<unsigned long long>(p)));
    if (ldb_hi) a += static_cast<unsigned long long>(static_cast<unsigned>(kk) * ldb_hi) << 32;
    return reinterpret_cast<const char *>(a);
}

// A value as it travels between lanes, and as the step takes it.
__device__ __forceinline__ float lane_val(float v) { return v; }
__device__ __forceinline__ unsigned lane_val(uint16_t v) { return v; }

// CTAs per SM to leave registers for. The gathers live on warps in flight, and a spill or a step
// that waits for registers costs more than a CTA gives, so the line is measured per kind of kernel,
// 2 to 6 CTAs each on four matrices (uniform rows of 3 and of 20, power-law rows of 4.2M and 16.8M
// entries, widths 16 to 256); geometric means of the time against that of the row-by-row walk:
// - four (64 registers) wherever a step's loads and the running sums are at most 24 registers: fp32
//   float4 0.78 with four, 0.84 with three, 0.86 with five; fused bf16 of 256 columns 0.93 with four
//   in spite of 88 bytes spilled, 1.10 with two, 1.02 with five;
// - three (80 registers) where a lane holds two vectors and a step takes eight entries of narrow
//   ones (0.68-0.71; 0.76-0.78 with four, which spilled 128-156 bytes; 0.76-0.80 with two), and for
//   the fused fp32 float4 x 2 (0.75; 0.78 with two, 0.85 with four);
// - else two: fp32 float4 x 2 0.81 (three 0.81, and a fifth slower on the smaller power-law matrix),
//   bf16 of 512 columns 0.81 (three 0.81, four 0.99), eight entries of bf16 x 8 0.61 (three 0.65).
// Uniform rows of 20 lose by the walk in some kernels whatever the count: scalar lanes x 2 in fp32
// up to 1.28 (mean 0.90), eight entries of float4 by sixteens up to 1.24 (mean 0.73).
template <int VB, int CPL, int U, int E, bool FUSE>
constexpr int ctas_per_sm() {
    constexpr int regs = U * CPL * VB / 4 + CPL * E;
    if (CPL == 2 && (U == 8 ? regs <= 24 : FUSE && regs > 24 && regs <= 40)) return 3;
    return regs <= 24 ? 4 : 2;
}

template <typename T, int VB, int GROUP, int CPL, int U, bool FUSE>
__global__ void __launch_bounds__(kThreads, ctas_per_sm<VB, CPL, U, Vec<T, VB>::E, FUSE>())
spmm_nnzsplit(int M, int K, int N, int nnz, int CH, const int *__restrict__ rowptr,
              const int *__restrict__ colind, const T *__restrict__ val,
              const T *__restrict__ B, long ldb, float *__restrict__ C, long ldc, float beta,
              float *__restrict__ carry, int *__restrict__ fix, unsigned *status,
              const T *__restrict__ F, long ldf, const int *__restrict__ perm,
              float *__restrict__ dA, uint16_t *__restrict__ C16, bool relu, bool c_vec,
              bool carry_vec) {
    using V = Vec<T, VB>;
    constexpr int E = V::E;
    constexpr int TILE = GROUP * E * CPL;
    static_assert(GROUP % U == 0, "a batch is whole steps");
    const int lane = threadIdx.x & 31;
    const int g = threadIdx.x % GROUP;
    const unsigned gmask =
        GROUP == 32 ? 0xffffffffu : (((1u << GROUP) - 1u) << (lane & ~(GROUP - 1)));
    const long chunk = static_cast<long>(blockIdx.x) * (kThreads / GROUP) + threadIdx.x / GROUP;
    const long e0l = chunk * CH;
    if (e0l >= nnz) return;
    const int e0 = static_cast<int>(e0l);
    // entries past the last row's end (a row pointer that stops short of nnz) belong to no row
    const int e1 = static_cast<int>(max(
        0L, min(min(e0l + CH, static_cast<long>(nnz)), static_cast<long>(__ldg(rowptr + M)))));
    const int tile0 = blockIdx.y * TILE;
    auto count = [&](bool p) { return __popc(__ballot_sync(gmask, p) & gmask); };
    const char *bcol[CPL];  // this lane's columns of row 0 of B (column 0 for a lane past N)
#pragma unroll
    for (int j = 0; j < CPL; ++j) {
        const int cc = tile0 + (j * GROUP + g) * E;
        bcol[j] = reinterpret_cast<const char *>(B + (cc < N ? cc : 0));
    }
    const unsigned long long ldb_bytes = static_cast<unsigned long long>(ldb) * sizeof(T);
    const unsigned ldb_lo = static_cast<unsigned>(ldb_bytes);
    const unsigned ldb_hi = static_cast<unsigned>(ldb_bytes >> 32);

    int fix_row = -1;  // the row that started in an earlier chunk and ends in this one
    int r0 = e0 < e1 ? find_row<GROUP>(rowptr, M, e0, g, gmask) : 0;
    const int rs0 = __ldg(rowptr + r0);
    // the window of row ends: rows r, r + 1, ... (one per lane)
    auto ends = [&](int r) {
        const long i = static_cast<long>(r) + 1 + g;
        return i <= M ? __ldg(rowptr + i) : INT_MAX;
    };
    // a window that may be used: never falling, its first past entry e
    auto sound = [&](int w, int e) {
        const int below = __shfl_up_sync(gmask, w, 1, GROUP);
        return count(g > 0 ? w < below : w <= e) == 0;
    };
    using Val = decltype(lane_val(T()));
    // (unsigned: an entry ahead of 2^31 - 1 of them is past e1, not below zero)
    auto load_entry = [&](unsigned e, int &k, Val &v) {
        k = -1;
        v = 0;
        if (e < static_cast<unsigned>(e1)) {
            k = ld_stream(colind + e);
            v = lane_val(ld_stream(val + e));
        }
    };
    int re = ends(r0), k, base = e0;
    Val v;
    load_entry(static_cast<unsigned>(base) + g, k, v);
    bool good = e0 < e1 && rs0 >= 0 && rs0 <= e0 && sound(re, e0);
    if (e0 < e1 && !good) flag(status, kFlagBadRowptr);
    int row = r0;                      // the row that the running sums belong to
    int seg = e0;                      // its first entry in this chunk
    const bool head_split = rs0 < e0;  // the chunk's first row started in an earlier chunk
    float acc[CPL][E];
    auto start_row = [&]() {
#pragma unroll
        for (int j = 0; j < CPL; ++j)
#pragma unroll
            for (int i = 0; i < E; ++i) acc[j][i] = 0.0f;
        if (beta != 0.0f && row < M && __ldg(rowptr + row + 1) <= e1 && !(head_split && seg == e0)) {
#pragma unroll
            for (int j = 0; j < CPL; ++j) {
                const int cc = tile0 + (j * GROUP + g) * E;
#pragma unroll
                for (int i = 0; i < E; ++i)
                    if (cc < N) acc[j][i] = beta * C[row * ldc + cc + i];
            }
        }
    };
    // the running sums to C, or (a row that goes on in another chunk) to a carry slot
    auto store_row = [&](bool split) {
        float *dst = split ? carry + (2 * chunk + (seg == e0 ? 0 : 1)) * static_cast<long>(N)
                           : C + row * ldc;
        const bool vec = split ? carry_vec : c_vec;
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
            const int cc = tile0 + (j * GROUP + g) * E;
            if (cc < N) {
                if (!split && C16)
                    store_bf16<E>(C16 + row * ldc + cc, acc[j], relu);
                else
                    store_f32<E>(dst + cc, acc[j], vec);
            }
        }
    };
    start_row();
    // FUSE: the slices of F of the running row
    typename V::Raw fr[CPL];
    auto start_f = [&]() {
        if (row >= M) return;
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
            const int cc = tile0 + (j * GROUP + g) * E;
            fr[j] = V::raw(F + static_cast<long>(row) * ldf + (cc < N ? cc : 0));
        }
    };
    if constexpr (FUSE) start_f();

    while (base < e1 && good) {
        // This batch: entries base .. base + cnt - 1, cut where the window of row ends stops
        // short of it (runs of empty rows).
        const int last = __shfl_sync(gmask, re, GROUP - 1, GROUP);
        const int cnt = min(min(GROUP, e1 - base), last - base);
        const int next = base + cnt;
        // bit i: entry base + i is its row's last
        unsigned endm = re > base && re <= next ? 1u << (re - base - 1) : 0u;
#pragma unroll
        for (int off = GROUP / 2; off >= 1; off >>= 1)
            endm |= __shfl_xor_sync(gmask, endm, off, GROUP);
        // the next batch's entries and window, in flight meanwhile
        int kn, rn = r0 + count(re <= next), ren = ends(rn);
        Val vn;
        load_entry(static_cast<unsigned>(next) + g, kn, vn);
        if (g >= cnt) {
            k = -1;
        } else if (static_cast<unsigned>(k) >= static_cast<unsigned>(K)) {
            flag(status, kFlagBadColind);
            k = -1;
        }
        const bool clean = count(k >= 0) == GROUP;
#pragma unroll 1
        for (int t = 0; t < cnt; t += U) {
            int kk[U];
            Val vv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                kk[u] = __shfl_sync(gmask, k, t + u, GROUP);
                vv[u] = __shfl_sync(gmask, v, t + u, GROUP);
            }
            const unsigned em = endm >> t & ((1u << U) - 1u);
            // U entries' rows of B before any is used (a skipped entry reads row 0)
            typename V::Raw b[U][CPL];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int j = 0; j < CPL; ++j)
                    b[u][j] = V::raw(reinterpret_cast<const T *>(
                        row_at(bcol[j], max(kk[u], 0), ldb_lo, ldb_hi)));
            float d[U];
            auto apply = [&](int u) {
                d[u] = 0.0f;
#pragma unroll
                for (int j = 0; j < CPL; ++j) {
                    const bool in = tile0 + (j * GROUP + g) * E < N;
                    if constexpr (sizeof(T) == 4) {
                        float bf[E];
#pragma unroll
                        for (int i = 0; i < E; ++i) bf[i] = V::at(b[u][j], i);
                        fma_vec_f32<E>(bf, vv[u], acc[j]);
                        if constexpr (FUSE) {
                            float s = d[u];
#pragma unroll
                            for (int i = 0; i < E; ++i) s = fmaf(bf[i], V::at(fr[j], i), s);
                            if (in) d[u] = s;
                        }
                    } else {
                        V::fma(b[u][j], static_cast<unsigned short>(vv[u]), acc[j]);
                        if constexpr (FUSE) {
                            float s = d[u];
                            V::dot(b[u][j], fr[j], s);
                            if (in) d[u] = s;
                        }
                    }
                }
            };
            if (GROUP == 32 && clean && em == 0) {
#pragma unroll
                for (int u = 0; u < U; ++u) apply(u);
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    d[u] = 0.0f;
                    if (kk[u] >= 0) apply(u);
                    if (em >> u & 1u) {  // the row ends here
                        const bool split = head_split && seg == e0;
                        store_row(split);
                        if (split) fix_row = row;
                        seg = base + t + u + 1;
                        row = r0 + count(re <= seg);
                        start_row();
                        if constexpr (FUSE) start_f();
                    }
                }
            }
            if constexpr (FUSE) write_dots<U, GROUP>(d, kk, gmask, g, base + t, nnz, perm, dA, status);
        }
        // on to the next batch; where the window's rows all ended, look for the next row that
        // holds an entry
        if (next < e1) {
            if (rn == r0 + GROUP) {
                int empty = count(ren <= next);
                while (empty == GROUP) {
                    rn += GROUP;
                    ren = ends(rn);
                    empty = count(ren <= next);
                }
                if (empty) {
                    rn += empty;
                    ren = ends(rn);
                }
            }
            if (!sound(ren, next)) {
                flag(status, kFlagBadRowptr);
                good = false;
            }
            if (row != rn) {  // the row after a run of empty ones
                row = rn;
                start_row();
                if constexpr (FUSE) start_f();
            }
        }
        r0 = rn;
        re = ren;
        k = kn;
        v = vn;
        base = next;
    }
    if (good && seg < e1 && row < M) store_row(true);  // the last row goes on in the next chunk
    if (blockIdx.y == 0 && g == 0) fix[chunk] = fix_row;
}

// Multi-entry form, for narrow rows of B (GROUP * E < 32 lanes' worth): a warp takes a chunk,
// and its S = 32 / GROUP sub-groups of GROUP lanes take every S-th entry of each row segment
// (sub-group s: entries s, s + S, s + 2S, ... of each 32-entry block), so one load
// instruction brings S entries' rows and the broadcasts, addresses and loop control are shared
// by S entries. A sub-group chains its entries in CSR order; at the segment's end the S partial
// sums are added by a butterfly over the sub-groups (lane l adds lane l ^ off, off = GROUP ..
// 16), then beta * C. Deterministic, but not the single CSR chain of the other kernels. Carry
// slots, fix-up and empty rows as in spmm_nnzsplit; FUSE as there (each dot product over one
// sub-group's GROUP lanes), with one column tile.
template <int U, int GROUP>
__device__ __forceinline__ void write_dots_me(float (&d)[U], const int (&kk)[U], unsigned gmask,
                                              int g, int e0, int stride, int nnz,
                                              const int *__restrict__ perm, float *__restrict__ dA,
                                              unsigned *status) {
    unsigned ok = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) ok |= (kk[u] >= 0 ? 1u : 0u) << u;
    const float sum = reduce_entries<U, GROUP>(d, gmask, g);
    constexpr int SUB = GROUP / U;
    const int u = g / SUB;
    if (g % SUB == 0 && ((ok >> u) & 1u)) store_dot(e0 + stride * u, sum, nnz, perm, dA, status);
}

template <typename T, int VB, int GROUP, int U, bool FUSE>
__global__ void __launch_bounds__(kThreads)
spmm_nnzme(int M, int K, int N, int nnz, int CH, const int *__restrict__ rowptr,
           const int *__restrict__ colind, const T *__restrict__ val, const T *__restrict__ B,
           long ldb, float *__restrict__ C, long ldc, float beta, float *__restrict__ carry,
           int *__restrict__ fix, unsigned *status, const T *__restrict__ F, long ldf,
           const int *__restrict__ perm, float *__restrict__ dA, uint16_t *__restrict__ C16,
           bool relu) {
    using V = Vec<T, VB>;
    constexpr int E = V::E;
    constexpr int S = 32 / GROUP;
    constexpr int TILE = GROUP * E;
    static_assert(S >= 1 && U <= GROUP, "shape");
    const int lane = threadIdx.x & 31;
    const int g = lane % GROUP, sg = lane / GROUP;
    const unsigned gmask =
        GROUP == 32 ? 0xffffffffu : (((1u << GROUP) - 1u) << (lane & ~(GROUP - 1)));
    const long chunk = static_cast<long>(blockIdx.x) * (kThreads / 32) + threadIdx.x / 32;
    const long e0l = chunk * CH;
    if (e0l >= nnz) return;  // the whole warp leaves together
    const int e0 = static_cast<int>(e0l);
    const int e1 = static_cast<int>(e0l + CH < nnz ? e0l + CH : nnz);
    const int cc = blockIdx.y * TILE + g * E;  // this lane's columns
    const bool col_ok = cc < N;
    int r = find_row<32>(rowptr, M, e0, lane, 0xffffffffu);
    int e = e0;
    int fix_row = -1;
    while (e < e1 && r < M) {  // uniform across the warp
        const int rs = __ldg(rowptr + r), re = __ldg(rowptr + r + 1);
        if (re <= e || rs > e) {
            if (rs > e || re < rs) {
                flag(status, kFlagBadRowptr);
                break;
            }
            ++r;
            continue;
        }
        const int se = re < e1 ? re : e1;
        const bool split = rs < e0 || re > e1;
        if (rs < e0 && re <= e1) fix_row = r;
        typename V::Raw fr;  // FUSE: this row's slice of F
        if constexpr (FUSE) fr = V::raw(F + static_cast<long>(r) * ldf + (col_ok ? cc : 0));
        float acc[E];
#pragma unroll
        for (int i = 0; i < E; ++i) acc[i] = 0.0f;
        const unsigned last = static_cast<unsigned>(se);  // unsigned: entries ahead of it stay above
        for (unsigned base = e; base < last; base += 32) {
            const unsigned ee = base + lane;
            int k = -1;
            float v = 0.0f;
            if (ee < last) {
                k = ld_stream(colind + ee);
                v = to_f32(ld_stream(val + ee));
                if (static_cast<unsigned>(k) >= static_cast<unsigned>(K)) {
                    flag(status, kFlagBadColind);
                    k = -1;
                }
            }
            const int cnt = static_cast<int>(min(32u, last - base));
            for (int t = 0; t < cnt; t += S * U) {  // sub-group sg: entries t + sg + S*u
                int kk[U];
                float vv[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = t + sg + S * u;
                    kk[u] = __shfl_sync(0xffffffffu, k, j & 31);
                    vv[u] = __shfl_sync(0xffffffffu, v, j & 31);
                    if (j >= cnt) kk[u] = -1;
                }
                if constexpr (sizeof(T) == 4) {
                    float b[U][E];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (col_ok && kk[u] >= 0) {
                            V::load(B + static_cast<long>(kk[u]) * ldb + cc, b[u]);
                        } else {
#pragma unroll
                            for (int i = 0; i < E; ++i) b[u][i] = 0.0f;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (kk[u] >= 0) fma_vec_f32<E>(b[u], vv[u], acc);
                    if constexpr (FUSE) {
                        float d[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            d[u] = 0.0f;
                            if (col_ok)
#pragma unroll
                                for (int i = 0; i < E; ++i) d[u] = fmaf(b[u][i], V::at(fr, i), d[u]);
                        }
                        write_dots_me<U, GROUP>(d, kk, gmask, g, static_cast<int>(base) + t + sg, S, nnz, perm, dA,
                                                status);
                    }
                } else {
                    typename V::Raw b[U];
#pragma unroll
                    for (int u = 0; u < U; ++u)  // branch-free: a skipped entry reads row 0
                        b[u] = V::raw(B + static_cast<long>(kk[u] < 0 ? 0 : kk[u]) * ldb +
                                      (col_ok ? cc : 0));
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (kk[u] < 0) continue;
                        const unsigned short vu =
                            static_cast<unsigned short>(__float_as_uint(vv[u]) >> 16);
                        V::fma(b[u], vu, acc);
                    }
                    if constexpr (FUSE) {
                        float d[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            d[u] = 0.0f;
                            if (col_ok) V::dot(b[u], fr, d[u]);
                        }
                        write_dots_me<U, GROUP>(d, kk, gmask, g, static_cast<int>(base) + t + sg, S, nnz, perm, dA,
                                                status);
                    }
                }
            }
        }
#pragma unroll
        for (int off = GROUP; off < 32; off <<= 1)  // the sub-groups' partial sums
#pragma unroll
            for (int i = 0; i < E; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
        if (sg == 0 && col_ok) {
            if (split) {
                float *dst = carry + (2 * chunk + (e == e0 ? 0 : 1)) * static_cast<long>(N) + cc;
#pragma unroll
                for (int i = 0; i < E; ++i) dst[i] = acc[i];
            } else if (C16) {
                store_bf16<E>(C16 + r * ldc + cc, acc, relu);
            } else {
                float *dst = C + r * ldc + cc;
#pragma unroll
                for (int i = 0; i < E; ++i) dst[i] = beta != 0.0f ? fmaf(beta, dst[i], acc[i]) : acc[i];
            }
        }
        e = se;
        ++r;
    }
    if (blockIdx.y == 0 && lane == 0) fix[chunk] = fix_row;
}

constexpr int kShortSpan = 8;  // rows over at most this many chunks: the one-pass fix-up
constexpr int kFixBatch = 8;  // partial loads in flight per thread on a long span (16 measured slower)

template <int VW>
struct Lanes;  // VW consecutive fp32 columns of a carry row, one load
template <>
struct Lanes<4> {
    __device__ static void load(const float *p, float *v) {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
};
template <>
struct Lanes<1> {
    __device__ static void load(const float *p, float *v) { v[0] = *p; }
};

// Rows that end in chunk c after starting in an earlier chunk: sum their partials. A CTA takes
// kFixChunks consecutive chunks, one per warp.
//  - A row over at most kShortSpan chunks (nearly all of them): the chunk's warp alone, each
//    lane VW columns at a time, the chunks' partials loaded together and added in chunk order.
//  - A longer row, afterwards with the whole CTA: the threads split into R consecutive runs of
//    the row's chunks times groups of VW columns (R = threads / column groups, so all threads
//    load at once); each sums its run in chunk order, kFixBatch loads in flight, and the runs
//    are then added in run order.
// Both orders are fixed by the row's span and N, so the result is deterministic. (One row of a
// power-law graph can span thousands of chunks: that CTA is the fix-up's critical path. One
// CTA per chunk made the many short fix-ups cost more in CTA launches than in loads.)
constexpr int kFixChunks = kThreads / 32;

template <int VW>
__device__ __forceinline__ void store_out(float *C, uint16_t *C16, long off, float beta, float v,
                                          bool relu) {
    if (C16)
        C16[off] = f32_to_bf16(relu_if(v, relu));
    else
        C[off] = beta == 0.0f ? v : fmaf(beta, C[off], v);
}

template <int VW>
__global__ void __launch_bounds__(kThreads)
spmm_nnz_fixup(int M, int N, long nchunks, int CH, const int *__restrict__ rowptr,
               const float *__restrict__ carry, const int *__restrict__ fix,
               float *__restrict__ C, long ldc, float beta, uint16_t *__restrict__ C16,
               bool relu) {
    __shared__ float part[kThreads * VW];
    __shared__ int long_rows[kFixChunks];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the chunk's row to fix (-1: none) and its span
    auto span = [&](long chunk, int &r, int &rs, long &c_first, long &n) {
        r = chunk < nchunks ? fix[chunk] : -1;  // recorded by the first pass
        if (r < 0 || r >= M) {
            r = -1;
            return;
        }
        rs = __ldg(rowptr + r);
        c_first = rs / CH;
        n = chunk - c_first + 1;
    };
    // slot 1 holds the first chunk's partial when the row starts inside that chunk
    auto row_of = [&](long cc, long c_first, int rs) {
        return (2 * cc + ((cc == c_first && static_cast<long>(rs) != cc * CH) ? 1 : 0)) *
               static_cast<long>(N);
    };
    {
        int r, rs = 0;
        long c_first = 0, n = 0;
        span(static_cast<long>(blockIdx.x) * kFixChunks + warp, r, rs, c_first, n);
        if (lane == 0) long_rows[warp] = r >= 0 && n > kShortSpan;
        if (r >= 0 && n <= kShortSpan) {
            for (int col = lane * VW; col < N; col += 32 * VW) {
                float v[kShortSpan][VW];
#pragma unroll
                for (int i = 0; i < kShortSpan; ++i) {
                    if (i < n) {
                        Lanes<VW>::load(carry + row_of(c_first + i, c_first, rs) + col, v[i]);
                    } else {
#pragma unroll
                        for (int j = 0; j < VW; ++j) v[i][j] = 0.0f;
                    }
                }
#pragma unroll
                for (int j = 0; j < VW; ++j) {
                    float acc = v[0][j];
#pragma unroll
                    for (int i = 1; i < kShortSpan; ++i)
                        if (i < n) acc += v[i][j];
                    store_out<VW>(C, C16, r * ldc + col + j, beta, acc, relu);
                }
            }
        }
    }
    __syncthreads();
    for (int w = 0; w < kFixChunks; ++w) {
        if (!long_rows[w]) continue;  // shared: the same for the whole CTA
        int r, rs = 0;
        long c_first = 0, n = 0;
        span(static_cast<long>(blockIdx.x) * kFixChunks + w, r, rs, c_first, n);
        const int ncg = N / VW;  // column groups (the launcher guarantees N % VW == 0)
        for (int cg0 = 0; cg0 < ncg; cg0 += kThreads) {
            const int cgs = min(kThreads, ncg - cg0);
            const int R = kThreads / cgs;
            const int run = threadIdx.x / cgs, gi = threadIdx.x % cgs;
            const int col = (cg0 + gi) * VW;
            float acc[VW];
#pragma unroll
            for (int j = 0; j < VW; ++j) acc[j] = 0.0f;
            if (run < R) {
                const long b0 = c_first + n * run / R, b1 = c_first + n * (run + 1) / R;
                for (long cc = b0; cc < b1; cc += kFixBatch) {
                    float v[kFixBatch][VW];
#pragma unroll
                    for (int i = 0; i < kFixBatch; ++i) {
                        if (cc + i < b1) {
                            Lanes<VW>::load(carry + row_of(cc + i, c_first, rs) + col, v[i]);
                        } else {
#pragma unroll
                            for (int j = 0; j < VW; ++j) v[i][j] = 0.0f;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < kFixBatch; ++i)
                        if (cc + i < b1)
#pragma unroll
                            for (int j = 0; j < VW; ++j) acc[j] += v[i][j];
                }
#pragma unroll
                for (int j = 0; j < VW; ++j) part[(run * cgs + gi) * VW + j] = acc[j];
            }
            __syncthreads();
            if (run == 0) {
#pragma unroll
                for (int j = 0; j < VW; ++j) {
                    float t = part[gi * VW + j];
                    for (int q = 1; q < R; ++q) t += part[(q * cgs + gi) * VW + j];
                    store_out<VW>(C, C16, r * ldc + col + j, beta, t, relu);
                }
            }
            __syncthreads();  // part[] is reused by the next column block or row
        }
    }
}

// Rows without entries get beta * C. A warp checks 32 consecutive rows with one load each and
// writes only the empty ones, 32 columns at a time.
__global__ void __launch_bounds__(kThreads)
spmm_empty_rows(int M, int N, const int *__restrict__ rowptr, float *__restrict__ C, long ldc,
                float beta, uint16_t *__restrict__ C16) {
    const long base = (static_cast<long>(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5)) * 32;
    const int lane = threadIdx.x & 31;
    if (base >= M) return;  // the same for the whole warp
    const long r = base + lane;
    const bool empty = r < M && __ldg(rowptr + r) == __ldg(rowptr + r + 1);
    for (unsigned m = __ballot_sync(0xffffffffu, empty); m; m &= m - 1) {
        const long rr = base + (__ffs(m) - 1);
        for (int col = lane; col < N; col += 32) {
            if (C16)
                C16[rr * ldc + col] = 0;
            else
                C[rr * ldc + col] = beta == 0.0f ? 0.0f : beta * C[rr * ldc + col];
        }
    }
}

size_t carry_size(long nchunks, int N) {
    return (sizeof(float) * static_cast<size_t>(2 * nchunks) * N + 255) & ~size_t(255);
}

// ME: the multi-entry kernel (spmm_nnzme, CPL 1); else spmm_nnzsplit.
template <typename T, int VB, int G, int CPL, int U, bool FUSE, bool ME = false>
as_status launch(as_ctx *ctx, const SpmmArgs &a, int CH, const SddmmFuse *fu, cudaStream_t s) {
    static_assert(!ME || CPL == 1, "multi-entry kernels hold one vector per lane");
    constexpr int E = Vec<T, VB>::E;
    constexpr int TILE = G * E * CPL;
    const int esz = sizeof(T);
    if ((a.N % E) || (a.ldb % E) || (reinterpret_cast<uintptr_t>(a.B) % (E * esz)))
        return fail(AS_ERR_UNSUPPORTED, "spmm nnz-split: layout does not fit the vector width");
    if (ceil_div(a.N, TILE) > 65535 || ceil_div(a.N, 32) > 65535)
        return fail(AS_ERR_UNSUPPORTED, "spmm nnz-split: N too large");
    if (a.C16 && (a.beta != 0.0f || (a.ldc % E) ||
                  (reinterpret_cast<uintptr_t>(a.C16) % (2 * E > 16 ? 16 : 2 * E))))
        return fail(AS_ERR_UNSUPPORTED,
                    "spmm nnz-split: bf16 output needs beta = 0 and C aligned to the vectors");
    if (FUSE && (a.N > TILE || (fu->ldf % E) || (reinterpret_cast<uintptr_t>(fu->F) % (E * esz))))
        return fail(AS_ERR_UNSUPPORTED,
                    "spmm+sddmm: the variant's column tile must cover N, F aligned to its vectors");
    const long nchunks = ceil_div(a.nnz, CH);
    void *w = nullptr;
    const size_t carry_bytes = carry_size(nchunks, a.N);
    as_status st = scratch(ctx, spmm_nnz_scratch(a.nnz, a.N, CH), &w);
    if (st != AS_OK) return st;
    float *carry = static_cast<float *>(w);
    int *fix = reinterpret_cast<int *>(static_cast<char *>(w) + carry_bytes);
    if (nchunks > 0) {
        if constexpr (ME) {
            dim3 g1(static_cast<unsigned>(ceil_div(nchunks, kThreads / 32)),
                    static_cast<unsigned>(ceil_div(a.N, TILE)));
            spmm_nnzme<T, VB, G, U, FUSE><<<g1, kThreads, 0, s>>>(
                a.M, a.K, a.N, a.nnz, CH, a.rowptr, a.colind, static_cast<const T *>(a.val),
                static_cast<const T *>(a.B), a.ldb, a.C, a.ldc, a.beta, carry, fix, a.status,
                FUSE ? static_cast<const T *>(fu->F) : nullptr, FUSE ? fu->ldf : 0,
                FUSE ? fu->perm : nullptr, FUSE ? fu->dA : nullptr, a.C16, a.relu);
        } else {
            const bool c_vec = a.ldc % 4 == 0 && reinterpret_cast<uintptr_t>(a.C) % 16 == 0;
            dim3 g1(static_cast<unsigned>(ceil_div(nchunks, kThreads / G)),
                    static_cast<unsigned>(ceil_div(a.N, TILE)));
            spmm_nnzsplit<T, VB, G, CPL, U, FUSE><<<g1, kThreads, 0, s>>>(
                a.M, a.K, a.N, a.nnz, CH, a.rowptr, a.colind, static_cast<const T *>(a.val),
                static_cast<const T *>(a.B), a.ldb, a.C, a.ldc, a.beta, carry, fix, a.status,
                FUSE ? static_cast<const T *>(fu->F) : nullptr, FUSE ? fu->ldf : 0,
                FUSE ? fu->perm : nullptr, FUSE ? fu->dA : nullptr, a.C16, a.relu, c_vec,
                a.N % 4 == 0);
        }
        dim3 g2(static_cast<unsigned>(ceil_div(nchunks, kFixChunks)));
        if (a.N % 4 == 0)  // carry rows are 16-byte aligned: whole-vector loads
            spmm_nnz_fixup<4><<<g2, kThreads, 0, s>>>(a.M, a.N, nchunks, CH, a.rowptr, carry, fix,
                                                      a.C, a.ldc, a.beta, a.C16, a.relu);
        else
            spmm_nnz_fixup<1><<<g2, kThreads, 0, s>>>(a.M, a.N, nchunks, CH, a.rowptr, carry, fix,
                                                      a.C, a.ldc, a.beta, a.C16, a.relu);
        ctx->launches += 2;
    }
    spmm_empty_rows<<<static_cast<unsigned>(ceil_div(a.M, kThreads)), kThreads, 0, s>>>(
        a.M, a.N, a.rowptr, a.C, a.ldc, a.beta, a.C16);
    ctx->launches++;
    return check_cuda(cudaGetLastError(), "spmm nnz-split launch");
}

template <typename T, int VB, int G, int CPL>
as_status launch_u(as_ctx *ctx, const SpmmArgs &a, int CH, int unroll, const SddmmFuse *fu,
                   cudaStream_t s) {
    // fused: four entries per step whatever the variant (the sums do not depend on the step)
    if (fu) return launch<T, VB, G, CPL, 4, true>(ctx, a, CH, fu, s);
    return unroll == 8 ? launch<T, VB, G, CPL, 8, false>(ctx, a, CH, fu, s)
                       : launch<T, VB, G, CPL, 4, false>(ctx, a, CH, fu, s);
}

template <typename T, int VB, int G>
as_status launch_me(as_ctx *ctx, const SpmmArgs &a, int CH, const SddmmFuse *fu, cudaStream_t s) {
    return fu ? launch<T, VB, G, 1, 4, true, true>(ctx, a, CH, fu, s)
              : launch<T, VB, G, 1, 4, false, true>(ctx, a, CH, fu, s);
}

}  // namespace

size_t spmm_nnz_scratch(int nnz, int N, int chunk) {
    const long nchunks = ceil_div(nnz, chunk);
    return carry_size(nchunks, N) + sizeof(int) * static_cast<size_t>(nchunks);
}

as_status spmm_nnzme_launch(as_ctx *ctx, int dtype, int vb, int group, int chunk,
                            const SpmmArgs &a, cudaStream_t s, const SddmmFuse *fuse) {
#define AS_ME_CASE(T, VBV, G) \
    if (vb == VBV && group == G) return launch_me<T, VBV, G>(ctx, a, chunk, fuse, s);
    if (dtype == 0) {
        AS_ME_CASE(float, 16, 8) AS_ME_CASE(float, 16, 16) AS_ME_CASE(float, 8, 8)
        AS_ME_CASE(float, 8, 16)
    } else {
        AS_ME_CASE(uint16_t, 16, 8) AS_ME_CASE(uint16_t, 16, 16) AS_ME_CASE(uint16_t, 8, 8)
        AS_ME_CASE(uint16_t, 8, 16)
    }
#undef AS_ME_CASE
    return fail(AS_ERR_UNSUPPORTED, "spmm multi-entry: configuration not instantiated");
}

as_status spmm_nnz_launch(as_ctx *ctx, int dtype, int vb, int group, int cpl, int chunk,
                          int unroll, const SpmmArgs &a, cudaStream_t s, const SddmmFuse *fuse) {
#define AS_NNZ_CASE(T, VBV, G, C)            \
    if (vb == VBV && group == G && cpl == C) \
        return launch_u<T, VBV, G, C>(ctx, a, chunk, unroll, fuse, s);
    if (dtype == 0) {
        AS_NNZ_CASE(float, 16, 8, 1) AS_NNZ_CASE(float, 16, 16, 1) AS_NNZ_CASE(float, 16, 32, 1)
        AS_NNZ_CASE(float, 16, 32, 2) AS_NNZ_CASE(float, 4, 32, 1) AS_NNZ_CASE(float, 4, 32, 2)
    } else {
        AS_NNZ_CASE(uint16_t, 16, 8, 1) AS_NNZ_CASE(uint16_t, 16, 16, 1)
        AS_NNZ_CASE(uint16_t, 16, 32, 1) AS_NNZ_CASE(uint16_t, 16, 32, 2)
        AS_NNZ_CASE(uint16_t, 4, 32, 1) AS_NNZ_CASE(uint16_t, 4, 32, 2)
        AS_NNZ_CASE(uint16_t, 2, 32, 1) AS_NNZ_CASE(uint16_t, 2, 32, 2)
    }
#undef AS_NNZ_CASE
    return fail(AS_ERR_UNSUPPORTED, "spmm nnz-split: configuration not instantiated");
}

}  // namespace as
