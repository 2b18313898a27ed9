// Long rows of the row-split SpMM (sm_103a), bit-identical to rowBaseSpmm3 (SDMM.cpp:90-114).
//
// A row-split group walks its row's entries one after another, so one row with 10^5 entries
// (a hub of a power-law graph) keeps a single group busy long after the rest of the grid has
// finished. The row-split kernels therefore leave every row longer than a threshold to this
// kernel: they append the row number to a list (one atomic per long row) and skip it; this
// kernel, launched right after on the same stream, takes the listed rows. Rows longer than
// kHugeRow entries are listed from the other end of the list and taken first, so the longest
// chains start at once instead of behind shorter rows.
//
// The same kernel takes the long rows of the other row-oriented SpMMs, with their own chain
// step (OP below): the reduce aggregations (spmm_reduce.cu), the 1x4-blocked layout
// (spmm_vcsr4.cu) and the row-pair layout (spmm_rowpair.cu: a listed pair gives a unit per
// row, whose chain runs over the entries that the unit includes).
//
// Each output element is still one chain over the row's entries in CSR order (the order
// cannot be split without changing the bits): the floor of a row is its length times the
// latency of one fused multiply-add (4 cycles), and the kernel's work is to keep that chain
// fed. A unit is a (long row, column slice); a slice is 32 words of a row of B (32 fp32 or 64
// bf16 columns). A CTA walks its units as one stream of blocks of kBlk entries, without a
// barrier between units; its warps split by role:
//  - warp 0 is the consumer: lane l runs the chains of its one (fp32) or two (bf16) columns out
//    of shared memory. A slot holds the block transposed by fours: the words of four
//    consecutive entries of one lane lie together, so one 16-byte read brings four entries and
//    the chain is not held up by the rate at which one warp issues shared-memory reads (32-bit
//    reads: 5.8 cycles per entry; 128-bit reads: 4.5). The 16 entries after the ones whose
//    steps run are always being read meanwhile, also across the end of a block, and the next
//    block's barrier is tested a block ahead;
//  - six producer warps take the blocks in turn. For its block a warp loads the entries'
//    segments (all kBlk in flight; the indices were loaded one turn earlier), 16 bytes per lane
//    and four entries per load where the layout allows, waits until the slot's last block has
//    been consumed, and stores segments and values (word c of a segment belongs to consumer
//    lane c % 4 * 8 + c / 4, which makes these stores free of bank conflicts). Positions that
//    add nothing (past a row's end, or entries a row-pair unit leaves out) get the word -0.0 and
//    the value 1, which keep every accumulator as it is, so the consumer runs one form of the
//    step.
// The consumer shares its SM sub-partition with an idle warp only (warp 4): the chain issues
// one step every four cycles and loses a share of that rate to every busy neighbour.
//
// Measured on GB300: one row of 300,000 entries takes 1.02 ms over 32 fp32 columns (6.8 cycles per
// entry at 2070 MHz; 64-column slices read 32 bits at a time, copied by cp.async and handed over
// through flags: 1.9 ms, 13 cycles), 1.27 ms where B (153 MB) comes from DRAM, 1.67 ms where B's
// rows allow 4-byte loads only. The loads of a block are volatile because their order is the
// point: left to the compiler, they were moved down to their uses (3.1 ms in place of 1.3), as
// was each load put under a condition of its own (5.1 ms in place of 1.7).
//
// Every wait is bounded; a wait that gives up sets the timeout flag and an abort flag that
// makes the other role leave too; a row whose wait gave up is left unwritten. Loads land in
// registers, so nothing is in flight when a warp leaves. A malformed column index is flagged
// and its entry gets a zero segment (nothing is read for it).
//
// The list counters and a CTA-done counter live in the context's device words; the last CTA
// to finish resets them, so the next call starts from zero without a memset.
#include <algorithm>
#include <math.h>

#include "common.cuh"
#include "internal.h"
#include "spmm_vec.cuh"

namespace as {
namespace {

constexpr int kBlk = 64;        // entries per block: two per lane while they are staged
constexpr int kProducers = 6;
constexpr int kSlots = 6;       // ring slots: block g is in slot g % kSlots
constexpr int kWarps = 8;       // warp 0 the consumer, warp 4 idle
constexpr int kThreads = 32 * kWarps;
constexpr int kGrp = 8;         // entries read into registers together
constexpr unsigned kSpinLimit = 1u << 22;  // polls of a producer's wait
constexpr unsigned kAll = 0xffffffffu;
static_assert(kSlots % kProducers == 0, "a slot is always refilled by the same producer warp");

constexpr int kSlotBytes = kBlk * 128;  // [kBlk / 4][32 lanes][4 entries] words
constexpr int kRing = kSlots * kSlotBytes;
constexpr int kVals = kSlots * kBlk * 4;
constexpr int kSmem = kRing + kVals + 2 * kSlots * 8 + 16;

// producer index (0-5) of a warp, or -1 for the consumer and the idle warp
__device__ __forceinline__ int producer_of(int warp) {
    return (warp & 3) != 0 ? warp - 1 - (warp >> 2) : -1;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Whether the barrier's phase of this parity has completed (waits a short, bounded time).
__device__ __forceinline__ bool mbar_try(uint32_t bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// The same without waiting.
__device__ __forceinline__ bool mbar_test(uint32_t bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for a barrier's phase; false when `limit` polls pass or the other role gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, unsigned parity, unsigned limit,
                                          const volatile int *abort_flag) {
    for (unsigned i = 0; i < limit; ++i) {
        if (mbar_try(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    return false;
}

// One chain step for each of a lane's columns, from the entry's 32-bit word of B (a float, or
// two bf16) and its staged value: OP 0 the SpMM's fused multiply-add (acc = fma(b, v, acc)),
// 1 the unweighted copy-sum (acc + b), 2 max from -inf (fmaxf(acc, v * b)), 3 the DGL max
// (acc > v * b ? acc : v * b), 4 the fused multiply-add skipping zero values (the 1x4-blocked
// layout's empty slots), 5 the fused multiply-add over the entries a row-pair unit includes. The
// max forms find 1.0f as the value of an unweighted entry (x * 1.0f is x).
template <int OP>
__device__ __forceinline__ void step(float (&acc)[1], unsigned w, float v) {
    const float b = __uint_as_float(w);
    if constexpr (OP == 0 || OP == 5) acc[0] = fmaf(b, v, acc[0]);
    if constexpr (OP == 1) acc[0] = __fadd_rn(acc[0], b);
    if constexpr (OP == 2) acc[0] = fmaxf(acc[0], __fmul_rn(v, b));
    if constexpr (OP == 3) {
        const float x = __fmul_rn(v, b);
        acc[0] = acc[0] > x ? acc[0] : x;
    }
    if constexpr (OP == 4) acc[0] = v != 0.0f ? fmaf(b, v, acc[0]) : acc[0];
}
template <int OP>
__device__ __forceinline__ void step(float (&acc)[2], unsigned w, float v) {
    fma_bf16x2(w, static_cast<unsigned short>(__float_as_uint(v)), acc[0], acc[1]);
}
// The staged form of a value: a float's bits, or a bf16's 16 bits in a word.
__device__ __forceinline__ float staged(float v) { return v; }
__device__ __forceinline__ float staged(uint16_t v) { return __uint_as_float(v); }

// The word of a segment that consumer lane l holds.
__device__ __forceinline__ int word_of(int l) { return l % 8 * 4 + l / 8; }

__device__ __forceinline__ void prefetch_l2(const void *p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// How the rows of B can be read: 16 bytes at a time, 4 bytes, or (bf16) 2 bytes.
enum Access { kVec, kWord, kHalf };

// Loads of B, volatile: issued where they stand, all of a block before the wait for its slot.
// A lane's word of one entry's segment (p: its first column): a float, or two bf16 (kHalf: with
// two 2-byte loads).
template <int ACC>
__device__ __forceinline__ unsigned load_word(const void *p, bool second) {
    unsigned v;
    if constexpr (ACC != kHalf) {
        asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    } else {
        unsigned short lo, hi;
        asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(lo) : "l"(p));
        // a lane without a second column in the row reads its first again
        asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(hi)
                     : "l"(static_cast<const char *>(p) + (second ? 2 : 0)));
        v = lo | static_cast<unsigned>(hi) << 16;
    }
    return v;
}
__device__ __forceinline__ void load_vec(const void *p, unsigned *b) {
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                 : "l"(p));
}

// kGrp entries of a block in the consumer's registers: this lane's words of B and the values.
// The reads are volatile: they are issued where they stand, ahead of the steps of the group
// before.
struct Group {
    unsigned b[kGrp];
    float v[kGrp];
    __device__ __forceinline__ void read(uint32_t bs, uint32_t vs, int grp) {
#pragma unroll
        for (int i = 0; i < kGrp; i += 4) {
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3])
                         : "r"(vs + 4 * (grp * kGrp + i)));
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(b[i]), "=r"(b[i + 1]), "=r"(b[i + 2]), "=r"(b[i + 3])
                         : "r"(bs + 128 * (grp * kGrp + i)));
        }
    }
    template <int OP, int CPL>
    __device__ __forceinline__ void steps(float (&acc)[CPL]) const {
#pragma unroll
        for (int i = 0; i < kGrp; ++i) step<OP>(acc, b[i], v[i]);
    }
};

// T: storage type of val and B (float or uint16_t = bf16); ACC: how B is read; OP: the
// chain step above (the steps other than 0 take fp32 only). pair_flag: the row-pair layout's
// flags (OP 5 only).
template <typename T, int ACC, int OP>
__global__ void __launch_bounds__(kThreads, 2)
spmm_long(int M, int K, int N, int nnz, const int *__restrict__ rowptr,
          const int *__restrict__ colind, const T *__restrict__ val, const T *__restrict__ B,
          long ldb, float *__restrict__ C, long ldc, float beta, unsigned *status,
          const int *__restrict__ list, unsigned *counters, uint16_t *__restrict__ C16,
          bool relu, unsigned spin_limit, const uint8_t *__restrict__ pair_flag) {
    constexpr int CPL = 4 / static_cast<int>(sizeof(T));  // columns per lane
    constexpr int kCols = 32 * CPL;                       // columns per slice
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *ring = smem;                              // [kSlots][kSlotBytes]
    float *vals = reinterpret_cast<float *>(smem + kRing);   // [kSlots][kBlk]
    // per slot: filled (one arrival by its producer), consumed (one by the consumer)
    const uint32_t full_bar = smem_u32(smem + kRing + kVals), empty_bar = full_bar + 8 * kSlots;
    volatile int *abort_flag =
        reinterpret_cast<volatile int *>(smem + kRing + kVals + 2 * kSlots * 8);

    // launched as a programmatic dependent of the row-split kernel: wait for it to finish
    // (and its list writes to be visible) before reading the list
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned cap = static_cast<unsigned>(M);
    const int n_long = static_cast<int>(min(*reinterpret_cast<volatile unsigned *>(counters), cap));
    const int n_huge =
        static_cast<int>(min(*reinterpret_cast<volatile unsigned *>(counters + 2), cap));
    if (n_long + n_huge == 0) return;  // nothing listed: every CTA sees that, nothing to reset
    if (tid < 2 * kSlots) mbar_init(full_bar + 8 * tid, 1);
    if (tid == 0) *abort_flag = 0;
    __syncthreads();

    // row-pair mode: a listed item is a pair's even row; each pair gives two rows' units
    constexpr int kRowsPerItem = OP == 5 ? 2 : 1;
    const int n_slices = static_cast<int>(ceil_div(N, kCols)) * kRowsPerItem;
    const long units_huge = static_cast<long>(n_huge) * n_slices;
    const long units = units_huge + static_cast<long>(n_long) * n_slices;
    // This CTA's units. The huge rows' units (listed from the end) come first. Where they are
    // fewer than half of the CTAs, each has a CTA of its own and the others share the rest:
    // the longest chain is the call's critical path, and nothing is queued behind it.
    long u_first = blockIdx.x, u_step = gridDim.x, u_end = units;
    if (units_huge > 0 && 2 * units_huge <= gridDim.x) {
        if (blockIdx.x < units_huge)
            u_end = units_huge;
        else
            u_step = gridDim.x - units_huge;
    }
    const int pw = producer_of(warp);
    const bool weighted = val != nullptr;
    unsigned seq = 0;  // blocks of the CTA's stream before the current batch of units
    bool dead = warp != 0 && pw < 0;  // the idle warp leaves at once

    // the units in batches of 32, one per lane; every warp walks the same stream
    for (long ub = u_first; ub < u_end && !dead; ub += 32 * u_step) {
        const long u = ub + lane * u_step;
        int m_r = -1, m_lo = 0, m_lo1 = 0, m_L1 = 0, m_L = 0, m_slice = 0, m_nb = 0;
        if (u < u_end) {
            const bool huge = u < units_huge;
            const long v = huge ? u : u - units_huge;
            const int item = static_cast<int>(v / n_slices);
            const int sub = static_cast<int>(v - static_cast<long>(item) * n_slices);
            const int which = sub % kRowsPerItem;  // row-pair mode: 0 the even row, 1 the odd
            const int r0 = huge ? list[M - 1 - item] : list[item];
            if (r0 >= 0 && r0 + which < M) {
                // Row-pair mode: the even row chains over its segment's unflagged entries (all
                // of them when it has no partner); the odd row over the even segment's flagged
                // entries, then over its own segment (entries at positions L1.. map to lo1..).
                int hi, hi1 = 0;
                row_range(rowptr, r0, nnz, status, m_lo, hi);
                if (OP == 5 && which == 1) row_range(rowptr, r0 + 1, nnz, status, m_lo1, hi1);
                m_r = r0 + which;
                m_L1 = hi - m_lo;
                m_L = m_L1 + (hi1 - m_lo1);
                m_slice = sub / kRowsPerItem * kCols;
                m_nb = max(1, static_cast<int>(ceil_div(m_L, kBlk)));
            }
        }
        int incl = m_nb;  // blocks of the batch's units up to and with this lane's
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kAll, incl, o);
            if (lane >= o) incl += y;
        }
        const int n_units = static_cast<int>(min(32ll, ceil_div(u_end - ub, u_step)));
        for (int j = 0; j < n_units && !dead; ++j) {
            const int nb = __shfl_sync(kAll, m_nb, j);
            if (nb == 0) continue;  // a malformed list entry
            const unsigned base = seq + static_cast<unsigned>(__shfl_sync(kAll, incl, j) - nb);
            const int L = __shfl_sync(kAll, m_L, j);
            const int r = __shfl_sync(kAll, m_r, j);
            const int slice0 = __shfl_sync(kAll, m_slice, j);
            const int w = min(kCols, N - slice0);  // columns of this slice

            if (warp == 0) {
                // ---- consumer: the chains of columns c0 .. c0 + CPL - 1 of the slice ----
                constexpr float kInit = OP == 2 ? -INFINITY : OP == 3 ? -10000.0f : 0.0f;
                const int c0 = CPL * word_of(lane);
                const long out = static_cast<long>(r) * ldc + slice0 + c0;
                float acc[CPL];
#pragma unroll
                for (int c = 0; c < CPL; ++c)
                    acc[c] = beta != 0.0f && c0 + c < w ? C[out + c] * beta : kInit;
                auto full_of = [&](unsigned g) { return full_bar + 8 * (g % kSlots); };
                auto wait_full = [&](unsigned g) {  // block g of the stream is in its slot
                    const bool ok = __all_sync(
                        kAll, mbar_wait(full_of(g), g / kSlots & 1, spin_limit, abort_flag));
                    if (!ok) {
                        if (lane == 0) {
                            flag(status, kFlagTimeout);
                            *abort_flag = 1;
                        }
                        dead = true;
                    }
                    return ok;
                };
                auto release = [&](unsigned g) {  // its slot can be refilled
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty_bar + 8 * (g % kSlots));
                };
                auto b_of = [&](unsigned g) { return smem_u32(ring) + g % kSlots * kSlotBytes + 16 * lane; };
                auto v_of = [&](unsigned g) { return smem_u32(vals) + g % kSlots * (kBlk * 4); };
                const int nfull = L / kBlk;  // whole blocks
                unsigned g = base;
                if (nfull > 0 && wait_full(g)) {
                    uint32_t bs = b_of(g), vs = v_of(g);
                    constexpr int kG = kBlk / kGrp;  // groups per block, a multiple of four
                    Group q[4];  // three groups are read ahead of the one that runs
                    q[0].read(bs, vs, 0);
                    q[1].read(bs, vs, 1);
                    q[2].read(bs, vs, 2);
#pragma unroll 1
                    for (int t = 0; t < nfull; ++t, ++g) {
                        const bool more = t + 1 < nfull;
                        const bool ready = more && mbar_test(full_of(g + 1), (g + 1) / kSlots & 1);
#pragma unroll
                        for (int i = 0; i < kG; ++i) {
                            if (i == kG - 3) {
                                if (more && !__all_sync(kAll, ready) && !wait_full(g + 1)) break;
                                if (more) bs = b_of(g + 1), vs = v_of(g + 1);
                            }
                            // (past the last whole block: reads of it again, not used)
                            q[(i + 3) % 4].read(bs, vs, (i + 3) % kG);
                            q[i % 4].template steps<OP>(acc);
                        }
                        if (dead) break;
                        release(g);
                    }
                }
                // the last, partial block: its groups that hold an entry
                if (g != base + nb && !dead && wait_full(g)) {
                    const int n = L - nfull * kBlk;
#pragma unroll 1
                    for (int i = 0; i * kGrp < n; ++i) {
                        Group p;
                        p.read(b_of(g), v_of(g), i);
                        p.template steps<OP>(acc);
                    }
                    release(g);
                }
                if (!dead) {
#pragma unroll
                    for (int c = 0; c < CPL; ++c) {
                        if (c0 + c >= w) continue;
                        if (C16)
                            C16[out + c] = f32_to_bf16(relu_if(acc[c], relu));
                        else
                            C[out + c] = acc[c];
                    }
                }
            } else {
                // ---- producer pw: the blocks g of the stream with g % kProducers == pw ----
                const int t0 = static_cast<int>((kProducers + pw - base % kProducers) % kProducers);
                if (t0 >= nb) continue;
                const int lo = __shfl_sync(kAll, m_lo, j);
                int lo1 = 0, L1 = L, which = 0;
                bool partner = false;
                if constexpr (OP == 5) {
                    lo1 = __shfl_sync(kAll, m_lo1, j);
                    L1 = __shfl_sync(kAll, m_L1, j);
                    which = r & 1;  // pairs start at even rows
                    partner = (r | 1) < M;
                }
                // this lane's words of a segment (a lane past the slice repeats one in range):
                // four of every fourth entry (kVec), or its consumer lane's one
                const int words = static_cast<int>(ceil_div(w, CPL));
                const int wd = ACC == kVec ? min(lane % 8 * 4, words - 4) : min(word_of(lane), words - 1);
                const int sub = lane / 8;
                const bool second = CPL * wd + 1 < w;
                const T *bcol = B + slice0 + CPL * wd;
                constexpr unsigned kSkipWord = sizeof(T) == 4 ? 0x80000000u : 0x80008000u;  // -0.0
                const float one = sizeof(T) == 4 ? 1.0f : __uint_as_float(0x3f80u);  // staged 1
                // column index (-1: the position adds nothing, -2: out of range) and value of
                // this lane's entries of block t
                auto load = [&](int t, int (&k)[2], float (&x)[2]) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        int e = t * kBlk + 32 * h + lane;
                        k[h] = -1;
                        x[h] = OP == 4 ? 0.0f : one;
                        // the max steps: a position past the end repeats the last entry (which
                        // leaves them as they are)
                        if (OP == 2 || OP == 3) e = min(e, L - 1);
                        if (t >= nb || e >= L || e < 0) continue;
                        int idx = lo + e;
                        if constexpr (OP == 5) {
                            if (e >= L1)
                                idx = lo1 + (e - L1);
                            else if (partner && (__ldg(pair_flag + idx) != 0) != (which == 1))
                                continue;  // the other row's: neither checked nor read
                        }
                        k[h] = ld_stream(colind + idx);
                        if (weighted) x[h] = staged(ld_stream(val + idx));
                        // OP 4: an empty slot (value 0) may point past K; only a filled one is bad
                        if (OP == 4 && x[h] == 0.0f)
                            k[h] = -1;
                        else if (static_cast<unsigned>(k[h]) >= static_cast<unsigned>(K))
                            k[h] = -2;
                    }
                };
                int k[2];
                float x[2];
                load(t0, k, x);
#pragma unroll 1
                for (int t = t0; t < nb; t += kProducers) {
                    const unsigned g = base + static_cast<unsigned>(t);
                    const int slot = static_cast<int>(g % kSlots);
                    if (k[0] == -2 || k[1] == -2) flag(status, kFlagBadColind);
                    unsigned char *dst = ring + slot * kSlotBytes;
                    // the consumer is done with block g - kSlots
                    auto slot_free = [&] {
                        if (g < kSlots) return true;
                        return static_cast<bool>(
                            __all_sync(kAll, mbar_wait(empty_bar + 8 * slot, (g / kSlots - 1) & 1,
                                                       kSpinLimit, abort_flag)));
                    };
                    int nk[2];
                    float nx[2];
                    if constexpr (ACC == kVec) {
                        int kk[kBlk / 4];
                        unsigned b[kBlk];
#pragma unroll
                        for (int i = 0; i < kBlk / 4; ++i)
                            kk[i] = __shfl_sync(kAll, k[i / 8], i % 8 * 4 + sub);
                        if (__all_sync(kAll, k[0] >= 0 && k[1] >= 0)) {
#pragma unroll
                            for (int i = 0; i < kBlk / 4; ++i) load_vec(bcol + kk[i] * ldb, b + 4 * i);
                        } else {
#pragma unroll
                            for (int i = 0; i < kBlk / 4; ++i) {
#pragma unroll
                                for (int u = 0; u < 4; ++u) b[4 * i + u] = kk[i] == -1 ? kSkipWord : 0u;
                                if (kk[i] >= 0) load_vec(bcol + kk[i] * ldb, b + 4 * i);
                            }
                        }
                        load(t + kProducers, nk, nx);  // the next turn's, in flight meanwhile
                        if (!slot_free()) {
                            dead = true;
                            break;
                        }
#pragma unroll
                        for (int i = 0; i < kBlk; ++i)  // word 4 * (lane % 8) + i % 4 of an entry
                            *reinterpret_cast<unsigned *>(dst + 128 * i + lane % 8 * 16 + sub * 4) =
                                b[i];
                    } else {
                        // one word per lane and entry: in two halves, which the registers hold
#pragma unroll 1
                        for (int h = 0; h < 2 && !dead; ++h) {
                            unsigned b[kBlk / 2];
                            const int kh = h ? k[1] : k[0];
                            const bool clean = __all_sync(kAll, kh >= 0);
#pragma unroll
                            for (int i0 = 0; i0 < kBlk / 2; i0 += 8) {
                                int kk[8];
#pragma unroll
                                for (int i = 0; i < 8; ++i) kk[i] = __shfl_sync(kAll, kh, i0 + i);
                                if (clean) {
#pragma unroll
                                    for (int i = 0; i < 8; ++i)
                                        b[i0 + i] = load_word<ACC>(bcol + kk[i] * ldb, second);
                                } else {
#pragma unroll
                                    for (int i = 0; i < 8; ++i) {
                                        b[i0 + i] = kk[i] == -1 ? kSkipWord : 0u;
                                        if (kk[i] >= 0)
                                            b[i0 + i] = load_word<ACC>(bcol + kk[i] * ldb, second);
                                    }
                                }
                            }
                            if (h == 0) {
                                load(t + kProducers, nk, nx);
                                dead = !slot_free();
                                if (dead) break;
                            }
#pragma unroll
                            for (int i = 0; i < kBlk / 2; i += 4)
                                *reinterpret_cast<uint4 *>(dst + 128 * (32 * h + i) + 16 * lane) =
                                    make_uint4(b[i], b[i + 1], b[i + 2], b[i + 3]);
                        }
                        if (dead) break;
                    }
                    vals[slot * kBlk + lane] = x[0];
                    vals[slot * kBlk + 32 + lane] = x[1];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full_bar + 8 * slot);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        k[h] = nk[h];
                        x[h] = nx[h];
                        // the next turn's segments on their way into L2
                        if (k[h] >= 0) prefetch_l2(B + slice0 + k[h] * ldb);
                    }
                }
            }
        }
        seq += static_cast<unsigned>(__shfl_sync(kAll, incl, 31));
    }

    // the last CTA out resets the list counters and the done counter for the next call
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const unsigned total = gridDim.x;
        if (atomicAdd(counters + 1, 1u) == total - 1) {
            counters[0] = 0;
            counters[1] = 0;
            counters[2] = 0;
            __threadfence();
        }
    }
}

template <typename T, int ACC, int OP = 0>
as_status launch(as_ctx *ctx, const SpmmArgs &a, const int *list, cudaStream_t s,
                 const uint8_t *pair_flag = nullptr) {
    auto k = spmm_long<T, ACC, OP>;
    static int per_sm[64] = {};  // resident CTAs per multiprocessor, per device
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64) return fail(AS_ERR_INVALID_VALUE, "spmm long rows: device index");
    if (!per_sm[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return check_cuda(e, "spmm long rows: shared memory attribute");
        int n = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kThreads, kSmem);
        if (e != cudaSuccess) return check_cuda(e, "spmm long rows: occupancy");
        per_sm[dev] = std::max(1, n);
    }
    // one wave of CTAs striding over the (row, slice) units
    const long max_units = static_cast<long>(a.M) * ceil_div(a.N, 128 / static_cast<int>(sizeof(T))) *
                           (OP == 5 ? 2 : 1);
    dim3 grid(static_cast<unsigned>(
        std::max(1L, std::min(max_units, static_cast<long>(per_sm[dev]) * ctx->sms))));
    // programmatic dependent launch (outside stream capture): the CTAs are scheduled while
    // the row-split kernel drains, hiding this launch when there are no long rows
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(s, &cap);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cap == cudaStreamCaptureStatusNone ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, k, a.M, a.K, a.N, a.nnz, a.rowptr, a.colind,
                                       static_cast<const T *>(a.val), static_cast<const T *>(a.B),
                                       a.ldb, a.C, a.ldc, a.beta, a.status, list, ctx->d_long,
                                       a.C16, a.relu, ctx->spin_limit, pair_flag);
    ctx->launches++;
    return check_cuda(e != cudaSuccess ? e : cudaGetLastError(), "spmm long rows launch");
}

}  // namespace

as_status spmm_long_launch(as_ctx *ctx, int dtype, const SpmmArgs &a, const int *list,
                           cudaStream_t s, int op, const uint8_t *pair_flag) {
    if (dtype != 0 && op != 0)
        return fail(AS_ERR_UNSUPPORTED, "spmm long rows: this step takes fp32");
    if (op == 5 && !pair_flag)
        return fail(AS_ERR_INVALID_VALUE, "spmm long rows: row pairs need their flags");
    const long esz = dtype == 0 ? 4 : 2;
    auto rows_of = [&](long bytes) {  // every row of B (and its last piece) in aligned pieces
        return a.N * esz % bytes == 0 && a.ldb * esz % bytes == 0 &&
               reinterpret_cast<uintptr_t>(a.B) % bytes == 0;
    };
    const bool vec = rows_of(16);
    if (dtype != 0) {
        if (vec) return launch<uint16_t, kVec>(ctx, a, list, s);
        return rows_of(4) ? launch<uint16_t, kWord>(ctx, a, list, s)
                          : launch<uint16_t, kHalf>(ctx, a, list, s);
    }
#define AS_LONG_OP(O)                                                                        \
    case O:                                                                                  \
        return vec ? launch<float, kVec, O>(ctx, a, list, s, pair_flag)                      \
                   : launch<float, kWord, O>(ctx, a, list, s, pair_flag);
    switch (op) { AS_LONG_OP(0) AS_LONG_OP(1) AS_LONG_OP(2) AS_LONG_OP(3) AS_LONG_OP(4) AS_LONG_OP(5) }
#undef AS_LONG_OP
    return fail(AS_ERR_INVALID_VALUE, "spmm long rows: unknown reduction");
}

}  // namespace as
