// CSR -> CSC transpose, CSR validation and small conversion kernels (sm_103a).
//
// Transpose = stable sort of the CSR entries by column. The CSR order is already
// row-ascending, so a stable sort by column leaves rows ascending inside every column:
// exactly the canonical CSC that scipy's tocsc() builds on the reference's GCN path
// (gcn/pytorch-custom/gcn_custom.py:52), and the order the reference's counting transpose
// (sparseTranspose.cpp:95-142) gives when its scatter runs in order. The sort is an LSD
// radix sort over digits of the column id, ceil(bits / 8) passes of equal width (20 bits: three
// digits of 7), each pass:
//   1. tile histogram   -- each CTA counts the digits of its tile of entries into
//                          hist[digit * tiles + tile] (shared-memory atomics on counts:
//                          the counts, unlike positions, do not depend on ordering);
//   2. exclusive scan   -- over hist in (digit, tile) order, giving every (digit, tile) its
//                          first output slot;
//   3. stable scatter   -- each warp of a CTA ranks the entries of its own consecutive part of
//                          the tile among equal digits before them (a ballot per bit finds
//                          the lanes of a digit, a warp-private count those before them),
//                          one scan over warps and digits turns ranks into slots of the tile,
//                          the tile is parked in shared memory sorted by digit, then key, row
//                          and value are written out in that order, so each digit's entries
//                          leave as one coalesced run.
// The first pass works out each entry's row from the row pointer as it goes (each row marks its
// first entry in the tile, a running maximum gives the rest), so row ids are never written and
// read just to be sorted.
// What bounds a pass is its traffic (12 bytes read and written per entry) and how long the runs
// are that leave a tile: 4096 entries and 128 digits give runs of 128 bytes. Measured on 16.8M
// entries and 1M columns: a pass's scatter takes 110 us (2,048-entry tiles ranked in eight rounds
// with a CTA barrier each: 166; ranks by __match_any_sync in place of the ballots: 150-169), the
// rows 63 us more in the first pass (an expansion pass of its own: 79 us and its traffic), the
// whole call 479 us (751 before). Matrices of few entries take tiles of 1024, which spread over
// the chip (20,000 entries: 43 us, 68 before).
// No position depends on timing, so the output is identical run to run. colptr comes
// from the sorted keys (first slot of every column). All indices stay inside their
// buffers for any input; malformed input sets the status word instead of faulting.
#include "common.cuh"
#include "internal.h"

namespace as {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kSortThreads = 512;   // of a tile's CTA
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kLargeItems = 8;      // entries per thread of a tile
constexpr int kSmallItems = 2;
// From here on large tiles. Both, on square, narrow and wide matrices: 100,000 entries 41-72 us with
// small tiles, 39-80 with large ones; 300,000 43-67 and 47-74; 350,000 to 400,000 the same within 4 %;
// 500,000 49-79 and 47-74; 1M 62-97 and 53-84.
constexpr int kLargeNnz = 300000;
constexpr int kBins = 256;          // digits per pass at most

// ---- exclusive scan of int32 (three phases, no cross-CTA waits) ---------------------------
constexpr int kScanItems = 8;
constexpr int kScanChunk = kThreads * kScanItems;  // 2048 per CTA

__device__ __forceinline__ int block_exclusive_scan(int v, int *smem_warp, int &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < kWarps ? smem_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kWarps) smem_warp[lane] = w;  // inclusive warp totals
    }
    __syncthreads();
    total = smem_warp[kWarps - 1];
    const int before = warp ? smem_warp[warp - 1] : 0;
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(kThreads)
scan_reduce(const int *__restrict__ in, long n, int *__restrict__ block_sums) {
    __shared__ int sw[kWarps];
    const long base = static_cast<long>(blockIdx.x) * kScanChunk;
    int s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const long idx = base + static_cast<long>(i) * kThreads + threadIdx.x;
        if (idx < n) s += in[idx];
    }
    int total;
    block_exclusive_scan(s, sw, total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// One CTA: the exclusive scan of nb block sums in place, a chunk at a time.
__global__ void __launch_bounds__(kThreads) scan_block_sums(int *sums, long nb) {
    __shared__ int sw[kWarps];
    int carry = 0;
    for (long base = 0; base < nb; base += kScanChunk) {
        const long first = base + static_cast<long>(threadIdx.x) * kScanItems;
        int v[kScanItems];
        int s = 0;
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            v[i] = first + i < nb ? sums[first + i] : 0;
            s += v[i];
        }
        int total;
        int run = block_exclusive_scan(s, sw, total) + carry;
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            if (first + i < nb) sums[first + i] = run;
            run += v[i];
        }
        carry += total;
    }
}

// Each CTA adds up the sums of the CTAs before it (`scanned`: finds the total in its own place),
// then scans its own chunk.
__global__ void __launch_bounds__(kThreads)
scan_downsweep(const int *__restrict__ in, long n, const int *__restrict__ block_sums,
               int *__restrict__ out, bool vec, bool scanned) {
    __shared__ int sw[kWarps];
    const long base = static_cast<long>(blockIdx.x) * kScanChunk;
    int prefix;
    if (scanned) {
        prefix = block_sums[blockIdx.x];
    } else {
        int before = 0;
        for (unsigned i = threadIdx.x; i < blockIdx.x; i += kThreads) before += block_sums[i];
        block_exclusive_scan(before, sw, prefix);
    }
    // blocked layout: thread t owns items [t*kScanItems, (t+1)*kScanItems)
    const long first = base + static_cast<long>(threadIdx.x) * kScanItems;
    const bool whole = vec && first + kScanItems <= n;
    int v[kScanItems];
    int s = 0;
    if (whole) {
#pragma unroll
        for (int i = 0; i < kScanItems; i += 4) {
            const int4 q = *reinterpret_cast<const int4 *>(in + first + i);
            v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) v[i] = first + i < n ? in[first + i] : 0;
    }
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) s += v[i];
    int total;
    int run = block_exclusive_scan(s, sw, total) + prefix;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const int t = v[i];
        v[i] = run;
        run += t;
    }
    if (whole) {
#pragma unroll
        for (int i = 0; i < kScanItems; i += 4)
            *reinterpret_cast<int4 *>(out + first + i) = make_int4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; ++i)
            if (first + i < n) out[first + i] = v[i];
    }
}

// The scan of n ints in launches on s; returns their number. Every CTA adding up the block sums
// before it saves a launch while they are few; the additions grow with the square of n, so past
// kManyBlocks (17M ints) one CTA scans the block sums first (400M row counts: 2.35 ms less of a
// format conversion's 43.2; 24M and 40M the same either way).
constexpr long kManyBlocks = 8192;
int launch_scan(const int *in, int *out, long n, int *block_sums, bool vec, cudaStream_t s) {
    const long nb = ceil_div(n, kScanChunk);
    const unsigned grid = static_cast<unsigned>(nb);
    const bool many = nb > kManyBlocks;
    scan_reduce<<<grid, kThreads, 0, s>>>(in, n, block_sums);
    if (many) scan_block_sums<<<1, kThreads, 0, s>>>(block_sums, nb);
    scan_downsweep<<<grid, kThreads, 0, s>>>(in, n, block_sums, out, vec, many);
    return many ? 3 : 2;
}

// One CTA, n <= kScanChunk: the scan in place in one launch.
__global__ void __launch_bounds__(kThreads) scan_one_block(int *data, long n) {
    __shared__ int sw[kWarps];
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const long idx = static_cast<long>(threadIdx.x) * kScanItems + i;
        v[i] = idx < n ? data[idx] : 0;
        s += v[i];
    }
    int total;
    int run = block_exclusive_scan(s, sw, total);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const long idx = static_cast<long>(threadIdx.x) * kScanItems + i;
        if (idx < n) data[idx] = run;
        run += v[i];
    }
}

// ---- transpose kernels -----------------------------------------------------------------
// Inclusive maximum over the CTA's threads before and with each (values >= 0).
__device__ __forceinline__ int block_max_scan(int v, int *smem_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v = max(v, y);
    }
    if (lane == 31) smem_warp[warp] = v;
    __syncthreads();
    for (int w = 0; w < warp; ++w) v = max(v, smem_warp[w]);
    __syncthreads();
    return v;
}

template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads)
radix_histogram(const int *__restrict__ keys, int nnz, int shift, int bins, int tiles, int N,
                int *__restrict__ hist, unsigned *status, int check_range, bool vec) {
    __shared__ int h[kBins];
    if (threadIdx.x < kBins) h[threadIdx.x] = 0;
    __syncthreads();
    const long base = static_cast<long>(blockIdx.x) * kSortThreads * ITEMS;
    int kv[ITEMS];  // all of this thread's keys are loaded before any is counted
    const long first = base + static_cast<long>(threadIdx.x) * ITEMS;
    int n = ITEMS;
    if (ITEMS % 4 == 0 && vec && base + kSortThreads * ITEMS <= nnz) {
#pragma unroll
        for (int i = 0; i + 3 < ITEMS; i += 4) {
            const int4 q = *reinterpret_cast<const int4 *>(keys + first + i);
            kv[i] = q.x; kv[i + 1] = q.y; kv[i + 2] = q.z; kv[i + 3] = q.w;
        }
    } else {
        n = static_cast<int>(min(static_cast<long>(ITEMS), max(0L, nnz - first)));
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) kv[i] = i < n ? keys[first + i] : 0;
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (i < n) {
            const int k = kv[i];
            if (check_range && static_cast<unsigned>(k) >= static_cast<unsigned>(N))
                flag(status, kFlagBadColind);
            atomicAdd(&h[(static_cast<unsigned>(k) >> shift) & (bins - 1)], 1);
        }
    }
    __syncthreads();
    if (threadIdx.x < bins)
        hist[static_cast<long>(threadIdx.x) * tiles + blockIdx.x] = h[threadIdx.x];
}

// rows null: the first pass, rows from rowptr (an entry that no well-formed row holds is flagged
// and given row 0, as are all when the pointer does not run from 0 to nnz, so every row written
// is in [0, M)). vals null: no payload, or with iota each entry's position.
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads, 2)
radix_scatter(const int *__restrict__ keys, const int *__restrict__ rows,
              const unsigned *__restrict__ vals, bool iota, int nnz, int shift, int bins, int tiles,
              const int *__restrict__ offsets, int *__restrict__ okeys, int *__restrict__ orows,
              unsigned *__restrict__ ovals, int M, const int *__restrict__ rowptr,
              unsigned *status) {
    constexpr int kTile = kSortThreads * ITEMS;
    __shared__ int start[kBins];               // first local slot of each digit in this tile
    __shared__ int goff[kBins];                // its first global slot, less the local one
    __shared__ unsigned short cnt[kSortWarps][kBins];  // per warp and digit: count, then first slot
    __shared__ int sw[kSortWarps];
    __shared__ int row_span[2];
    extern __shared__ int parked[];            // the tile, sorted by digit (stable)
    int *sk = parked, *sr = parked + kTile;
    unsigned *sv = reinterpret_cast<unsigned *>(parked + 2 * kTile);  // value bits or position
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long base = static_cast<long>(blockIdx.x) * kTile;
    const int n_tile = static_cast<int>(nnz - base < kTile ? nnz - base : kTile);
    const int w0 = warp * (32 * ITEMS) + lane;  // this lane's first entry in the tile
    int kr[ITEMS], rr[ITEMS];
    unsigned vr[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int li = w0 + 32 * i;
        kr[i] = 0;
        rr[i] = 0;
        vr[i] = 0u;
        if (li < n_tile) {
            kr[i] = keys[base + li];
            if (rows) rr[i] = rows[base + li];
            if (vals)
                vr[i] = vals[base + li];
            else if (iota)
                vr[i] = static_cast<unsigned>(base + li);  // the entry's CSR position
        }
    }
    for (int i = tid; i < kSortWarps * kBins; i += kSortThreads) (&cnt[0][0])[i] = 0;
    if (!rows) {
        // Rows of the tile's entries: each row marks its first entry of the tile (of rows that
        // start at one entry the last is the one that holds it), and the running maximum over
        // the tile is every entry's row.
        const bool ends = __ldg(rowptr) == 0 && __ldg(rowptr + M) == nnz;
        if (!ends && tid == 0 && blockIdx.x == 0) flag(status, kFlagBadRowptr);
        if (warp < 2) {
            const int r = find_row<32>(rowptr, M, warp == 0 ? base : base + n_tile - 1, lane, 0xffffffffu);
            if (lane == 0) row_span[warp] = r;
        }
        for (int i = tid; i < kTile; i += kSortThreads) sr[i] = 0;
        __syncthreads();
        const int ra = row_span[0], rb = row_span[1];
        // A tile across a long run of empty rows: each entry looks its row up instead of the CTA
        // marking them all (10M rows, 1M entries of which the last follows 9M empty rows: 5.0
        // and 0.12 ms for the call).
        const bool search = rb - ra > 16 * kTile;
        for (long r = static_cast<long>(ra) + tid; r <= rb && !search; r += kSortThreads) {
            const long at = static_cast<long>(__ldg(rowptr + r)) - base;
            if (r == ra || (at > 0 && at < n_tile))
                atomicMax(sr + (r == ra ? 0 : at), static_cast<int>(r));
        }
        __syncthreads();
        int m = 0, mine[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            m = max(m, sr[tid * ITEMS + i]);
            mine[i] = m;
        }
        const int upto = block_max_scan(m, sw);
        int prev = __shfl_up_sync(0xffffffffu, upto, 1);
        if (lane == 0) sw[warp] = 0;
        __syncthreads();
        if (lane == 31 && warp + 1 < kSortWarps) sw[warp + 1] = upto;
        __syncthreads();
        if (lane == 0) prev = sw[warp];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) sr[tid * ITEMS + i] = max(mine[i], prev);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int li = w0 + 32 * i;
            if (!ends || li >= n_tile) continue;
            const long e = base + li;
            int r = sr[li];
            if (search) {  // the last row of the span that starts at or before the entry
                r = ra;
                for (int hi = rb; r < hi;) {
                    const int mid = r + (hi - r + 1) / 2;
                    if (__ldg(rowptr + mid) <= e)
                        r = mid;
                    else
                        hi = mid - 1;
                }
            }
            const int rs = __ldg(rowptr + r), re = __ldg(rowptr + r + 1);
            if (rs < 0 || re > nnz || e < rs || e >= re)
                flag(status, kFlagBadRowptr);  // malformed pointers: row 0
            else
                rr[i] = r;
        }
    }
    __syncthreads();
    // ranks among equal digits of the warp's entries before each
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned short *mine = cnt[warp];
    // lanes whose digit is this lane's: a ballot per bit
    unsigned peers[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        peers[i] = __ballot_sync(0xffffffffu, w0 + 32 * i < n_tile);
    for (int bit = 1; bit < bins; bit <<= 1) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const bool one = (static_cast<unsigned>(kr[i]) >> shift) & bit;
            const unsigned m = __ballot_sync(0xffffffffu, one);
            peers[i] &= one ? m : ~m;
        }
    }
    int rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const bool valid = w0 + 32 * i < n_tile;
        const int d = static_cast<int>((static_cast<unsigned>(kr[i]) >> shift) & (bins - 1));
        const int lower = __popc(peers[i] & lt_mask);
        const int before = valid ? mine[d] : 0;
        __syncwarp();
        if (valid && lower == 0) mine[d] = static_cast<unsigned short>(before + __popc(peers[i]));
        __syncwarp();
        rank[i] = before + lower;
    }
    __syncthreads();
    {   // per digit: exclusive prefix over warps; then over digits
        int acc = 0;
        if (tid < bins) {
#pragma unroll
            for (int w = 0; w < kSortWarps; ++w) {
                const int c = cnt[w][tid];
                cnt[w][tid] = static_cast<unsigned short>(acc);
                acc += c;
            }
        }
        int v = acc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane == 31) sw[warp] = v;
        __syncthreads();
        int st = v - acc;
        for (int w = 0; w < warp; ++w) st += sw[w];
        if (tid < bins) {
            start[tid] = st;
            goff[tid] = offsets[static_cast<long>(tid) * tiles + blockIdx.x] - st;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (w0 + 32 * i < n_tile) {
            const int d = static_cast<int>((static_cast<unsigned>(kr[i]) >> shift) & (bins - 1));
            const int pos = start[d] + mine[d] + rank[i];
            sk[pos] = kr[i];
            sr[pos] = rr[i];
            sv[pos] = vr[i];
        }
    }
    __syncthreads();
    // write out in local (digit-sorted) order: a digit's entries go to consecutive global
    // slots, so neighbouring threads write neighbouring addresses
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int p = tid + i * kSortThreads;
        if (p < n_tile) {
            const int k = sk[p];
            const int g = goff[(static_cast<unsigned>(k) >> shift) & (bins - 1)] + p;
            okeys[g] = k;
            orows[g] = sr[p];
            if (ovals) ovals[g] = sv[p];
        }
    }
}

// colptr[c] = first slot whose key >= c, from the sorted keys (256-byte aligned scratch): eight
// consecutive slots per thread.
constexpr int kColSlots = 8;
__global__ void __launch_bounds__(kThreads)
colptr_from_keys(const int *__restrict__ skeys, int nnz, int N, int *__restrict__ colptr) {
    const long p0 = (static_cast<long>(blockIdx.x) * kThreads + threadIdx.x) * kColSlots;
    if (p0 > nnz) return;
    int k[kColSlots];
    if (p0 + kColSlots <= nnz) {
#pragma unroll
        for (int i = 0; i < kColSlots; i += 4) {
            const int4 v = *reinterpret_cast<const int4 *>(skeys + p0 + i);
            k[i] = v.x; k[i + 1] = v.y; k[i + 2] = v.z; k[i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kColSlots; ++i) k[i] = p0 + i < nnz ? skeys[p0 + i] : N;
    }
    // keys out of range were flagged: clamped to [-1, N] they move no column pointer out of place
    int prev = p0 == 0 ? -1 : max(skeys[p0 - 1], -1);
#pragma unroll
    for (int i = 0; i < kColSlots; ++i) {
        if (p0 + i > nnz) break;
        const int p = static_cast<int>(p0) + i;
        const int cur = p == nnz ? N : min(k[i], N);
        for (int c = prev + 1; c <= cur && prev < N; ++c) colptr[c] = p;
        prev = max(k[i], -1);
    }
}

// ---- validation --------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
csr_validate(int n_rows, int n_cols, int nnz, const int *__restrict__ rowptr,
             const int *__restrict__ colind, int require_sorted, unsigned *result) {
    const long r = static_cast<long>(blockIdx.x) * kThreads + threadIdx.x;
    if (r == 0 && (__ldg(rowptr) != 0 || __ldg(rowptr + n_rows) != nnz)) atomicOr(result, 1u);
    if (r >= n_rows) return;
    int lo = __ldg(rowptr + r), hi = __ldg(rowptr + r + 1);
    if (hi < lo || lo < 0 || hi > nnz) {
        atomicOr(result, 2u);
        return;
    }
    int prev = -1;
    for (int e = lo; e < hi; ++e) {
        const int c = __ldg(colind + e);
        if (static_cast<unsigned>(c) >= static_cast<unsigned>(n_cols)) atomicOr(result, 4u);
        if (require_sorted && c <= prev) atomicOr(result, 8u);
        prev = c;
    }
}

__global__ void __launch_bounds__(kThreads)
f32_to_bf16_kernel(long n, const float *__restrict__ src, uint16_t *__restrict__ dst) {
    for (long i = static_cast<long>(blockIdx.x) * kThreads + threadIdx.x; i < n;
         i += static_cast<long>(gridDim.x) * kThreads)
        dst[i] = f32_to_bf16(src[i]);
}

__global__ void zero_u32(unsigned *p) { *p = 0u; }

// Digits of an N-column matrix: as few passes as digits of at most 8 bits give, of equal width.
struct Digits {
    int passes, bits;
};
Digits radix_digits(int N) {
    int bits = 1;
    while (bits < 31 && (1L << bits) < N) ++bits;
    const int passes = (bits + 7) / 8;
    return {passes, (bits + passes - 1) / passes};
}
int tile_entries(int nnz) { return kSortThreads * (nnz >= kLargeNnz ? kLargeItems : kSmallItems); }

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

// Exclusive scan of n ints (in may equal out); `work` holds ceil(n / 2048) ints.
static as_status exclusive_scan(as_ctx *ctx, const int *in, int *out, long n, int *work,
                                cudaStream_t s) {
    if (n == 0) return AS_OK;
    const bool vec = (reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
    ctx->launches += launch_scan(in, out, n, work, vec, s);
    return check_cuda(cudaGetLastError(), "scan launch");
}

as_status exclusive_scan_i32(as_ctx *ctx, const int *in, int *out, long n, cudaStream_t s) {
    void *w = nullptr;
    as_status st = scratch(ctx, sizeof(int) * static_cast<size_t>(ceil_div(n, kScanChunk) + 1), &w);
    if (st != AS_OK) return st;
    return exclusive_scan(ctx, in, out, n, static_cast<int *>(w), s);
}

// Raw launches of the passes, shared by the two entry points (the caller reads the launch error).
// Keys alternate between keysA and keysB. Rows and values of a non-last pass go to either the
// scratch buffer or the caller's output (free until the last pass), chosen backwards from the
// last pass so that no pass reads and writes the same buffer and the last pass reads scratch and
// writes rowind / final_v. Returns the number of launches.
struct SortBuffers {
    int *keysA, *keysB, *rowsT;
    unsigned *valsT;
    int *hist, *sums;
};
static int sort_by_column(int M, int N, int nnz, const int *rowptr, const int *colind,
                          const unsigned *vals, bool iota, int *colptr, int *rowind,
                          unsigned *final_v, const SortBuffers &w, unsigned *status,
                          cudaStream_t s) {
    const Digits dg = radix_digits(N);
    const int bins = 1 << dg.bits;
    const bool large = nnz >= kLargeNnz;
    const int tile = tile_entries(nnz);
    const unsigned tiles = static_cast<unsigned>(ceil_div(nnz, tile));
    const long hist_n = static_cast<long>(tiles) * bins;
    const unsigned nb = static_cast<unsigned>(ceil_div(hist_n, kScanChunk));
    const size_t smem = 3 * sizeof(int) * static_cast<size_t>(tile);
    int launches = 0;
    if (large)  // past the 48 KB that need no opt-in, with the static arrays
        cudaFuncSetAttribute(radix_scatter<kLargeItems>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem));
    const int *src_k = colind;
    const int *src_r = nullptr;  // the first pass takes them from rowptr
    const unsigned *src_v = vals;
    for (int pass = 0; pass < dg.passes; ++pass) {
        const bool last = pass == dg.passes - 1;
        const bool to_scratch = ((dg.passes - 1 - pass) & 1) != 0;
        int *dk = (pass & 1) ? w.keysB : w.keysA;
        int *dr = (last || !to_scratch) ? rowind : w.rowsT;
        unsigned *dv = final_v ? ((last || !to_scratch) ? final_v : w.valsT) : nullptr;
        const int shift = dg.bits * pass;
        const bool vec = reinterpret_cast<uintptr_t>(src_k) % 16 == 0;
        if (large)
            radix_histogram<kLargeItems><<<tiles, kSortThreads, 0, s>>>(
                src_k, nnz, shift, bins, tiles, N, w.hist, status, pass == 0, vec);
        else
            radix_histogram<kSmallItems><<<tiles, kSortThreads, 0, s>>>(
                src_k, nnz, shift, bins, tiles, N, w.hist, status, pass == 0, vec);
        if (nb == 1) {
            scan_one_block<<<1, kThreads, 0, s>>>(w.hist, hist_n);
            launches += 1;
        } else {
            launches += launch_scan(w.hist, w.hist, hist_n, w.sums, true, s);
        }
        if (large)
            radix_scatter<kLargeItems><<<tiles, kSortThreads, smem, s>>>(
                src_k, src_r, src_v, iota && pass == 0, nnz, shift, bins, tiles, w.hist, dk, dr, dv, M,
                rowptr, status);
        else
            radix_scatter<kSmallItems><<<tiles, kSortThreads, smem, s>>>(
                src_k, src_r, src_v, iota && pass == 0, nnz, shift, bins, tiles, w.hist, dk, dr, dv, M,
                rowptr, status);
        launches += 2;
        src_k = dk;
        src_r = dr;
        src_v = dv;
    }
    colptr_from_keys<<<static_cast<unsigned>(ceil_div(static_cast<long>(nnz) + 1,
                                                      kThreads * kColSlots)),
                       kThreads, 0, s>>>(src_k, nnz, N, colptr);
    return launches + 1;
}

size_t csr2csc_scratch_bytes(int nnz, int N, bool with_val) {
    const long hist = ceil_div(nnz, tile_entries(nnz)) << radix_digits(N).bits;
    size_t b = 0;
    b += 2 * align256(sizeof(int) * static_cast<size_t>(nnz));    // keys ping-pong
    b += align256(sizeof(int) * static_cast<size_t>(nnz));        // rows (intermediate)
    if (with_val) b += align256(sizeof(float) * static_cast<size_t>(nnz));
    b += align256(sizeof(int) * static_cast<size_t>(hist));       // histogram / offsets
    b += align256(sizeof(int) * static_cast<size_t>(ceil_div(hist, kScanChunk) + 1));
    return b;
}

as_status csr2csc_launch(as_ctx *ctx, int M, int N, int nnz, const int *rowptr,
                         const int *colind, const float *val, int *colptr, int *rowind,
                         float *cscval, void *work, cudaStream_t s, int *perm) {
    if (nnz == 0) {
        if (cudaMemsetAsync(colptr, 0, sizeof(int) * (static_cast<size_t>(N) + 1), s) != cudaSuccess)
            return check_cuda(cudaGetLastError(), "csr2csc memset");
        return AS_OK;
    }
    if (M == 0) return fail(AS_ERR_INVALID_CSR, "csr2csc: nnz > 0 with zero rows");
    if (N == 0) return fail(AS_ERR_INVALID_CSR, "csr2csc: nnz > 0 with zero columns");
    // the payload: the values' bits, or (perm given) each entry's CSR position
    const bool wv = val != nullptr || perm != nullptr;
    unsigned *final_v = !wv ? nullptr : perm ? reinterpret_cast<unsigned *>(perm)
                                             : reinterpret_cast<unsigned *>(cscval);
    const long hist_n = ceil_div(nnz, tile_entries(nnz)) << radix_digits(N).bits;
    char *p = static_cast<char *>(work);
    auto take = [&](size_t bytes) { char *q = p; p += align256(bytes); return q; };
    SortBuffers w;
    w.keysA = reinterpret_cast<int *>(take(sizeof(int) * static_cast<size_t>(nnz)));
    w.keysB = reinterpret_cast<int *>(take(sizeof(int) * static_cast<size_t>(nnz)));
    w.rowsT = reinterpret_cast<int *>(take(sizeof(int) * static_cast<size_t>(nnz)));
    w.valsT = wv ? reinterpret_cast<unsigned *>(take(sizeof(unsigned) * static_cast<size_t>(nnz))) : nullptr;
    w.hist = reinterpret_cast<int *>(take(sizeof(int) * static_cast<size_t>(hist_n)));
    w.sums = reinterpret_cast<int *>(take(sizeof(int) * static_cast<size_t>(ceil_div(hist_n, kScanChunk) + 1)));
    ctx->launches += sort_by_column(M, N, nnz, rowptr, colind,
                                    perm ? nullptr : reinterpret_cast<const unsigned *>(val),
                                    perm != nullptr, colptr, rowind, final_v, w, ctx->d_status, s);
    return check_cuda(cudaGetLastError(), "csr2csc launch");
}

as_status csr_validate_launch(as_ctx *ctx, int n_rows, int n_cols, int nnz, const int *rowptr,
                              const int *colind, int require_sorted, unsigned *result,
                              cudaStream_t s) {
    zero_u32<<<1, 1, 0, s>>>(result);
    csr_validate<<<static_cast<unsigned>(ceil_div(static_cast<long>(n_rows) + 1, kThreads)),
                   kThreads, 0, s>>>(n_rows, n_cols, nnz, rowptr, colind, require_sorted, result);
    ctx->launches += 2;
    return check_cuda(cudaGetLastError(), "csr_validate launch");
}

// dst[i] = src[idx[i]] for i < n (idx in [0, n_src); others flag and give 0): values moved
// between orderings of the same entries, e.g. from CSC to CSR order through the inverse of
// as_csr2csc_perm's permutation. Four outputs per thread: one 16-byte index load, four
// independent gathers, one 16-byte store.
__global__ void __launch_bounds__(kThreads)
gather_f32(long n, long n_src, const float *__restrict__ src, const int *__restrict__ idx,
           float *__restrict__ dst, unsigned *status) {
    const long stride = static_cast<long>(gridDim.x) * kThreads * 4;
    for (long i = (static_cast<long>(blockIdx.x) * kThreads + threadIdx.x) * 4; i < n; i += stride) {
        if (i + 4 <= n) {
            const int4 k = __ldcs(reinterpret_cast<const int4 *>(idx + i));
            const int kk[4] = {k.x, k.y, k.z, k.w};
            float v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool ok = static_cast<unsigned long>(static_cast<unsigned>(kk[q])) <
                                static_cast<unsigned long>(n_src);
                if (!ok) flag(status, kFlagBadPerm);
                v[q] = ok ? __ldg(src + kk[q]) : 0.0f;
            }
            __stcs(reinterpret_cast<float4 *>(dst + i), make_float4(v[0], v[1], v[2], v[3]));
        } else {
            for (long j = i; j < n; ++j) {
                const int k = idx[j];
                const bool ok = k >= 0 && static_cast<long>(k) < n_src;
                if (!ok) flag(status, kFlagBadPerm);
                dst[j] = ok ? src[k] : 0.0f;
            }
        }
    }
}

as_status gather_f32_launch(as_ctx *ctx, long n, long n_src, const float *src, const int *idx,
                            float *dst, cudaStream_t s) {
    if (n == 0) return AS_OK;
    if (reinterpret_cast<uintptr_t>(idx) % 16 || reinterpret_cast<uintptr_t>(dst) % 16)
        return fail(AS_ERR_UNSUPPORTED, "gather_f32: idx and dst must be 16-byte aligned");
    long blocks = ceil_div(ceil_div(n, 4), kThreads);
    if (blocks > static_cast<long>(ctx->sms) * 16) blocks = static_cast<long>(ctx->sms) * 16;
    gather_f32<<<static_cast<unsigned>(blocks), kThreads, 0, s>>>(n, n_src, src, idx, dst,
                                                                  ctx->d_status);
    ctx->launches++;
    return check_cuda(cudaGetLastError(), "gather_f32 launch");
}

as_status f32_to_bf16_launch(as_ctx *ctx, long n, const float *src, uint16_t *dst,
                             cudaStream_t s) {
    long blocks = ceil_div(n, kThreads);
    if (blocks > 152L * 16) blocks = 152L * 16;
    f32_to_bf16_kernel<<<static_cast<unsigned>(blocks), kThreads, 0, s>>>(n, src, dst);
    ctx->launches++;
    return check_cuda(cudaGetLastError(), "f32_to_bf16 launch");
}

}  // namespace as

// ---- no-allocation transpose -----------------------------------------------------------------
// as_csr2csc_static: the same transpose with its scratch in a file-scope device array, for
// callers that cannot allocate device memory. The array is sized for
// AS_CSR2CSC_STATIC_MAX_NNZ entries; every GPU that loads this library holds it until the
// process exits. Host code only knows the array through the address cudaGetSymbolAddress
// returns for the current device (the symbol itself is a host-side stand-in), fetched once
// per device by the first call on that device and kept for the life of the process.
#include <mutex>

namespace as {
namespace {

constexpr size_t align256c(size_t b) { return (b + 255) & ~size_t(255); }
constexpr long kStaticTile = kSortThreads * kSmallItems;
static_assert(AS_CSR2CSC_STATIC_MAX_NNZ < kLargeNnz, "small tiles only");
constexpr long kStaticTiles = (AS_CSR2CSC_STATIC_MAX_NNZ + kStaticTile - 1) / kStaticTile;
constexpr long kStaticHist = kStaticTiles * kBins;
constexpr size_t kStaticScratchBytes =
    4 * align256c(sizeof(int) * static_cast<size_t>(AS_CSR2CSC_STATIC_MAX_NNZ)) +
    align256c(sizeof(int) * static_cast<size_t>(kStaticHist)) +
    align256c(sizeof(int) * static_cast<size_t>((kStaticHist + kScanChunk - 1) / kScanChunk + 1));
constexpr int kStaticMaxDevices = 64;

}  // namespace

static __device__ __align__(256) unsigned char g_csr2csc_static_scratch[kStaticScratchBytes];
static __device__ unsigned g_csr2csc_static_status;

namespace {

struct StaticSlot {
    bool ready = false;
    unsigned char *scratch = nullptr;
    unsigned *status = nullptr;
};
std::mutex g_static_mu;
StaticSlot g_static_slots[kStaticMaxDevices];

// Device addresses of the static scratch and status word on the current device.
cudaError_t static_slot(int dev, StaticSlot *out) {
    std::lock_guard<std::mutex> lock(g_static_mu);
    StaticSlot &s = g_static_slots[dev];
    if (!s.ready) {
        void *p = nullptr, *q = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_csr2csc_static_scratch);
        if (e != cudaSuccess) return e;
        e = cudaGetSymbolAddress(&q, g_csr2csc_static_status);
        if (e != cudaSuccess) return e;
        s.scratch = static_cast<unsigned char *>(p);
        s.status = static_cast<unsigned *>(q);
        s.ready = true;
    }
    *out = s;
    return cudaSuccess;
}

// The launch sequence of csr2csc_launch, reporting through cudaError_t only.
cudaError_t csr2csc_static_run(int M, int N, int nnz, const int *rowptr, const int *colind,
                               const float *val, int *colptr, int *rowind, float *cscval,
                               unsigned char *work, unsigned *status, cudaStream_t s) {
    const size_t cap = align256c(sizeof(int) * static_cast<size_t>(AS_CSR2CSC_STATIC_MAX_NNZ));
    SortBuffers w;
    w.keysA = reinterpret_cast<int *>(work);
    w.keysB = reinterpret_cast<int *>(work + cap);
    w.rowsT = reinterpret_cast<int *>(work + 2 * cap);
    w.valsT = reinterpret_cast<unsigned *>(work + 3 * cap);
    w.hist = reinterpret_cast<int *>(work + 4 * cap);
    w.sums = reinterpret_cast<int *>(work + 4 * cap + align256c(sizeof(int) * kStaticHist));
    (void)sort_by_column(M, N, nnz, rowptr, colind, reinterpret_cast<const unsigned *>(val), false,
                         colptr, rowind, val ? reinterpret_cast<unsigned *>(cscval) : nullptr, w,
                         status, s);
    return cudaGetLastError();
}

}  // namespace
}  // namespace as

extern "C" as_status as_csr2csc_static(int M, int N, int nnz, const int *rowptr,
                                       const int *colind, const float *val, int *colptr,
                                       int *rowind, float *cscval, void *stream) {
    using namespace as;
    if (M < 0 || N < 0 || nnz < 0) return AS_ERR_INVALID_VALUE;
    if (nnz > AS_CSR2CSC_STATIC_MAX_NNZ) return AS_ERR_UNSUPPORTED;
    if (!rowptr || !colptr || (nnz > 0 && (!colind || !rowind))) return AS_ERR_INVALID_VALUE;
    if ((val == nullptr) != (cscval == nullptr)) return AS_ERR_INVALID_VALUE;
    if (nnz > 0 && (M == 0 || N == 0)) return AS_ERR_INVALID_CSR;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return AS_ERR_CUDA;
    if (dev < 0 || dev >= kStaticMaxDevices) return AS_ERR_UNSUPPORTED;
    // a launch error left pending by earlier, unrelated work would otherwise be returned as this
    // call's: take it off first, so the status below belongs to this call's own launches
    (void)cudaGetLastError();
    StaticSlot slot;
    if (static_slot(dev, &slot) != cudaSuccess) return AS_ERR_CUDA;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // slot.status only gives the kernels a word to flag malformed input into; nothing reads it
    // (the entry point reports argument errors only), so it is not reset between calls
    if (nnz == 0) {
        return cudaMemsetAsync(colptr, 0, sizeof(int) * (static_cast<size_t>(N) + 1), s) ==
                       cudaSuccess
                   ? AS_OK
                   : AS_ERR_CUDA;
    }
    return csr2csc_static_run(M, N, nnz, rowptr, colind, val, colptr, rowind, cscval,
                              slot.scratch, slot.status, s) == cudaSuccess
               ? AS_OK
               : AS_ERR_CUDA;
}
