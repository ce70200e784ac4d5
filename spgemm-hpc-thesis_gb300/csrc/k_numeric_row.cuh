// K4 numeric phase: every output row sorted, summed and written without zeros.
//
// For a row with P products the kernel
//   1. enumerates the products in reference order (spg_enum.cuh): product t gets
//      its column, sequence number t and value __dmul_rn(a, b) (one rounding, as
//      `const double product = aValue * b` in spgemm_exchange.cpp:287);
//   2. sorts the products by column so that equal columns stay in product
//      order.  A warp row sorts one packed word (column - min) << s | sequence
//      number per product in registers (warp_sort); a CTA row distributes its
//      products over fine buckets (bucket_order), then every warp settles the
//      order inside the buckets of its share in registers (settle), again on
//      packed words.  Where the column range and the sequence number do not fit
//      32 bits: a stable LSD radix sort (warp rows), 64-bit words (CTA rows);
//      a CTA row that repeats a column often takes the radix sort too;
//   3. sums each run of equal columns sequentially in product order with
//      __dadd_rn, starting from its first product (the `emplace` then `+=` of
//      spgemm_exchange.cpp:288-293), and keeps the sums that are != 0.0
//      (spgemm_exchange.cpp:304; NaN and infinities are kept);
//   4. writes the kept (column, sum) pairs, already in column order, at the
//      row's output offset (job.cnt[row]) and the kept count into job.nz[row].
// Every coordinate is therefore bit-identical to the serial reference.  Rows of
// <= 512 products run one per warp (num_warp_kernel), rows of <= 8192 one per
// CTA with the keys in shared memory and the values in shared memory or a
// per-CTA global slab (num_block_kernel).  Heavier rows are split by column
// range into pieces that run on the same pipeline (num_piece_kernel) in the
// upper-bound layout, and in the exact layout where memory allows (else rows of
// <= 16384 run one per CTA with a value slab and heavier ones with the whole sort in
// a global slab, num_heavy_kernel, k_numeric.cu).  Many rows of <= 64 products run
// several per warp (num_rows_kernel, k_numeric_warp.cu).
#pragma once

#include <atomic>

#include <type_traits>

#include "spg_enum.cuh"
#include "spg_warp_sort.cuh"

namespace spg {
namespace {

template <int W>
__device__ inline void row_sync() {
    if (W == 1) __syncwarp();
    else __syncthreads();
}

constexpr int log2_ceil_c(int x) { return x <= 1 ? 0 : 1 + log2_ceil_c((x + 1) / 2); }

// Digit counters of W warps: counter (digit d, warp w) lives at hidx<W>(d, w),
// digit-major with an odd stride kHistStride >= W, so that the counters one
// warp's lanes touch for different digits fall in different banks (with stride
// W they would share 32 / W banks).
template <int W>
constexpr int kHistStride = W == 1 ? 1 : (W % 2 == 0 ? W + 1 : W + 2);
template <int W>
constexpr int kHistWords = 256 * kHistStride<W>;
template <int W>
__device__ __forceinline__ int hidx(int d, int w) {
    return W == 1 ? d : d * kHistStride<W> + w;
}

// Buckets of a CTA row (bucket_order below): coarse buckets (their table of one
// word each, then their counters) and at most one fine bucket per product (and
// one word past the last).
template <int W>
constexpr int kCoarseBits = W <= 4 ? 7 : 8;
template <int W>
constexpr int kCoarse = 1 << kCoarseBits<W>;
template <int W, int ITEMS>
constexpr int kBucketWords = W == 1 ? 4 : 2 * kCoarse<W> + W * 32 * ITEMS + 4;
// A warp finishes the sort of its share of a CTA row's positions, rounded to
// whole buckets, in registers: kShareItems per lane.  A fine bucket larger than
// the rounding allows sends the row to the radix sort.
// Against ranking every product inside its bucket by a loop over the bucket in
// shared memory, then moving it (65-75% of the sort's instructions, waiting on
// shared memory): rows of 1,025-1,536 products 0.44 -> 0.35 ms (16 uneven
// uniform products), of which settling the order takes 0.02 ms; power-law
// product, all bins 11.6 -> 9.3 ms with the other changes of this file.
template <int ITEMS>
constexpr int kShareItems = ITEMS + 2;
constexpr uint32_t kMaxFine = 32;

// A team's shared memory.  SV: product values in shared memory (else in a per-CTA global slab).
template <int W, int ITEMS, bool SV = true>
struct RowSmem {
    static constexpr int kCap = W * 32 * ITEMS;
    static constexpr int kSeqBits = log2_ceil_c(kCap);
    double vals[SV ? kCap : 1];  // product values by sequence number; run sums in place
    RowSegs<W * 32, W * 32 * ITEMS> seg;  // enumeration batch
    int64_t warp_tmp[W + 1];    // block scans
    alignas(16) uint32_t keys[kCap];  // columns (unpacked) or packed (column, sequence) words
    union {
        alignas(16) uint32_t hist[kHistWords<W>];  // digit counters of the radix sort at hidx<W>(digit, warp)
        alignas(16) uint32_t bk[kBucketWords<W, ITEMS>];  // bucket counters, then bucket starts (CTA rows)
    };
    uint32_t cnt[W * ITEMS];    // kept entries per (warp, item)
    uint16_t seqs[kCap];        // sequence numbers of the unpacked path
    int32_t red[2 * W];         // min / max column reduction
    uint32_t step_cnt[64];      // kept counts of one filtered enumeration step (row pieces)
};

// Exclusive scan of the NDIG*W digit counters in (digit, warp) order (logical
// index L = d * W + w): NDIG/32 consecutive counters per thread, one for the
// first 16*W threads when NDIG is 16.
template <int W, int NDIG = 256>
__device__ inline void scan_counters(uint32_t* c, int64_t* tmp) {
    constexpr int kPer = NDIG >= 32 ? NDIG / 32 : 1;
    constexpr int kTot = NDIG * W;
    const int lane = threadIdx.x & 31;
    const int warp = W == 1 ? 0 : (threadIdx.x >> 5);
    const int tid = W == 1 ? lane : threadIdx.x;
    const bool act = NDIG >= 32 || tid < kTot;
    auto phys = [](int L) { return W == 1 ? L : hidx<W>(L / W, L % W); };
    uint32_t v[kPer];
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        v[j] = act ? c[phys(tid * kPer + j)] : 0u;
        sum += v[j];
    }
    const uint32_t incl = warp_incl_scan(sum, lane);
    uint32_t base = incl - sum;
    if (W > 1) {  // every warp scans the W warp totals itself: one barrier
        if (lane == 31) tmp[warp] = incl;
        __syncthreads();
        const uint32_t t = lane < W ? static_cast<uint32_t>(tmp[lane]) : 0u;
        base += __shfl_sync(0xffffffffu, warp_incl_scan(t, lane) - t, warp);
    }
    if (act) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            c[phys(tid * kPer + j)] = base;
            base += v[j];
        }
    }
}

// Zeroes the counters of the first ndig digits (ndig * kHistStride<W> words, a
// multiple of four) with 16-byte stores; h is 16-byte aligned.
template <int W>
__device__ inline void clear_counters(uint32_t* h, int ndig, int tid) {
    uint4* h4 = reinterpret_cast<uint4*>(h);
    const int n4 = ndig * kHistStride<W> / 4;
    for (int d = tid; d < n4; d += W * 32) h4[d] = make_uint4(0u, 0u, 0u, 0u);
}

// Lanes of the warp holding the same NB-bit digit: the intersection of one
// ballot per digit bit (a ballot for each set bit, its complement for each
// clear bit).  Eight votes cost a fraction of one __match_any_sync on GB300.
template <int NB = 8>
__device__ inline unsigned digit_peers(uint32_t d) {
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const unsigned bit = (d >> b) & 1u;
        const unsigned set = __ballot_sync(0xffffffffu, bit);
        peers &= set ^ (bit - 1u);  // set where this lane's bit is 1, ~set where it is 0
    }
    return peers;
}

// Stable rank of one striped item against this warp's digit counters: the
// group of lanes holding the same digit (digit_peers); its first lane advances
// the counter by the group size (one shared atomic) and broadcasts the old
// value.  Items of a warp are ranked in order, so ranks follow
// (warp, item, lane) order.
template <int NB = 8>
__device__ inline uint32_t rank_item(uint32_t d, uint32_t* counter_of_d, int lane) {
    const unsigned peers = digit_peers<NB>(d);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter_of_d, static_cast<uint32_t>(__popc(peers)));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + __popc(peers & lanemask_lt());
}

// Exclusive scan of the W*ITEMS per-(warp, item) kept counts by warp 0; the
// total goes to red[0].
template <int W, int ITEMS>
__device__ inline void scan_kept(uint32_t* cnt, int32_t* red, int warp, int lane) {
    constexpr int kN = W * ITEMS;
    constexpr int kPer = (kN + 31) / 32;
    if (warp == 0) {
        uint32_t v[kPer];
        uint32_t tot = 0;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int idx = lane * kPer + j;
            v[j] = idx < kN ? cnt[idx] : 0u;
            tot += v[j];
        }
        const uint32_t incl = warp_incl_scan(tot, lane);
        uint32_t base = incl - tot;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int idx = lane * kPer + j;
            if (idx < kN) cnt[idx] = base;
            base += v[j];
        }
        if (lane == 31) red[0] = static_cast<int32_t>(incl);
    }
}

// Where a row's result goes, read once from the Job (locals, not reloaded
// through the Job reference after every global store).
struct RowOut {
    int32_t* __restrict__ c_col;
    double* __restrict__ c_val;
    int64_t out0;       // first slot of the row in C_tmp
    int64_t* nz;        // the row's stored-entry count
    int32_t holes;      // upper-bound mode: slot-per-position output with holes
};

// The sum of `all` over the warps before this one, and the team-wide maximum of m
// (red: 2*W words; one barrier).  red is next written after later barriers of the
// row, so no barrier protects it here.
template <int W>
__device__ inline uint32_t block_warps_before(uint32_t all, uint32_t m, int32_t* red, int lane, int warp, uint32_t& mx) {
    const uint32_t wm = __reduce_max_sync(0xffffffffu, m);
    if (lane == 31) {
        red[warp] = static_cast<int32_t>(all);
        red[W + warp] = static_cast<int32_t>(wm);
    }
    __syncthreads();
    uint32_t base = 0, gm = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        base += w < warp ? static_cast<uint32_t>(red[w]) : 0u;
        gm = max(gm, static_cast<uint32_t>(red[W + w]));
    }
    mx = gm;
    return base;
}

// Zeroes the counters of a CTA row of P products, which bucket_order expects to
// find cleared: after the row's enumeration, before the barrier of its column
// range.
template <int W, int ITEMS, bool SV>
__device__ __forceinline__ void clear_buckets(RowSmem<W, ITEMS, SV>& sm, int P, int tid) {
    uint4* b4 = reinterpret_cast<uint4*>(sm.bk + kCoarse<W>);  // coarse counters, fine counters 0 .. P
    const int n4 = (kCoarse<W> + P + 4) / 4;
    for (int i = tid; i < n4; i += W * 32) b4[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Orders a CTA row's products (columns at keys[0..P), sequence number =
// position, offsets k = column - cmin of nbits >= 1 bits) by fine bucket, in any
// order inside a bucket: seqs then holds their sequence numbers (the columns stay
// where they are), the fine counters hold the bucket starts.
//   * coarse buckets: the top bits of k;
//   * coarse bucket c of n_c products gets 2^fb_c fine buckets over its column
//     span, fb_c = min(span bits, floor(log2 n_c)), so that dense parts of the row
//     (the diagonal band of a banded product) get finer buckets than sparse ones:
//     one or two products per bucket on average;
//   * the fine histogram's atomics give every product its arrival index in its
//     bucket, so that it is placed without a second round of atomics.
// Instruction cost per product does not grow with the column range, unlike a
// digit pass.  The passes of these kernels over the shared-memory banks (74% of
// the time busy) bound them as much as the issue slots do.  With the table in one
// word per bucket instead of two, stored by vectors, and the scan's lanes side by
// side: rows of 1,537-2,048 products 0.49 -> 0.46 ms, of 1,025-1,536 0.348 -> 0.338
// (16 uneven uniform products), power-law product, all bins 8.94 -> 8.74.
// Returns the largest bucket's size; above kMaxFine seqs is not written.
template <int W, int ITEMS, bool SV>
__device__ __forceinline__ uint32_t bucket_order(RowSmem<W, ITEMS, SV>& sm, int P, uint32_t cmin, int nbits, int lane,
                                                 int warp, int tid, int& nfine) {
    constexpr int NT = W * 32;
    uint32_t* info = sm.bk;                         // first fine bucket | shift << 16
    uint32_t* cc = sm.bk + kCoarse<W>;              // coarse counters
    uint32_t* fc = sm.bk + 2 * kCoarse<W>;          // fine counters, then starts
    const int sc = max(nbits - kCoarseBits<W>, 0);  // column bits inside a coarse bucket
    const uint32_t inside = (1u << sc) - 1u;
    uint32_t f[ITEMS];
    // Position i * NT + tid: whole steps past P are skipped, and no warp is left
    // with less than its share when P is below the capacity.
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (i * NT >= P) break;
        const int pos = i * NT + tid;
        if (pos < P) atomicAdd(&cc[(sm.keys[pos] - cmin) >> sc], 1u);
    }
    __syncthreads();
    // every warp computes the whole table and stores it (the same words with the
    // same values), so that only a warp-level barrier precedes its use
    {
        constexpr int kPer = kCoarse<W> / 32;
        uint32_t n[kPer], bits[kPer], sum = 0;
#pragma unroll
        for (int j = 0; j < kPer; j += 4) *reinterpret_cast<uint4*>(n + j) = *reinterpret_cast<const uint4*>(cc + lane * kPer + j);
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            bits[j] = min(31u - __clz(n[j] | 1u), static_cast<uint32_t>(sc));
            n[j] = n[j] ? 1u << bits[j] : 0u;
            sum += n[j];
        }
        const uint32_t incl = warp_incl_scan(sum, lane);
        nfine = static_cast<int>(__shfl_sync(0xffffffffu, incl, 31));
        uint32_t base = incl - sum;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            bits[j] = base | (static_cast<uint32_t>(sc) - bits[j]) << 16;
            base += n[j];
        }
#pragma unroll
        for (int j = 0; j < kPer; j += 4)
            *reinterpret_cast<uint4*>(info + lane * kPer + j) = make_uint4(bits[j], bits[j + 1], bits[j + 2], bits[j + 3]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (i * NT >= P) break;
        if (i * NT + tid < P) {
            const uint32_t k = sm.keys[i * NT + tid] - cmin;
            const uint32_t in = info[k >> sc];
            f[i] = (in & 0xffffu) + ((k & inside) >> (in >> 16));
            f[i] |= atomicAdd(&fc[f[i]], 1u) << 16;  // arrival in the high half
        }
    }
    __syncthreads();
    // exclusive scan of the fine counters, a warp's 32 * ITEMS consecutive ones by
    // C chunks: lane l takes those from l * V of every chunk, so that its wide
    // accesses follow the other lanes' (ITEMS consecutive ones per lane meet in a
    // half or a quarter of the banks); two chunks share a scan
    uint32_t gmax;
    {
        constexpr int V = ITEMS % 8 == 0 ? 4 : ITEMS, C = ITEMS / V;
        constexpr int VL = V % 4 == 0 ? 4 : (V % 2 == 0 ? 2 : 1);  // words per access
        static_assert(C == 1 || C % 2 == 0, "two chunks share a scan");
        using Vec = std::conditional_t<VL == 4, uint4, std::conditional_t<VL == 2, uint2, uint32_t>>;
        const int w0 = warp * 32 * ITEMS + lane * V;
        uint32_t x[ITEMS], sum[C], mx = 0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            sum[c] = 0;
            if (w0 + c * 32 * V > nfine) continue;  // the bucket past the last is needed: its start is P
            uint32_t* xc = x + c * V;
#pragma unroll
            for (int j = 0; j < V; j += VL) *reinterpret_cast<Vec*>(xc + j) = *reinterpret_cast<const Vec*>(fc + w0 + c * 32 * V + j);
#pragma unroll
            for (int j = 0; j < V; ++j) {
                if (w0 + c * 32 * V + j >= nfine) xc[j] = 0u;  // not cleared past P
                sum[c] += xc[j];
                mx = max(mx, xc[j]);
            }
        }
        uint32_t at[C], all = 0;  // every chunk's products before the lane's; the warp's
        if constexpr (C == 1) {
            const uint32_t incl = warp_incl_scan(sum[0], lane);
            at[0] = incl - sum[0];
            all = __shfl_sync(0xffffffffu, incl, 31);
        } else {
#pragma unroll
            for (int c = 0; c < C; c += 2) {
                const uint32_t both = sum[c] | sum[c + 1] << 16;
                const uint32_t incl = warp_incl_scan(both, lane), tot = __shfl_sync(0xffffffffu, incl, 31);
                at[c] = all + ((incl - both) & 0xffffu);
                all += tot & 0xffffu;
                at[c + 1] = all + ((incl - both) >> 16);
                all += tot >> 16;
            }
        }
        const uint32_t before = block_warps_before<W>(all, mx, sm.red, lane, warp, gmax);
        if (gmax > kMaxFine) return gmax;  // uniform: every thread saw the same maximum
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (w0 + c * 32 * V > nfine) continue;
            uint32_t* xc = x + c * V;
            uint32_t base = before + at[c];
#pragma unroll
            for (int j = 0; j < V; ++j) {
                const uint32_t n = xc[j];
                xc[j] = base;
                base += n;
            }
#pragma unroll
            for (int j = 0; j < V; j += VL) *reinterpret_cast<Vec*>(fc + w0 + c * 32 * V + j) = *reinterpret_cast<const Vec*>(xc + j);
        }
        if (tid == 0 && nfine == W * 32 * ITEMS) fc[nfine] = static_cast<uint32_t>(P);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (i * NT >= P) break;
        const int pos = i * NT + tid;
        if (pos < P) {
            sm.seqs[fc[f[i] & 0xffffu] + (f[i] >> 16)] = static_cast<uint16_t>(pos);
        }
    }
    __syncthreads();
    return gmax;
}

// The warp's share of the positions [0, P): from the bucket that holds position
// warp * ceil(P / W) to the one that holds the next warp's first.  Bucket starts
// are monotone: each half of the warp narrows its bound 16-fold per step.
template <int W, int ITEMS, bool SV>
__device__ __forceinline__ void warp_share(const RowSmem<W, ITEMS, SV>& sm, int P, int nfine, int lane, int warp, int& x0,
                                           int& x1) {
    const uint32_t* fc = sm.bk + 2 * kCoarse<W>;
    const int share = (P + W - 1) / W;
    const int half = lane >> 4, l = lane & 15;
    const int m = (warp + half) * share;
    int lo = 0, n = 1;
    uint32_t v = 0;
    for (int range = nfine + 1; range > 1;) {
        const int stride = (range + 15) >> 4;
        const int i = lo + l * stride;
        v = i <= nfine ? fc[i] : 0xffffu;
        const unsigned below = __ballot_sync(0xffffffffu, static_cast<int>(v) <= m);
        n = __popc((below >> (half * 16)) & 0xffffu);
        lo += (n - 1) * stride;
        range = stride;
    }
    v = __shfl_sync(0xffffffffu, v, half * 16 + n - 1);
    const int x = m >= P ? P : static_cast<int>(v);
    x0 = __shfl_sync(0xffffffffu, x, 0);
    x1 = __shfl_sync(0xffffffffu, x, 16);
}

// Odd-even transposition of a warp's 32 * N keys (lane l holds keys l * N ... of
// the sequence, N even): `rounds` rounds sort a sequence whose keys are out of
// order only inside runs of at most `rounds` positions.
template <int N, typename K>
__device__ __forceinline__ void settle(K (&k)[N], int rounds, int lane) {
    static_assert(N % 2 == 0, "pairs keep their parity from lane to lane");
    for (int r = 0; r < rounds; r += 2) {
#pragma unroll
        for (int i = 0; i + 1 < N; i += 2) compare_exchange(k, i, i + 1);
        const K up = __shfl_down_sync(0xffffffffu, k[0], 1), down = __shfl_up_sync(0xffffffffu, k[N - 1], 1);
#pragma unroll
        for (int i = 1; i + 1 < N; i += 2) compare_exchange(k, i, i + 1);
        if (lane < 31) k[N - 1] = min(k[N - 1], up);
        if (lane > 0) k[0] = max(k[0], down);
    }
}

// Sorts a share whose (column, sequence) pairs do not fit 32 bits, at keys /
// seqs [0, n) in bucket order, as 64-bit keys.
template <int N>
__device__ __noinline__ void settle_wide(uint32_t* keys, uint16_t* seqs, int n, int rounds, int lane) {
    unsigned long long k[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int p = lane * N + i;
        k[i] = p < n ? (static_cast<unsigned long long>(keys[p]) << 16) | seqs[p] : ~0ull;
    }
    settle(k, rounds, lane);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int p = lane * N + i;
        if (p < n) {
            keys[p] = static_cast<uint32_t>(k[i] >> 16);
            seqs[p] = static_cast<uint16_t>(k[i]);
        }
    }
    __syncwarp();
}

// True unless v is +0.0 or -0.0 (NaN included), without the FP64 pipe, which
// takes 16 cycles for a warp's instruction.
__device__ __forceinline__ bool nonzero(double v) {
    return (static_cast<unsigned long long>(__double_as_longlong(v)) << 1) != 0ull;
}

// The stable LSD radix sort of a row's products by column: 8-bit digits over
// the bits of max(col) - min(col), and with kNarrow a last pass of at most 4
// bits (four votes, 16 counters per warp) when no more remain.  Leaves columns
// in keys and sequence numbers in seqs.
template <int W, int ITEMS, bool SV, bool kNarrow>
__device__ __forceinline__ void radix_sort_row(RowSmem<W, ITEMS, SV>& sm, int P, uint32_t cmin, int nbits, int lane,
                                               int warp, int tid) {
    auto digits_from = [&](int shift) { return (kNarrow && nbits - shift <= 4) ? 16 : 256; };
    for (int i = tid; i < P; i += W * 32) sm.seqs[i] = static_cast<uint16_t>(i);
    if (nbits > 0) clear_counters<W>(sm.hist, digits_from(0), tid);
    row_sync<W>();
    // One pass over the digit of NB bits at `shift` (NB = 8, or 4 for the last).
    auto pass = [&](auto nb, int shift) {
        constexpr int NB = decltype(nb)::value;
        constexpr uint32_t kMask = (1u << NB) - 1u;
        uint32_t* hist = sm.hist;
        uint32_t k[ITEMS], rk[ITEMS];
        uint16_t sq[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int pos = (warp * ITEMS + i) * 32 + lane;
            const bool valid = pos < P;
            k[i] = valid ? sm.keys[pos] : 0u;
            sq[i] = valid ? sm.seqs[pos] : uint16_t{0};
            const uint32_t d = valid ? (((k[i] - cmin) >> shift) & kMask) : kMask;
            rk[i] = rank_item<NB>(d, &hist[hidx<W>(d, warp)], lane);
        }
        row_sync<W>();
        scan_counters<W, (1 << NB)>(hist, sm.warp_tmp);
        row_sync<W>();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int pos = (warp * ITEMS + i) * 32 + lane;
            const uint32_t d = pos < P ? (((k[i] - cmin) >> shift) & kMask) : kMask;
            const uint32_t dst = hist[hidx<W>(d, warp)] + rk[i];
            if (dst < static_cast<uint32_t>(P)) {  // padding ranks last
                sm.keys[dst] = k[i];
                sm.seqs[dst] = sq[i];
            }
        }
    };
    for (int shift = 0; shift < nbits;) {
        if (!kNarrow || nbits - shift > 4) {
            pass(std::integral_constant<int, 8>{}, shift);
            shift += 8;
        } else {
            if constexpr (kNarrow) pass(std::integral_constant<int, 4>{}, shift);
            shift += 4;
        }
        row_sync<W>();  // the scatter above still reads the counters
        if (shift < nbits) clear_counters<W>(sm.hist, digits_from(shift), tid);
        row_sync<W>();
    }
}

constexpr uint32_t kDeadKey = 0xffffffffu;

// The words of a sorted region, lane l's at keys[l * N ...].  kWhole: the region has
// room for all 32 * N words and starts at 16 bytes, so that they go in the widest
// stores: one word at a time the lanes meet in a bank N-fold for N = 4, 8 and 16
// (rows of 385-512 products: 0.50 -> 0.45 ms, 65,536 rows of 256: 0.146 -> 0.140).
// A share of a CTA row has an even N twice an odd number: two lanes meet, and pairs
// of words, with the shares moved to even words, measured 2-7% slower.
template <int N, bool kWhole>
__device__ __forceinline__ void store_words(const uint32_t (&k)[N], uint32_t* keys, int n, int lane) {
    uint32_t* to = keys + lane * N;
    if constexpr (kWhole && N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4) *reinterpret_cast<uint4*>(to + i) = make_uint4(k[i], k[i + 1], k[i + 2], k[i + 3]);
    } else if constexpr (kWhole && N % 2 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 2) *reinterpret_cast<uint2*>(to + i) = make_uint2(k[i], k[i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (kWhole || lane * N + i < n) to[i] = k[i];
    }
}

// Step 3 of a sorted region of n positions, by one warp: lane l holds the words
// (column offset << S | sequence number) of positions l * N ... in k.  Stores
// them at keys[0..n), sums every run of equal column offsets in product order
// into the value of its first product, and turns the words of the run's other
// products into kDeadKey (no word's column offset is all ones).  The runs of
// more than one product are first listed (list: n 16-bit words), so that the
// warp sums 32 of them at a time: an FP64 instruction takes 16 cycles of an SM
// whether one lane needs it or all.
template <int N, int S, bool kWhole>
__device__ __forceinline__ void fold_runs(const uint32_t (&k)[N], uint32_t* keys, uint16_t* list, double* vals, int n,
                                          int lane) {
    using Mask = std::conditional_t<(N < 32), uint32_t, unsigned long long>;
    const uint32_t before = __shfl_up_sync(0xffffffffu, k[N - 1], 1);
    Mask same = 0;  // positions that continue a run
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint32_t p = i ? k[i - 1] : before;
        if (((k[i] ^ p) >> S) == 0u) same |= Mask{1} << i;
    }
    store_words<N, kWhole>(k, keys, n, lane);
    if (lane == 0) same &= ~Mask{1};
    const int mine = min(max(n - lane * N, 0), N);
    same &= (Mask{1} << mine) - 1;
    const uint32_t next = __shfl_down_sync(0xffffffffu, static_cast<uint32_t>(same), 1);
    Mask starts = ~same & ((same >> 1) | (lane < 31 ? static_cast<Mask>(next & 1u) << (N - 1) : Mask{0}));
    __syncwarp();
    if (!__any_sync(0xffffffffu, starts != 0)) return;
    const uint32_t count = N < 32 ? __popc(static_cast<uint32_t>(starts)) : __popcll(starts);
    const uint32_t incl = warp_incl_scan(count, lane);
    const uint32_t runs = __shfl_sync(0xffffffffu, incl, 31);
    for (uint32_t at = incl - count; starts; starts &= starts - 1) {
        const int i = (N < 32 ? __ffs(static_cast<uint32_t>(starts)) : __ffsll(static_cast<long long>(starts))) - 1;
        list[at++] = static_cast<uint16_t>(lane * N + i);
    }
    __syncwarp();
    constexpr uint32_t kSeq = (1u << S) - 1u;
    for (uint32_t j = lane; j < runs; j += 32) {
        int q = list[j];
        const uint32_t key = keys[q];
        double acc = vals[key & kSeq];
        for (++q; q < n; ++q) {
            const uint32_t other = keys[q];
            if ((other ^ key) >> S) break;
            acc = __dadd_rn(acc, vals[other & kSeq]);
            keys[q] = kDeadKey;
        }
        vals[key & kSeq] = acc;
    }
    __syncwarp();
}

// Upper-bound mode, step 4 of a region after fold_runs: position p owns slot p
// of [oc, ov); a run's first position writes (column, sum) when the sum is != 0,
// every other slot column -1.  A slot without an entry gets its value written
// all the same: a sector of DRAM written in part costs a read.  Returns the
// region's kept sums.
template <int S>
__device__ __forceinline__ uint32_t write_slots(const uint32_t* keys, const double* vals, int n, uint32_t first,
                                                int32_t* __restrict__ oc, double* __restrict__ ov, int lane) {
    constexpr int U = 4;
    uint32_t kept = 0;
    for (int p0 = lane; p0 - lane < n; p0 += 32 * U) {
        uint32_t key[U];
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int p = p0 + u * 32;
            key[u] = p < n ? keys[p] : kDeadKey;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = key[u] != kDeadKey ? vals[key[u] & ((1u << S) - 1u)] : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int p = p0 + u * 32;
            const bool keep = nonzero(v[u]);
            if (p < n) {
                oc[p] = keep ? static_cast<int32_t>((key[u] >> S) + first) : -1;
                ov[p] = v[u];
            }
            kept += __popc(__ballot_sync(0xffffffffu, keep));
        }
    }
    return kept;
}

// Exact layout, step 4 of a region after fold_runs: the kept sums of the region
// counted, or packed at [oc, ov).
template <int S>
__device__ __forceinline__ uint32_t count_kept(const uint32_t* keys, const double* vals, int n, int lane) {
    uint32_t kept = 0;
    for (int p0 = 0; p0 < n; p0 += 32) {
        const uint32_t key = p0 + lane < n ? keys[p0 + lane] : kDeadKey;
        kept += __popc(__ballot_sync(0xffffffffu, key != kDeadKey && nonzero(vals[key & ((1u << S) - 1u)])));
    }
    return kept;
}
template <int S>
__device__ __forceinline__ uint32_t write_kept(const uint32_t* keys, const double* vals, int n, uint32_t first,
                                               int32_t* __restrict__ oc, double* __restrict__ ov, int lane) {
    uint32_t kept = 0;
#pragma unroll 4
    for (int p0 = 0; p0 < n; p0 += 32) {
        const uint32_t key = p0 + lane < n ? keys[p0 + lane] : kDeadKey;
        const double v = key != kDeadKey ? vals[key & ((1u << S) - 1u)] : 0.0;
        const bool keep = nonzero(v);
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const uint32_t at = kept + __popc(m & lanemask_lt());
            oc[at] = static_cast<int32_t>((key >> S) + first);
            ov[at] = v;
        }
        kept += __popc(m);
    }
    return kept;
}

// The kept sums of a CTA row in the exact layout, every warp its share's after
// those of the warps before it.  Returns the row's kept sums.  (Out of line: the
// upper-bound layout's kernels ran 1-4% slower with it inline.)
template <int W, int S>
__device__ __noinline__ int32_t write_share(const uint32_t* keys, const double* vals, int n, uint32_t first, int32_t* oc,
                                            double* ov, int32_t* red, int lane, int warp) {
    const uint32_t kept = count_kept<S>(keys, vals, n, lane);
    if (lane == 0) red[warp] = static_cast<int32_t>(kept);
    __syncthreads();
    int at = 0, all = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const int32_t m = red[w];
        at += w < warp ? m : 0;
        all += m;
    }
    write_kept<S>(keys, vals, n, first, oc + at, ov + at, lane);
    return all;
}

// The sum of the products at positions [q, hi) of column c, after acc, in order, for
// rows that keep columns and sequence numbers apart; the columns ascend.  A run's adds
// follow one another, its loads need not: four at a time, rows of 2,500 products in
// one column take 1.42 ms (5,000 rows), of 10,000 in three columns 8.0; one at a time
// 2.70 and 14.4 (with the loop inlined in the row's code 2.50 and 13.2).
__device__ __forceinline__ double sum_run(const uint32_t* keys, const uint16_t* seqs, const double* vals, int q, int hi,
                                          uint32_t c, double acc) {
    constexpr int U = 4;
    for (; q + U <= hi && keys[q + U - 1] == c; q += U) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = vals[seqs[q + u]];
#pragma unroll
        for (int u = 0; u < U; ++u) acc = __dadd_rn(acc, v[u]);
    }
    for (; q < hi && keys[q] == c; ++q) acc = __dadd_rn(acc, vals[seqs[q]]);
    return acc;
}

// write_slots for the rows that keep columns and sequence numbers apart: slots
// [x0, x1) of a row whose runs may start or end anywhere in [lo, hi).  Returns
// the warp's kept sums.
__device__ __noinline__ uint32_t write_slots_plain(const uint32_t* keys, const uint16_t* seqs, const double* vals, int x0,
                                                   int x1, int lo, int hi, int32_t* oc, double* ov, int lane) {
    uint32_t kept = 0;
    for (int p = x0 + lane; p < x1; p += 32) {
        const uint32_t c = keys[p];
        double acc = 0.0;
        if (p == lo || keys[p - 1] != c) {
            acc = sum_run(keys, seqs, vals, p + 1, hi, c, vals[seqs[p]]);
        }
        const bool keep = nonzero(acc);
        oc[p] = keep ? static_cast<int32_t>(c) : -1;
        ov[p] = acc;
        kept += keep;
    }
    __syncwarp();
    return __reduce_add_sync(0xffffffffu, kept);
}

// The same in the exact layout, for a whole row by its team: steps 3 and 4.
// Returns the row's kept sums.
template <int W, int ITEMS, bool SV>
__device__ __forceinline__ uint32_t write_kept_plain(RowSmem<W, ITEMS, SV>& sm, double* vals, int P, int32_t* oc, double* ov,
                                                  int lane, int warp) {
    // runs of equal columns summed in product order; each run's sum is stored in
    // place of its first product's value
#pragma unroll 1
    for (int i = 0; i < ITEMS; ++i) {
        const int pos = (warp * ITEMS + i) * 32 + lane;
        bool keep = false;
        if (pos < P) {
            const uint32_t c = sm.keys[pos];
            if (pos == 0 || sm.keys[pos - 1] != c) {
                const uint32_t s0 = sm.seqs[pos];
                const double acc = sum_run(sm.keys, sm.seqs, vals, pos + 1, P, c, vals[s0]);
                vals[s0] = acc;
                keep = nonzero(acc);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) sm.cnt[warp * ITEMS + i] = __popc(m);
    }
    row_sync<W>();
    scan_kept<W, ITEMS>(sm.cnt, sm.red, warp, lane);
    row_sync<W>();
    // kept (column, sum) pairs in sorted order
#pragma unroll 1
    for (int i = 0; i < ITEMS; ++i) {
        const int pos = (warp * ITEMS + i) * 32 + lane;
        bool keep = false;
        uint32_t c = 0;
        double v = 0.0;
        if (pos < P) {
            c = sm.keys[pos];
            if (pos == 0 || sm.keys[pos - 1] != c) {
                v = vals[sm.seqs[pos]];
                keep = nonzero(v);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const int idx = static_cast<int>(sm.cnt[warp * ITEMS + i]) + __popc(m & lanemask_lt());
            oc[idx] = static_cast<int32_t>(c);
            ov[idx] = v;
        }
    }
    if constexpr (W == 1) __syncwarp();
    return static_cast<uint32_t>(sm.red[0]);
}

// The radix sort of the CTA rows with a large bucket (a column repeated more
// than kMaxFine times).  Out of line: inlined, the kernels of 64 registers spill more
// (4x12 378 / 286 bytes of stores / loads against 192 / 180, 8x12 338 / 266 against
// 192 / 180).  They still spill: what the row keeps across the calls of paths that it
// seldom takes lies in local memory (1.8 M loads and 2.3 M stores in 183 M warp
// instructions of the 4x12 kernel; 0.36 and 0.43 M in the kernel before it).
template <int W, int ITEMS, bool SV>
__device__ __noinline__ void radix_sort_cta(RowSmem<W, ITEMS, SV>& sm, int P, uint32_t cmin, int nbits, int lane, int warp,
                                            int tid) {
    radix_sort_row<W, ITEMS, SV, false>(sm, P, cmin, nbits, lane, warp, tid);
}

// Steps 2-4 of a row for one key layout (PACKED: (col - cmin) << kSeqBits | seq
// words, warp rows only; otherwise columns and 16-bit sequence numbers).
// Returns the stored entries this thread accounts for (its warp's on lane 0 in
// upper-bound mode, the row's on thread 0 in exact mode, else 0).  No barrier
// ends the row: the next row's enumeration passes a barrier before it writes
// what this phase reads (keys, values, sequence numbers, bucket starts, kept
// counts).
template <int W, int ITEMS, bool SV, bool PACKED>
__device__ __forceinline__ uint32_t finish_row(const RowOut& out, RowSmem<W, ITEMS, SV>& sm, double* vals, int P,
                                               uint32_t cmin, uint32_t range, int nbits, int lane, int warp, int tid) {
    using Sm = RowSmem<W, ITEMS, SV>;
    constexpr int kSeqBits = Sm::kSeqBits;
    constexpr uint32_t kMaxRange = 0xffffffffu >> kSeqBits;  // below it no packed word is kDeadKey
    // 2. sort by column: warp rows in registers (the padding words above P sort
    //    last: a real word is all ones only when P is the row's capacity), CTA
    //    rows by bucket and then, inside the buckets, in registers, and by the
    //    radix sort where a bucket is large.  Warp rows, against the radix sort of
    //    rows of <= 192 products and the bucket sort of 193-512 (power-law product,
    //    one bin at a time): <= 512 products 0.95 -> 0.49 ms, <= 384 0.79 -> 0.50,
    //    <= 256 0.35 -> 0.23, <= 192 0.37 -> 0.25, <= 128 0.145 -> 0.094; 65,536 rows
    //    of 256: 0.190 -> 0.147 ms.  Issue slots bound these kernels, and the network
    //    takes about half the instructions of either sort (about 90 a key), none of
    //    them waiting on shared memory.
    uint32_t kept = 0;
    if constexpr (W == 1 && PACKED) {
        uint32_t k[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int pos = i * 32 + lane;
            k[i] = pos < P ? ((sm.keys[pos] - cmin) << kSeqBits) | static_cast<uint32_t>(pos) : 0xffffffffu;
        }
        warp_sort(k, lane);
        __syncwarp();
        fold_runs<ITEMS, kSeqBits, true>(k, sm.keys, sm.seqs, vals, P, lane);
        int32_t* oc = out.c_col + out.out0;
        double* ov = out.c_val + out.out0;
        kept = out.holes ? write_slots<kSeqBits>(sm.keys, vals, P, cmin, oc, ov, lane)
                         : write_kept<kSeqBits>(sm.keys, vals, P, cmin, oc, ov, lane);
        __syncwarp();
        if (lane == 0) *out.nz = kept;
        return lane == 0 ? kept : 0u;
    } else if constexpr (W == 1) {
        radix_sort_row<W, ITEMS, SV, true>(sm, P, cmin, nbits, lane, warp, tid);
    } else {
        constexpr int N = kShareItems<ITEMS>;
        int x0 = warp * ((P + W - 1) / W), x1 = x0 + (P + W - 1) / W, nfine = 0;
        bool by_share = false, written = false;
        if (nbits == 0) {
            for (int i = tid; i < P; i += W * 32) sm.seqs[i] = static_cast<uint16_t>(i);
            __syncthreads();
        } else {
            const uint32_t biggest = bucket_order(sm, P, cmin, nbits, lane, warp, tid, nfine);
            if (biggest > kMaxFine) {
                radix_sort_cta(sm, P, cmin, nbits, lane, warp, tid);
            } else {
                // Every warp settles the order inside the buckets of its share:
                // from here on the warps work without a barrier.
                by_share = true;
                warp_share(sm, P, nfine, lane, warp, x0, x1);
                const int n = x1 - x0;
                uint32_t* keys = sm.keys + x0;
                uint16_t* seqs = sm.seqs + x0;
                // column offsets from `first`: the row's smallest column where the row's
                // range and sequence numbers fit 32 bits, else the share's
                uint32_t first = cmin;
                bool wide = false;
                if (range >= kMaxRange) {
                    uint32_t lo = 0xffffffffu, hi = 0;
                    for (int p = lane; p < n; p += 32) {
                        const uint32_t c = sm.keys[seqs[p]];
                        lo = min(lo, c);
                        hi = max(hi, c);
                    }
                    first = __reduce_min_sync(0xffffffffu, lo);
                    hi = __reduce_max_sync(0xffffffffu, hi);
                    wide = n > 0 && hi - first >= kMaxRange;
                }
                uint32_t k[N];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const int p = lane * N + i;
                    k[i] = kDeadKey;
                    if (p < n) {
                        const uint32_t s = seqs[p];
                        k[i] = wide ? sm.keys[s] : ((sm.keys[s] - first) << kSeqBits) | s;
                    }
                }
                __syncthreads();  // every warp has read its columns: keys is free
                if (wide) {
#pragma unroll
                    for (int i = 0; i < N; ++i)
                        if (lane * N + i < n) keys[lane * N + i] = k[i];
                    __syncwarp();
                    settle_wide<N>(keys, seqs, n, static_cast<int>(biggest), lane);
                } else {
                    settle(k, static_cast<int>(biggest), lane);
                    if (out.holes || range < kMaxRange) {  // exact layout: no warp of the row is wide
                        fold_runs<N, kSeqBits, false>(k, keys, seqs, vals, n, lane);
                        if (!out.holes) {
                            const int32_t all = write_share<W, kSeqBits>(keys, vals, n, first, out.c_col + out.out0,
                                                                         out.c_val + out.out0, sm.red, lane, warp);
                            if (tid == 0) *out.nz = all;
                            return tid == 0 ? static_cast<uint32_t>(all) : 0u;
                        }
                        kept = write_slots<kSeqBits>(keys, vals, n, first, out.c_col + out.out0 + x0,
                                                     out.c_val + out.out0 + x0, lane);
                        written = true;
                    } else {
#pragma unroll
                        for (int i = 0; i < N; ++i) {
                            const int p = lane * N + i;
                            if (p < n) {
                                keys[p] = (k[i] >> kSeqBits) + first;
                                seqs[p] = static_cast<uint16_t>(k[i] & ((1u << kSeqBits) - 1u));
                            }
                        }
                    }
                }
                if (!out.holes) __syncthreads();
            }
        }
        if (out.holes) {
            x0 = min(x0, P);
            x1 = min(x1, P);
            if (!written)  // shares cut anywhere unless they are whole buckets: runs may cross them
                kept = write_slots_plain(sm.keys, sm.seqs, vals, x0, x1, by_share ? x0 : 0, by_share ? x1 : P,
                                         out.c_col + out.out0, out.c_val + out.out0, lane);
            if (lane == 0 && kept)  // the row's count was zeroed before its enumeration
                atomicAdd(reinterpret_cast<unsigned long long*>(out.nz), static_cast<unsigned long long>(kept));
            return lane == 0 ? kept : 0u;
        }
    }

    if constexpr (W == 1) {
        if (out.holes) {
            kept = write_slots_plain(sm.keys, sm.seqs, vals, 0, P, 0, P, out.c_col + out.out0, out.c_val + out.out0, lane);
            if (lane == 0) *out.nz = kept;
            return lane == 0 ? kept : 0u;
        }
    }
    kept = write_kept_plain(sm, vals, P, out.c_col + out.out0, out.c_val + out.out0, lane, warp);
    if (tid == 0) *out.nz = kept;
    return tid == 0 ? kept : 0u;
}


// A column range of a split row: the products with columns in [lo, hi), which
// own slots [slot_off, slot_off + count) of the row's reserved range.  The
// row's products are staged in product order at scol / sval.
struct Piece {
    int64_t item;
    int32_t lo, hi;
    int64_t slot_off;
    int64_t count;
    const int32_t* scol;
    const double* sval;
};

// One row (PIECE = false) or one column range of a row (PIECE = true, CTA
// rows in upper-bound mode only).  Returns the stored entries this thread
// accounts for (finish_row).
template <int W, int ITEMS, bool SV, bool PIECE = false>
__device__ uint32_t numeric_row(const Job& J, int row, RowSmem<W, ITEMS, SV>& sm, double* vals, ErrWord* err,
                            const Piece* pc = nullptr) {
    using Sm = RowSmem<W, ITEMS, SV>;
    constexpr int kSeqBits = Sm::kSeqBits;
    const int lane = threadIdx.x & 31;
    const int warp = W == 1 ? 0 : (threadIdx.x >> 5);
    const int tid = W == 1 ? lane : threadIdx.x;
    const int P = static_cast<int>(PIECE ? pc->count : J.ub[row]);
    if constexpr (W > 1) {
        // an upper-bound row's warps add their kept counts to its count after the
        // barriers below (a piece's row count was zeroed by the row work, or in a plan's replay)
        if (!PIECE && J.holes && tid == 0) J.nz[row] = 0;
    }

    // 1. products into shared memory
    int32_t lo = INT32_MAX, hi = INT32_MIN;
    const int32_t ncols = J.B.cols;
    auto put = [&](int32_t seq, int32_t c, double prod) {
        if (PIECE && seq >= P) {  // the planner counted fewer products in this range: never writes past P
            raise_error(err, kErrInvalid, 8, seq);
            return;
        }
        if (c < 0 || c >= ncols) {
            raise_error(err, kErrInvalid, 4, c);
            c = 0;
        }
        sm.keys[seq] = static_cast<uint32_t>(c);
        vals[seq] = prod;
        lo = min(lo, c);
        hi = max(hi, c);
    };
    if constexpr (PIECE)
        staged_products_in<W * 32>(pc->scol, pc->sval, static_cast<int32_t>(J.ub[row]), sm.step_cnt, tid, pc->lo,
                                   pc->hi, put);
    else
        team_row_products<W * 32, Sm::kCap>(J, row, sm.seg, sm.warp_tmp, tid,
                                            [&](int32_t seq, int32_t c, double b, double a) {
                                                put(seq, c, __dmul_rn(a, b));
                                            });
    // (the enumeration's barriers come after every warp's last use of the starts)
    if constexpr (W > 1) clear_buckets(sm, P, tid);
    lo = __reduce_min_sync(0xffffffffu, lo);  // one warp-wide reduction instruction each
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (W > 1) {
        if (lane == 0) {
            sm.red[warp] = lo;
            sm.red[W + warp] = hi;
        }
        __syncthreads();
        lo = sm.red[0];
        hi = sm.red[W];
#pragma unroll
        for (int w = 1; w < W; ++w) {
            lo = min(lo, sm.red[w]);
            hi = max(hi, sm.red[W + w]);
        }
    } else {
        __syncwarp();  // the enumeration's last batch ends without one
    }
    const uint32_t cmin = static_cast<uint32_t>(lo);
    const uint32_t range = P ? static_cast<uint32_t>(hi - lo) : 0u;
    const int nbits = range ? 32 - __clz(range) : 0;
    const RowOut out{J.c_col, J.c_val, J.cnt[row] + (PIECE ? pc->slot_off : 0), J.nz + row, J.holes};
    if constexpr (W == 1)
        if (range < (0xffffffffu >> kSeqBits)) return finish_row<W, ITEMS, SV, true>(out, sm, vals, P, cmin, range, nbits, lane, warp, tid);
    return finish_row<W, ITEMS, SV, false>(out, sm, vals, P, cmin, range, nbits, lane, warp, tid);
}

constexpr int kWarpKernelThreads = 256;

// Resident CTAs per SM the warp-row kernels are compiled for (caps registers
// at 128, 80 and 64 per thread).  Measured on power-law rows, one bin at a
// time, against one CTA more: 8 items 0.256 -> 0.228 ms, 6 items 0.263 ->
// 0.252, 12 and 16 items 0.49 -> 0.50 (but the concurrent phase 4% shorter).
constexpr int warp_kernel_min_blocks(int items) { return items >= 12 ? 2 : (items >= 6 ? 3 : 4); }

// The row kernels are persistent: a launch has at most a few waves of CTAs
// that loop over the bin's rows.  A warp-row kernel takes its rows by a fixed
// stride: its rows are many and light, and a ticket per row measured 4% slower
// on the uniform product (one counter for hundreds of thousands of rows).
template <int ITEMS>
__global__ void __launch_bounds__(kWarpKernelThreads, warp_kernel_min_blocks(ITEMS))
num_warp_kernel(const Job* __restrict__ jobs, const int64_t* __restrict__ items, int64_t count,
                Stats* __restrict__ stats, ErrWord* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Sm = RowSmem<1, ITEMS>;
    Sm& sm = reinterpret_cast<Sm*>(smem_raw)[threadIdx.x >> 5];
    __shared__ unsigned long long s_nz;
    if (threadIdx.x == 0) s_nz = 0;
    __syncthreads();
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (kWarpKernelThreads / 32);
    unsigned long long mine = 0;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * (kWarpKernelThreads / 32) + (threadIdx.x >> 5); i < count;
         i += warps) {
        const int64_t it = items[i];
        const Job& J = jobs[item_job(it)];
        const int row = item_row(it);
        mine += numeric_row<1, ITEMS, true>(J, row, sm, sm.vals, err);
    }
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&s_nz, mine);
    __syncthreads();
    if (threadIdx.x == 0 && s_nz) atomicAdd(&stats->nz_total, s_nz);
}

// A CTA-row kernel (and the split rows' pieces) pulls its rows from the
// launch's row queue: the CTA's first row is its index, each later one
// gridDim.x plus the next ticket of the bin's counter, so that rows of very
// different cost spread over the CTAs as they free up.  Thread 0 fetches the
// ticket at the start of the current row (the other warps start on the row
// meanwhile; fetching it a row ahead instead, in a register, measured slower)
// into one of two shared words (alternating rows); every thread reads it after
// the row, whose barriers order the store before the reads, and every read
// before the store two rows later.
struct RowQueue {
    int64_t next[2];
};

template <int W, int ITEMS, int MINB, bool SV>
__global__ void __launch_bounds__(W * 32, MINB)
num_block_kernel(const Job* __restrict__ jobs, const int64_t* __restrict__ items, int64_t count,
                 Stats* __restrict__ stats, ErrWord* __restrict__ err, double* __restrict__ gvals,
                 unsigned long long* __restrict__ ticket) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RowQueue q;
    using Sm = RowSmem<W, ITEMS, SV>;
    Sm& sm = *reinterpret_cast<Sm*>(smem_raw);
    double* vals = SV ? sm.vals : gvals + static_cast<size_t>(blockIdx.x) * Sm::kCap;
    unsigned long long mine = 0;
    int par = 0;
    for (int64_t i = blockIdx.x; i < count; par ^= 1) {
        if (threadIdx.x == 0)
            q.next[par] = static_cast<int64_t>(gridDim.x) + static_cast<int64_t>(atomicAdd(ticket, 1ull));
        const int64_t it = items[i];
        const Job& J = jobs[item_job(it)];
        const int row = item_row(it);
        mine += numeric_row<W, ITEMS, SV>(J, row, sm, vals, err);
        i = q.next[par];
    }
    if (mine) atomicAdd(&stats->nz_total, mine);
}

inline int capped(int64_t work, int per_block, int cap) {
    const int64_t g = (work + per_block - 1) / per_block;
    return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

// CTAs of a launch whose CTAs each own a global slab: minb per SM at most.
inline int slab_grid(int64_t count, int num_sms, int minb = 1) {
    const int64_t cap = static_cast<int64_t>(num_sms) * minb;
    return static_cast<int>(count < cap ? count : cap);
}

template <int ITEMS>
void run_warp(const Job* jobs, const int64_t* items, int64_t count, Stats* stats, ErrWord* err, cudaStream_t st,
              int num_sms) {
    const int smem = 8 * static_cast<int>(sizeof(RowSmem<1, ITEMS>));
    allow_smem<num_warp_kernel<ITEMS>>(smem);
    num_warp_kernel<ITEMS><<<capped(count, 8, num_sms * 16), kWarpKernelThreads, smem, st>>>(jobs, items, count, stats,
                                                                                           err);
}

template <int W, int ITEMS, int MINB, bool SV = true>
void run_block(const Job* jobs, const int64_t* items, int64_t count, Stats* stats, ErrWord* err, cudaStream_t st,
               int num_sms, unsigned long long* ticket, double* gvals = nullptr) {
    const int smem = static_cast<int>(sizeof(RowSmem<W, ITEMS, SV>));
    allow_smem<num_block_kernel<W, ITEMS, MINB, SV>>(smem);
    // One wave of resident CTAs: with the row queue, CTAs beyond it would start
    // only once the queue has run dry (slab bins: one slab per resident CTA).
    static std::atomic<int> resident{0};  // per instantiation (every device of this build is an sm_103a)
    int nb = resident.load(std::memory_order_relaxed);
    if (nb == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, num_block_kernel<W, ITEMS, MINB, SV>, W * 32, smem) !=
                cudaSuccess || nb < 1) {
            cudaGetLastError();
            nb = MINB;
        }
        resident.store(nb, std::memory_order_relaxed);
    }
    const int grid = SV ? capped(count, 1, num_sms * nb) : slab_grid(count, num_sms, MINB);
    num_block_kernel<W, ITEMS, MINB, SV><<<grid, W * 32, smem, st>>>(jobs, items, count, stats, err, gvals, ticket);
}

}  // namespace
}  // namespace spg
