// K4 numeric phase: the row bins that run one row per warp (<= 512 products;
// 1, 2, 3, 4, 6, 8, 12 or 16 products per lane).  The per-row pipeline of rows
// of more than 128 products is in k_numeric_row.cuh; shorter rows run several
// to a warp (num_rows_kernel).
#include "k_numeric_row.cuh"

namespace spg {
namespace {

// One warp's state for G rows of at most 32 * I products.
template <int I, int G>
struct RowsSmem {
    static constexpr int kRow = 32 * I;
    static constexpr int kAll = G * kRow;
    double vals[kAll];      // product values: row g at g * kRow, by sequence number
    uint32_t keys[kAll];    // columns by sequence number, then sorted words
    uint64_t colb[32], valb[32];  // segments (RowSegs)
    double scale[32];
    int32_t delta[32];      // place of a segment's product less its position among the rows' products
    uint2 word[G * I];
    uint16_t list[kAll];
};

// A row whose columns and sequence numbers do not fit 32-bit words: sorted as
// 64-bit words, columns and sequence numbers into cols / seqs, then summed and
// written.  Returns the kept sums.
template <int I>
__device__ __noinline__ uint32_t finish_wide_row(uint32_t* cols, uint16_t* seqs, const double* vals, int P, int32_t* oc,
                                                 double* ov, bool holes, int lane) {
    unsigned long long k[I];
#pragma unroll
    for (int i = 0; i < I; ++i) {
        const int p = i * 32 + lane;
        k[i] = p < P ? (static_cast<unsigned long long>(cols[p]) << 16) | static_cast<unsigned>(p) : ~0ull;
    }
    warp_sort(k, lane);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < I; ++i) {
        const int p = lane * I + i;
        if (p < P) {
            cols[p] = static_cast<uint32_t>(k[i] >> 16);
            seqs[p] = static_cast<uint16_t>(k[i]);
        }
    }
    __syncwarp();
    uint32_t kept = 0;
    for (int p0 = 0; p0 < P; p0 += 32) {
        const int p = p0 + lane;
        double acc = 0.0;
        uint32_t c = 0;
        if (p < P) {
            c = cols[p];
            if (p == 0 || cols[p - 1] != c) {
                acc = vals[seqs[p]];
                for (int q = p + 1; q < P && cols[q] == c; ++q) acc = __dadd_rn(acc, vals[seqs[q]]);
            }
        }
        const bool keep = nonzero(acc);
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        const int at = holes ? p : static_cast<int>(kept) + __popc(m & lanemask_lt());
        if (holes ? p < P : keep) {
            oc[at] = keep ? static_cast<int32_t>(c) : -1;
            ov[at] = acc;
        }
        kept += __popc(m);
    }
    __syncwarp();
    return kept;
}

template <typename T>
__device__ __forceinline__ T* shfl_ptr(T* p, int lane) {
    return reinterpret_cast<T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), lane));
}

// G rows of at most 32 * I products per warp.  A row this short leaves a warp
// that works on it alone waiting: five dependent loads (work item, offsets of A,
// A entry, offsets of B, B entry) for some ten instructions per product.  Here
// the rows' segments share the lanes of one enumeration and the rows' sorts, one
// register (or I) per row, are independent chains.  The passes over the L1 banks
// bound it then (80-88% of the time busy: B's offsets, columns and values lie in
// lines of their own for every segment, the shuffles and shared memory take the
// rest), so a row's first segment, result pointers and run marks stay in the lane
// that has them: 262,144 rows of 32 products 0.205 -> 0.189 ms, of 56 products
// 0.163 -> 0.159, against every lane holding all rows' segments and reading the
// job again per row.  When: launch_numeric_warp.
template <int I, int G>
__global__ void __launch_bounds__(kWarpKernelThreads, 4)
num_rows_kernel(const Job* __restrict__ jobs, const int64_t* __restrict__ items, int64_t count,
                Stats* __restrict__ stats, ErrWord* __restrict__ err) {
    using Sm = RowsSmem<I, G>;
    constexpr int S = log2_ceil_c(Sm::kRow);
    constexpr uint32_t kMaxRange = 0xffffffffu >> S;  // below it no packed word is kDeadKey
    constexpr uint32_t kSeq = (1u << S) - 1u;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Sm& sm = reinterpret_cast<Sm*>(smem_raw)[threadIdx.x >> 5];
    __shared__ unsigned long long s_nz;
    if (threadIdx.x == 0) s_nz = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const unsigned le_above0 = (lanemask_lt() | (1u << lane)) & ~1u;  // bits (0, lane]
    const int64_t stride = static_cast<int64_t>(gridDim.x) * (kWarpKernelThreads / 32) * G;
    unsigned long long mine = 0;
    for (int64_t i0 = (static_cast<int64_t>(blockIdx.x) * (kWarpKernelThreads / 32) + (threadIdx.x >> 5)) * G; i0 < count;
         i0 += stride) {
        // lane g: row g
        const Job* J = jobs;
        int row = 0, P = 0;
        int64_t a0 = 0, nseg = 0;
        int32_t* out_col = nullptr;
        double* out_val = nullptr;
        uint32_t ncols = 0;
        bool slots = false;  // upper-bound layout
        if (lane < G && i0 + lane < count) {
            const int64_t it = items[i0 + lane];
            J = jobs + item_job(it);
            row = item_row(it);
            P = static_cast<int>(J->ub[row]);
            a0 = J->A.rp[row];
            nseg = J->A.rp[row + 1] - a0 + (J->S.rp ? 1 : 0);
            const int64_t out0 = J->cnt[row];
            out_col = J->c_col + out0;
            out_val = J->c_val + out0;
            ncols = static_cast<uint32_t>(J->B.cols);
            slots = J->holes != 0;
        }
        int p_incl = P;
        int64_t s_incl = nseg;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const int p = __shfl_up_sync(0xffffffffu, p_incl, o);
            const int64_t s = __shfl_up_sync(0xffffffffu, s_incl, o);
            if (lane >= o) {
                p_incl += p;
                s_incl += s;
            }
        }
        const int64_t all_seg = __shfl_sync(0xffffffffu, s_incl, G - 1);
        const int64_t seg0 = s_incl - nseg;  // the row's first segment
        const unsigned slot_rows = __ballot_sync(0xffffffffu, slots);
        const int row_delta = lane * Sm::kRow - (p_incl - P);

        // 1. the rows' products into shared memory (team_row_products for G rows)
        int done = 0;
        for (int64_t e0 = 0; e0 < all_seg; e0 += 32) {
            const int64_t e = e0 + lane;
            // the rows that start before the batch, and in it up to this segment (a
            // row of the list has a segment: the last of them is the segment's)
            const int64_t in_batch = seg0 - e0;
            const unsigned starts_here =
                __reduce_or_sync(0xffffffffu, nseg > 0 && in_batch >= 0 && in_batch < 32 ? 1u << in_batch : 0u);
            const int earlier = __popc(__ballot_sync(0xffffffffu, nseg > 0 && in_batch < 0));
            const int g = earlier + __popc(starts_here & (le_above0 | 1u)) - 1;
            const int64_t first = __shfl_sync(0xffffffffu, seg0, g);
            const Job* Jg = reinterpret_cast<const Job*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(J), g));
            const int row_g = __shfl_sync(0xffffffffu, row, g);
            const int64_t a0_g = __shfl_sync(0xffffffffu, a0, g);
            const int delta_g = __shfl_sync(0xffffffffu, row_delta, g);
            const int32_t* cp = nullptr;
            const double* vp = nullptr;
            double sc = 1.0;
            int32_t len = 0;
            if (e < all_seg) row_segment(*Jg, row_g, a0_g, Jg->S.rp != nullptr, e - first, cp, vp, sc, len);
            // low 16 bits: products; high 16 bits: non-empty segments
            const uint32_t incl = warp_incl_scan(static_cast<uint32_t>(len) | (len > 0 ? 0x10000u : 0u), lane);
            const int total = static_cast<int>(__shfl_sync(0xffffffffu, incl, 31) & 0xffffu);
            const uint32_t s = (incl & 0xffffu) - static_cast<uint32_t>(len);
            // B's rows hold one entry (an aggregation's prolongation): every lane has
            // its product, without the table (262,144 rows of 32 products: 0.189 ->
            // 0.156 ms)
            if (__all_sync(0xffffffffu, len <= 1)) {
                if (len > 0) {
                    const int at = static_cast<int>(s) + delta_g + done;
                    sm.keys[at] = static_cast<uint32_t>(__ldg(cp));
                    sm.vals[at] = __dmul_rn(sc, __ldg(vp));
                }
                done += total;
                __syncwarp();
                continue;
            }
            if (len > 0) {
                const uint32_t r = (incl >> 16) - 1u;
                sm.colb[r] = reinterpret_cast<uint64_t>(cp) - 4u * static_cast<uint64_t>(s);
                sm.valb[r] = reinterpret_cast<uint64_t>(vp) - 8u * static_cast<uint64_t>(s);
                sm.scale[r] = sc;
                sm.delta[r] = delta_g + done;
            }
            // the start mask, one reduction per word (segments of one product would
            // all aim an atomic at one word), and every word's rank from the starts
            // before it
            uint32_t starts_w = 0;
            for (int w = 0; w * 32 < total; ++w) {
                const uint32_t m = __reduce_or_sync(0xffffffffu, len > 0 && static_cast<int>(s >> 5) == w ? 1u << (s & 31u) : 0u);
                if (lane == w) starts_w = m;
            }
            const uint32_t n_w = __popc(starts_w);
            uint32_t rank = n_w;
#pragma unroll
            for (int o = 1; o < G * I; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, rank, o);
                if (lane >= o) rank += t;
            }
            if (lane < G * I) sm.word[lane] = make_uint2(starts_w, rank - n_w - 1u + (starts_w & 1u));
            __syncwarp();
            constexpr int U = 4;
            for (int t0 = lane; t0 < total; t0 += 32 * U) {
                int r[U];
                int32_t c[U];
                double b[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int t = t0 + u * 32;
                    r[u] = 0;
                    if (t < total) {
                        const uint2 wd = sm.word[t >> 5];
                        r[u] = static_cast<int>(wd.y) + __popc(wd.x & le_above0);
                        c[u] = __ldg(reinterpret_cast<const int32_t*>(sm.colb[r[u]] + 4u * static_cast<uint64_t>(t)));
                        b[u] = __ldg(reinterpret_cast<const double*>(sm.valb[r[u]] + 8u * static_cast<uint64_t>(t)));
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int t = t0 + u * 32;
                    if (t < total) {
                        const int at = t + sm.delta[r[u]];
                        sm.keys[at] = static_cast<uint32_t>(c[u]);
                        sm.vals[at] = __dmul_rn(sm.scale[r[u]], b[u]);
                    }
                }
            }
            done += total;
            __syncwarp();  // the next batch rewrites the table
        }

        // 2. words of every row, sorted
        uint32_t k[G * I];
        uint32_t cmin = 0;  // lane g: row g's smallest column
        uint32_t kept = 0;  // lane g: row g's stored entries
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int Pg = __shfl_sync(0xffffffffu, P, g);
            const uint32_t ncols_g = __shfl_sync(0xffffffffu, ncols, g);
            uint32_t lo = 0xffffffffu, hi = 0;
#pragma unroll
            for (int i = 0; i < I; ++i) {
                const int p = i * 32 + lane;
                k[g * I + i] = 0u;
                if (p < Pg) {
                    uint32_t c = sm.keys[g * Sm::kRow + p];
                    if (c >= ncols_g) {  // negative columns included
                        raise_error(err, kErrInvalid, 4, static_cast<int32_t>(c));
                        c = 0;
                        sm.keys[g * Sm::kRow + p] = 0u;
                    }
                    k[g * I + i] = c;
                    lo = min(lo, c);
                    hi = max(hi, c);
                }
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == g) cmin = lo;
            const bool wide = Pg > 0 && hi - lo >= kMaxRange;
            if (wide) {
                int32_t* oc = shfl_ptr(out_col, g);
                double* ov = shfl_ptr(out_val, g);
                __syncwarp();
                const uint32_t n = finish_wide_row<I>(sm.keys + g * Sm::kRow, sm.list + g * Sm::kRow, sm.vals + g * Sm::kRow,
                                                      Pg, oc, ov, (slot_rows >> g & 1u) != 0, lane);
                if (lane == g) {
                    kept = n;
                    P = 0;
                    J->nz[row] = n;
                }
            }
#pragma unroll
            for (int i = 0; i < I; ++i)
                k[g * I + i] = !wide && i * 32 + lane < Pg ? ((k[g * I + i] - lo) << S) | static_cast<uint32_t>(i * 32 + lane) : kDeadKey;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) warp_sort(reinterpret_cast<uint32_t(&)[I]>(k[g * I]), lane);
        __syncwarp();

        uint32_t same;  // see 3.
        // 3. runs of equal columns (fold_runs over all rows): bit g * I + i of `same`
        //    is position lane * I + i of row g
        {
            constexpr uint32_t kFirst = [] {
                uint32_t m = 0;
                for (int g = 0; g < G; ++g) m |= 1u << (g * I);
                return m;
            }();
            same = 0;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const uint32_t before = __shfl_up_sync(0xffffffffu, k[g * I + I - 1], 1);
#pragma unroll
                for (int i = 0; i < I; ++i) {
                    const uint32_t w = k[g * I + i], p = i ? k[g * I + i - 1] : before;
                    if (((w ^ p) >> S) == 0u && w != kDeadKey && (i || lane)) same |= 1u << (g * I + i);
                    sm.keys[g * Sm::kRow + lane * I + i] = w;
                }
            }
            uint32_t next = __shfl_down_sync(0xffffffffu, same, 1);
            if (lane == 31) next = 0;
            uint32_t starts = ~same & (((same >> 1) & ~(kFirst << (I - 1))) | ((next & kFirst) << (I - 1)));
            __syncwarp();
            if (__any_sync(0xffffffffu, starts)) {
                const uint32_t n = __popc(starts);
                const uint32_t incl = warp_incl_scan(n, lane);
                const uint32_t runs = __shfl_sync(0xffffffffu, incl, 31);
                for (uint32_t at = incl - n; starts; starts &= starts - 1u) {
                    const int b = __ffs(starts) - 1;
                    sm.list[at++] = static_cast<uint16_t>((b / I) * Sm::kRow + lane * I + b % I);
                }
                __syncwarp();
                for (uint32_t j = lane; j < runs; j += 32) {
                    int q = sm.list[j];
                    double* vals = sm.vals + (q / Sm::kRow) * Sm::kRow;
                    const int end = (q / Sm::kRow + 1) * Sm::kRow;
                    const uint32_t key = sm.keys[q];
                    double acc = vals[key & kSeq];
                    for (++q; q < end; ++q) {
                        const uint32_t other = sm.keys[q];
                        if ((other ^ key) >> S) break;
                        acc = __dadd_rn(acc, vals[other & kSeq]);
                        if constexpr (I > 1) sm.keys[q] = kDeadKey;
                    }
                    vals[key & kSeq] = acc;
                }
                __syncwarp();
            }
        }

        // 4. the rows' slots (upper-bound layout) or kept entries (exact layout)
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int Pg = __shfl_sync(0xffffffffu, P, g);
            if (Pg == 0) continue;
            const uint32_t lo = __shfl_sync(0xffffffffu, cmin, g);
            int32_t* __restrict__ oc = shfl_ptr(out_col, g);
            double* __restrict__ ov = shfl_ptr(out_val, g);
            const bool holes = (slot_rows >> g & 1u) != 0;
            int n = 0;
#pragma unroll
            for (int i = 0; i < I; ++i) {
                const int p = i * 32 + lane;
                // (one word a lane: position lane, whose word the lane holds)
                const uint32_t key = I == 1   ? (same >> g & 1u ? kDeadKey : k[g])
                                     : p < Pg ? sm.keys[g * Sm::kRow + p]
                                              : kDeadKey;
                const double v = key != kDeadKey ? sm.vals[g * Sm::kRow + (key & kSeq)] : 0.0;
                const bool keep = nonzero(v);
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                const int at = holes ? p : n + __popc(m & lanemask_lt());
                if (holes ? p < Pg : keep) {
                    oc[at] = keep ? static_cast<int32_t>((key >> S) + lo) : -1;
                    ov[at] = v;
                }
                n += __popc(m);
            }
            if (lane == g) kept = static_cast<uint32_t>(n);
        }
        if (lane < G && P > 0) J->nz[row] = kept;
        mine += kept;
        __syncwarp();  // the next rows rewrite keys and values
    }
    mine = warp_sum(mine);
    if (lane == 0 && mine) atomicAdd(&s_nz, mine);
    __syncthreads();
    if (threadIdx.x == 0 && s_nz) atomicAdd(&stats->nz_total, s_nz);
}

template <int I, int G>
void run_rows(const Job* jobs, const int64_t* items, int64_t count, Stats* stats, ErrWord* err, cudaStream_t st,
              int num_sms) {
    const int smem = 8 * static_cast<int>(sizeof(RowsSmem<I, G>));
    allow_smem<num_rows_kernel<I, G>>(smem);
    num_rows_kernel<I, G><<<capped(count, 8 * G, num_sms * 16), kWarpKernelThreads, smem, st>>>(jobs, items, count, stats,
                                                                                              err);
}

}  // namespace

void launch_numeric_warp(int bin, const Job* d_jobs, const int64_t* d_items, int64_t count, int64_t entries,
                         Stats* d_stats, ErrWord* d_err, cudaStream_t st, int num_sms) {
    // Several short rows per warp: 0.160 -> 0.072 ms for 262,144 rows of 56 products
    // in 8 segments, 0.28 -> 0.21 ms for 262,144 rows of 32 products in 32
    // segments (bound there by the L1 lines that its gathers touch), against one
    // row per warp.  Rows of 65-128 products measure the same either way (two to a
    // warp: 0.110 and 0.113 ms on the power-law product, one: 0.102 and 0.094).
    const bool several = several_rows_per_warp(bin, count, entries, num_sms);
    switch (bin) {
        case 1:
            if (several) run_rows<1, 8>(d_jobs, d_items, count, d_stats, d_err, st, num_sms);
            else run_warp<1>(d_jobs, d_items, count, d_stats, d_err, st, num_sms);
            break;
        case 2:
            if (several) run_rows<2, 4>(d_jobs, d_items, count, d_stats, d_err, st, num_sms);
            else run_warp<2>(d_jobs, d_items, count, d_stats, d_err, st, num_sms);
            break;
        case 3: run_warp<3>(d_jobs, d_items, count, d_stats, d_err, st, num_sms); break;
        case 4: run_warp<4>(d_jobs, d_items, count, d_stats, d_err, st, num_sms); break;
        case 5: run_warp<6>(d_jobs, d_items, count, d_stats, d_err, st, num_sms); break;
        case 6: run_warp<8>(d_jobs, d_items, count, d_stats, d_err, st, num_sms); break;
        case 7: run_warp<12>(d_jobs, d_items, count, d_stats, d_err, st, num_sms); break;
        case 8: run_warp<16>(d_jobs, d_items, count, d_stats, d_err, st, num_sms); break;
        default: break;
    }
}

}  // namespace spg
