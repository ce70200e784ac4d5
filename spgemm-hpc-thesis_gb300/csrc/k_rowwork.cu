// K1 row-work binning, K1b bin scatter, K3 int64 scan and K5 zero compaction.
//
// K1 computes ub_i = nnz(S_i) + sum_{k in A_i} nnz(B_k), the number of scalar
// products of output row i (scalarMultiplicationCount, spgemm_common.cpp:474-487,
// per row).  It also validates every index it follows: A's row offsets, A's
// columns against B.rows (the reference throws "A contains a column index
// outside B's row range", spgemm_common.cpp:141-143) and the offsets of every
// referenced B row.  HBM traffic: A.rp (8 B/row), A.ci (4 B/entry) and one B.rp
// pair per A entry (16 B/entry).
#include <algorithm>
#include <type_traits>

#include "spg_common.cuh"

namespace spg {
namespace {

constexpr int kRowworkThreads = 256;

__device__ inline int job_of_row(const int64_t* job_row_base, int njobs, int64_t g) {
    int lo = 0, hi = njobs - 1;  // last job with base <= g
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (job_row_base[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Scalar products of the A entries [p0, a1) that a lane takes every `step` from
// p0 on, at most U of them, their loads issued together.
template <int U>
__device__ __forceinline__ int64_t entry_products(const Job& J, int64_t p0, int64_t a1, int step, ErrWord* err) {
    int32_t k[U];
    int64_t s[U], e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) k[u] = p0 + u * step < a1 ? J.A.ci[p0 + u * step] : 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        s[u] = e[u] = 0;
        if (p0 + u * step < a1) {
            if (k[u] < 0 || k[u] >= J.B.rows) {
                raise_error(err, kErrColumnRange, 1, p0 + u * step);
            } else {
                s[u] = J.B.rp[k[u]];
                e[u] = J.B.rp[k[u] + 1];
            }
        }
    }
    int64_t len = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (s[u] < 0 || e[u] < s[u] || e[u] > J.B.nnz) raise_error(err, kErrInvalid, 2, k[u]);
        else len += e[u] - s[u];
    }
    return len;
}

// T lanes per row, 32 / T rows per warp at a time; a row of more than 4 T
// entries gives the rest to the whole warp, so that a long row among short ones
// does not keep T lanes busy alone.  Bound by the gathers of B's offsets (and, at
// one warp per row, by the lanes that a short row leaves idle): see
// rowwork_lanes for the choice of T.  The counters are kept per lane and per
// CTA: a 64-bit atomic in shared memory is a compare-and-swap loop, and four of
// them per row took as long as the row.
template <int T>
__global__ void __launch_bounds__(kRowworkThreads)
rowwork_kernel(const Job* __restrict__ jobs, int njobs, const int64_t* __restrict__ job_row_base,
               int64_t total_rows, Stats* __restrict__ stats, ErrWord* __restrict__ err) {
    constexpr int U = 4, kRows = 32 / T;
    __shared__ unsigned int s_bins[kNumBins];
    __shared__ unsigned long long s_products, s_max, s_split, s_short[2];
    const int lane = threadIdx.x & 31, tl = lane % T;
    if (threadIdx.x < kNumBins) s_bins[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        s_products = 0;
        s_max = 0;
        s_split = 0;
        s_short[0] = s_short[1] = 0;
    }
    __syncthreads();

    int64_t products = 0, most = 0, split = 0, short1 = 0, short2 = 0;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * (kRowworkThreads / 32) * kRows;
    for (int64_t g0 = (static_cast<int64_t>(blockIdx.x) * (kRowworkThreads / 32) + (threadIdx.x >> 5)) * kRows;
         g0 < total_rows; g0 += stride) {
        const int64_t g = g0 + lane / T;
        int j = 0, row = 0;
        int64_t a0 = 0, a1 = 0, len = 0;
        if (g < total_rows) {
            j = job_of_row(job_row_base, njobs, g);
            row = static_cast<int>(g - job_row_base[j]);
            a0 = jobs[j].A.rp[row];
            a1 = jobs[j].A.rp[row + 1];
            if (a0 < 0 || a1 < a0 || a1 > jobs[j].A.nnz) {
                if (tl == 0) raise_error(err, kErrInvalid, 3, row);
                a0 = a1 = 0;
            }
            len = entry_products<U>(jobs[j], a0 + tl, a1, T, err);
        }
        unsigned rest = __ballot_sync(0xffffffffu, tl == 0 && a1 - a0 > U * T);
        while (rest) {
            const int src = __ffs(rest) - 1;
            rest &= rest - 1u;
            const Job& J = jobs[__shfl_sync(0xffffffffu, j, src)];
            const int64_t p1 = __shfl_sync(0xffffffffu, a1, src);
            int64_t more = 0;
            for (int64_t p = __shfl_sync(0xffffffffu, a0, src) + U * T + lane; p - lane < p1; p += 32 * U)
                more += entry_products<U>(J, p, p1, 32, err);
            more = warp_sum(more);
            if (lane == src) len += more;
        }
#pragma unroll
        for (int o = T / 2; o > 0; o >>= 1) len += __shfl_xor_sync(0xffffffffu, len, o);
        if (tl == 0 && g < total_rows) {
            const Job& J = jobs[j];
            if (J.S.rp) len += J.S.rp[row + 1] - J.S.rp[row];
            J.ub[row] = len;
            J.cnt[row] = len;  // upper-bound layout; the exact mode's symbolic phase overwrites it
            if (J.nz) J.nz[row] = 0;
            if (row == J.A.rows - 1) {  // the entries past the last row, which the scans turn into totals
                J.cnt[row + 1] = 0;
                if (J.nz) J.nz[row + 1] = 0;
            }
            atomicAdd(&s_bins[bin_of(len)], 1u);
            products += len;
            most = len > most ? len : most;
            if (len > kSplitThreshold) split += len;
            if (len > 0 && len <= bin_capacity(1)) short1 += a1 - a0;
            else if (len > 0 && len <= bin_capacity(2)) short2 += a1 - a0;
        }
    }
    products = warp_sum(products);
    most = warp_max(most);
    split = warp_sum(split);
    short1 = warp_sum(short1);
    short2 = warp_sum(short2);
    if (lane == 0 && products) {
        if (short1) atomicAdd(&s_short[0], static_cast<unsigned long long>(short1));
        if (short2) atomicAdd(&s_short[1], static_cast<unsigned long long>(short2));
        atomicAdd(&s_products, static_cast<unsigned long long>(products));
        atomicMax(&s_max, static_cast<unsigned long long>(most));
        if (split) atomicAdd(&s_split, static_cast<unsigned long long>(split));
    }
    __syncthreads();
    if (threadIdx.x < kNumBins && s_bins[threadIdx.x])
        atomicAdd(&stats->bin_count[threadIdx.x], static_cast<unsigned long long>(s_bins[threadIdx.x]));
    if (threadIdx.x == 0 && s_products) {
        atomicAdd(&stats->products, s_products);
        atomicMax(&stats->max_ub, s_max);
        if (s_split) atomicAdd(&stats->split_products, s_split);
        if (s_short[0]) atomicAdd(&stats->short_entries[0], s_short[0]);
        if (s_short[1]) atomicAdd(&stats->short_entries[1], s_short[1]);
    }
}

__device__ __forceinline__ void read_back(const Readback& r) {
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < r.words; i += blockDim.x) r.dst[i] = r.src[i];
}

// A CTA takes kScatterRows rows at a time, counts them by bin in shared memory
// (the counter's old value is the row's place among them) and takes one range of
// every bin's list: one global atomic per bin and CTA.  With one per bin and warp,
// 1,048,576 rows queued on 19 addresses for 77 us; now 9 us.
constexpr int kScatterItems = 4;
constexpr int kScatterRows = 256 * kScatterItems;

__global__ void __launch_bounds__(256)
bin_scatter_kernel(const Job* __restrict__ jobs, int njobs, const int64_t* __restrict__ job_row_base,
                   int64_t total_rows, const Stats* __restrict__ stats,
                   unsigned long long* __restrict__ cursor, int64_t* __restrict__ items, const Readback read) {
    read_back(read);
    __shared__ int64_t s_list[kNumBins];  // the lists follow one another in bin order
    __shared__ int64_t s_base[kNumBins];
    __shared__ unsigned int s_count[kNumBins];
    if (threadIdx.x < kNumBins) {
        int64_t before = 0;
        for (int b = 1; b < static_cast<int>(threadIdx.x); ++b) before += static_cast<int64_t>(stats->bin_count[b]);
        s_list[threadIdx.x] = before;
    }
    for (int64_t base = static_cast<int64_t>(blockIdx.x) * kScatterRows; base < total_rows;
         base += static_cast<int64_t>(gridDim.x) * kScatterRows) {
        if (threadIdx.x < kNumBins) s_count[threadIdx.x] = 0;
        __syncthreads();
        int bin[kScatterItems];
        unsigned int place[kScatterItems];
        int64_t item[kScatterItems];
#pragma unroll
        for (int i = 0; i < kScatterItems; ++i) {
            const int64_t g = base + i * 256 + threadIdx.x;
            bin[i] = kBinEmpty;
            if (g < total_rows) {
                const int j = job_of_row(job_row_base, njobs, g);
                const int row = static_cast<int>(g - job_row_base[j]);
                bin[i] = bin_of(jobs[j].ub[row]);
                item[i] = make_item(j, row);
            }
        }
#pragma unroll
        for (int i = 0; i < kScatterItems; ++i)
            if (bin[i] != kBinEmpty) place[i] = atomicAdd(&s_count[bin[i]], 1u);
        __syncthreads();
        if (threadIdx.x < kNumBins && s_count[threadIdx.x])
            s_base[threadIdx.x] = s_list[threadIdx.x] +
                                  static_cast<int64_t>(atomicAdd(&cursor[threadIdx.x], static_cast<unsigned long long>(s_count[threadIdx.x])));
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kScatterItems; ++i)
            if (bin[i] != kBinEmpty) items[s_base[bin[i]] + place[i]] = item[i];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// K3: exclusive int64 scan in two phases: tile sums, then every tile's scan from
// the sum of the tile sums before it, which its CTA adds up itself (a third
// kernel that scans the tile sums costs a launch; above kScanDirect tiles it
// pays).  One tile takes one launch.  No block waits on another block.  A thread
// takes eight consecutive counts in 16-byte loads: a transposition through
// shared memory put them in one bank.  65,537 counts in 12 -> 5 us,
// 1,048,577 in 18 -> 9.5 us.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int64_t kScanDirect = 2048;

__device__ inline int64_t block_excl_scan(int64_t v, int64_t* s_warp, int64_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int64_t incl = warp_incl_scan(v, lane);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int64_t w = lane < nw ? s_warp[lane] : 0;
        const int64_t wi = warp_incl_scan(w, lane);
        if (lane < nw) s_warp[lane] = wi - w;
        if (lane == nw - 1) s_warp[32] = wi;
    }
    __syncthreads();
    const int64_t out = s_warp[warp] + incl - v;
    total = s_warp[32];
    __syncthreads();
    return out;
}

// The thread's counts of its CTA's tile (data is 16-byte aligned), zero past n.
__device__ inline int64_t load_counts(const int64_t* __restrict__ data, int64_t n, int64_t (&v)[kScanItems]) {
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
    if (base + kScanItems <= n) {
#pragma unroll
        for (int i = 0; i < kScanItems; i += 2) {
            const longlong2 x = *reinterpret_cast<const longlong2*>(data + base + i);
            v[i] = x.x;
            v[i + 1] = x.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) v[i] = base + i < n ? data[base + i] : 0;
    }
    int64_t sum = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) sum += v[i];
    return sum;
}

__global__ void __launch_bounds__(kScanThreads)
scan_reduce_kernel(const int64_t* __restrict__ data, int64_t n, int64_t* __restrict__ partials) {
    __shared__ int64_t s_warp[kScanThreads / 32];
    int64_t v[kScanItems];
    const int64_t sum = warp_sum(load_counts(data, n, v));
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t total = 0;
        for (int w = 0; w < kScanThreads / 32; ++w) total += s_warp[w];
        partials[blockIdx.x] = total;
    }
}

__global__ void __launch_bounds__(1024)
scan_partials_kernel(int64_t* __restrict__ partials, int64_t nparts) {
    __shared__ int64_t s_warp[33];
    int64_t carry = 0;
    for (int64_t base = 0; base < nparts; base += blockDim.x) {
        const int64_t idx = base + threadIdx.x;
        const int64_t v = idx < nparts ? partials[idx] : 0;
        int64_t total;
        const int64_t ex = block_excl_scan(v, s_warp, total);
        if (idx < nparts) partials[idx] = carry + ex;
        carry += total;
    }
}

// partials: tile sums (sums != 0) or their exclusive scan.
__global__ void __launch_bounds__(kScanThreads)
scan_down_kernel(int64_t* __restrict__ data, int64_t n, const int64_t* __restrict__ partials, int sums) {
    __shared__ int64_t s_warp[33];
    __shared__ int64_t s_before[kScanThreads / 32];
    int64_t before = 0;
    if (sums) {
        for (int t = threadIdx.x; t < static_cast<int>(blockIdx.x); t += kScanThreads) before += partials[t];
        before = warp_sum(before);
        if ((threadIdx.x & 31) == 0) s_before[threadIdx.x >> 5] = before;
    }
    int64_t v[kScanItems];
    const int64_t sum = load_counts(data, n, v);
    int64_t total;
    int64_t at = block_excl_scan(sum, s_warp, total);  // its barriers order s_before too
    before = 0;
    if (sums) {
#pragma unroll
        for (int w = 0; w < kScanThreads / 32; ++w) before += s_before[w];
    } else {
        before = partials[blockIdx.x];
    }
    at += before;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const int64_t x = v[i];
        v[i] = at;
        at += x;
    }
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
    if (base + kScanItems <= n) {
#pragma unroll
        for (int i = 0; i < kScanItems; i += 2) *reinterpret_cast<longlong2*>(data + base + i) = make_longlong2(v[i], v[i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; ++i)
            if (base + i < n) data[base + i] = v[i];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) data[n] = before + total;
}

// K5: warp per row, copies the stored entries of a row from its C_tmp offset
// (job.cnt, scanned) to its final offset (job.nz, scanned).
__global__ void __launch_bounds__(256)
compact_kernel(const Job* __restrict__ job, int rows, int32_t* __restrict__ out_col, double* __restrict__ out_val) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
    for (int64_t r = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps) {
        const int64_t src = job->cnt[r], n = job->nz[r + 1] - job->nz[r];
        int32_t* oc = out_col;
        double* ov = out_val;
        int64_t dst = job->nz[r];
        if (!oc) {  // the job's own arrays
            oc = job->out_col;
            ov = job->out_val;
            dst -= job->nz[0];
        }
        for (int64_t q = lane; q < n; q += 32) {
            oc[dst + q] = job->c_col[src + q];
            ov[dst + q] = job->c_val[src + q];
        }
    }
}

// The rows of more than kLongSlots slots (long_rows, items of the bin lists), a
// CTA each: a step takes kChunks chunks of 32 slots per warp, whose counts place the
// warps' entries after one another.
__device__ void compact_long_rows(const Job* __restrict__ jobs, const int64_t* __restrict__ long_rows, int64_t n_long,
                                  int64_t first, int64_t step, int32_t* __restrict__ out_col,
                                  double* __restrict__ out_val) {
    constexpr int kChunks = 8, kWarps = 8;
    __shared__ int s_count[2][kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int side = 0;
    for (int64_t i = first; i < n_long; i += step) {
        const Job& J = jobs[item_job(long_rows[i])];
        const int r = item_row(long_rows[i]);
        int32_t* __restrict__ oc = out_col ? out_col : J.out_col;
        double* __restrict__ ov = out_col ? out_val : J.out_val;
        const int64_t end = J.cnt[r + 1];
        int64_t dst = J.nz[r] - (out_col ? 0 : J.nz[0]);
        for (int64_t q0 = J.cnt[r]; q0 < end; q0 += kWarps * kChunks * 32) {
            int32_t c[kChunks];
            double v[kChunks];
            const int64_t at = q0 + warp * (kChunks * 32) + lane;
#pragma unroll
            for (int u = 0; u < kChunks; ++u) {
                c[u] = at + u * 32 < end ? J.c_col[at + u * 32] : -1;
                v[u] = at + u * 32 < end ? J.c_val[at + u * 32] : 0.0;
            }
            int count = 0;
#pragma unroll
            for (int u = 0; u < kChunks; ++u) count += __popc(__ballot_sync(0xffffffffu, c[u] >= 0));
            if (lane == 0) s_count[side][warp] = count;
            __syncthreads();  // the other side's counts are written only after the next one
            int64_t to = dst;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const int n = s_count[side][w];
                dst += n;
                if (w < warp) to += n;
            }
            side ^= 1;
#pragma unroll
            for (int u = 0; u < kChunks; ++u) {
                const unsigned m = __ballot_sync(0xffffffffu, c[u] >= 0);
                if (c[u] >= 0) {
                    oc[to + __popc(m & lanemask_lt())] = c[u];
                    ov[to + __popc(m & lanemask_lt())] = v[u];
                }
                to += __popc(m);
            }
        }
    }
}

// K5 for rows written with holes (upper-bound mode): a warp takes `group`
// consecutive rows, whose reserved slots [cnt[r], cnt[r + group]) are contiguous
// as their entries in C are: the slots are read in order and those with a column
// >= 0 packed from the first row's final offset nz[r] on (ballot + popc).  Each
// warp loads its next group's offsets while it copies the current one, and issues
// eight chunks of 32 slots per step.  262,144 rows of 56 and of 32 slots: 0.068 ms
// together (0.188 with one row per warp, whose eight chunks were mostly empty).
// A step of a warp waits about 1 us for memory, so one row of 100,000 slots alone
// took a warp as long as the GPU needs for 100 M slots: rows of kLongBin and above
// are left to the first `long_ctas` CTAs.  Power-law squares of 65,539, 100,003 and
// 1 M rows (36, 56 and 595 M slots): 165, 244 and 2,204 us (339, 422 and 2,360
// before); the last is 6.3 TB/s, 94% of the measured copy bandwidth.
__global__ void __launch_bounds__(256)
compact_holes_kernel(const Job* __restrict__ jobs, int njobs, const int64_t* __restrict__ job_row_base,
                     int64_t total_rows, int group, const int64_t* __restrict__ long_rows, int64_t n_long,
                     int long_ctas, int32_t* __restrict__ out_col, double* __restrict__ out_val, const Readback read,
                     const Stats* full, int64_t slots, const ErrWord* err) {
    constexpr int kChunks = 8;
    read_back(read);
    if (full && (err->code != 0 || static_cast<int64_t>(full->nz_total) == slots)) return;
    if (static_cast<int>(blockIdx.x) < long_ctas) {
        compact_long_rows(jobs, long_rows, n_long, blockIdx.x, long_ctas, out_col, out_val);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int64_t stride = static_cast<int64_t>(gridDim.x - long_ctas) * (blockDim.x >> 5) * group;
    int64_t g = (static_cast<int64_t>(blockIdx.x - long_ctas) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * group;
    int64_t group_end = min(g + group, total_rows);
    int j = 0;
    int64_t n_src = 0, n_end = 0, n_dst = 0, n_row = 0;
    auto load_rows = [&](int64_t row) {  // the group's rows from `row` on, of one product
        j = job_of_row(job_row_base, njobs, row);
        n_row = min(group_end, job_row_base[j + 1]);
        const int r = static_cast<int>(row - job_row_base[j]);
        int r1 = static_cast<int>(n_row - job_row_base[j]);
        if (long_ctas) {  // up to the next long row, or past one
            for (int i = r; i < r1; i += 32) {
                const bool is_long = i + lane < r1 && jobs[j].cnt[i + lane + 1] - jobs[j].cnt[i + lane] > kLongSlots;
                const unsigned m = __ballot_sync(0xffffffffu, is_long);
                if (m) {
                    r1 = i + __ffs(m) - 1;
                    break;
                }
            }
            n_row = job_row_base[j] + max(r1, r + 1);
        }
        n_src = jobs[j].cnt[r];
        n_end = jobs[j].cnt[r1];
        n_dst = jobs[j].nz[r] - (out_col ? 0 : jobs[j].nz[0]);  // the job's own arrays start at its first row
    };
    if (g < total_rows) load_rows(g);
    while (g < total_rows) {
        const Job& J = jobs[j];
        int32_t* __restrict__ oc = out_col ? out_col : J.out_col;
        double* __restrict__ ov = out_col ? out_val : J.out_val;
        const int64_t src = n_src, end = n_end;
        int64_t dst = n_dst;
        g = n_row;
        if (g >= group_end) {
            g = group_end - group + stride;  // only the last group is shorter, and no group follows it
            group_end = min(g + group, total_rows);
        }
        if (g < total_rows) load_rows(g);
        // columns and values are loaded together (a hole's value is read and
        // dropped) so the loads do not wait on each other
        for (int64_t q0 = src; q0 < end; q0 += kChunks * 32) {
            int32_t c[kChunks];
            double v[kChunks];
#pragma unroll
            for (int u = 0; u < kChunks; ++u) {
                const int64_t q = q0 + u * 32 + lane;
                c[u] = q < end ? J.c_col[q] : -1;
                v[u] = q < end ? J.c_val[q] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kChunks; ++u) {
                const unsigned m = __ballot_sync(0xffffffffu, c[u] >= 0);
                if (c[u] >= 0) {
                    const int64_t at = dst + __popc(m & lanemask_lt());
                    oc[at] = c[u];
                    ov[at] = v[u];
                }
                dst += __popc(m);
            }
        }
    }
}

__global__ void starts_kernel(const int64_t* __restrict__ scanned, const int64_t* __restrict__ job_row_base, int64_t* dst,
                              int njobs, const Readback read) {
    read_back(read);
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < njobs; j += gridDim.x * blockDim.x)
        dst[j] = scanned[job_row_base[j] + j];
}

// Small device->host reads by a kernel storing into mapped page-locked memory:
// they do not queue on the copy engines behind bulk result copies.
__global__ void readback_kernel(const unsigned long long* __restrict__ src, unsigned long long* dst, int64_t words) {
    for (int64_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}

__global__ void add_offset_kernel(int64_t* __restrict__ d, int64_t n, int64_t add) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        d[i] += add;
}

// blockIdx.y selects product j: out[base_j + r] = scanned[base_j + r] - scanned[base_j]
// for r <= rows_j, where base_j = job_row_base[j] + j (each product's offsets
// restart at zero; the start stays in device memory).
__global__ void rebase_jobs_kernel(const int64_t* __restrict__ scanned, int64_t* __restrict__ out,
                                   const int64_t* __restrict__ job_row_base) {
    const int j = blockIdx.y;
    const int64_t base = job_row_base[j] + j;
    const int64_t rows = job_row_base[j + 1] - job_row_base[j];
    const int64_t start = scanned[base];
    for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r <= rows;
         r += static_cast<int64_t>(gridDim.x) * blockDim.x)
        out[base + r] = scanned[base + r] - start;
}

// One CTA per product: its scalar products, the sum of its rows' ub.
__global__ void job_products_kernel(const Job* __restrict__ jobs, const int64_t* __restrict__ job_row_base,
                                    int64_t* __restrict__ out) {
    __shared__ int64_t s_part[8];
    const int j = blockIdx.x;
    const int64_t rows = job_row_base[j + 1] - job_row_base[j];
    const int64_t* ub = jobs[j].ub;
    int64_t sum = 0;
    for (int64_t r = threadIdx.x; r < rows; r += blockDim.x) sum += ub[r];
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t t = 0;
        for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) t += s_part[w];
        out[j] = t;
    }
}

// blockIdx.y selects the product; threads stride over its rows + 1 offsets.
__global__ void rebase_kernel(const RebaseItem* __restrict__ items) {
    const RebaseItem it = items[blockIdx.y];
    for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r <= it.rows;
         r += static_cast<int64_t>(gridDim.x) * blockDim.x)
        it.rp[r] = it.src[r] - it.start;
}

int grid_for(int64_t work, int per_block, int cap) {
    const int64_t g = (work + per_block - 1) / per_block;
    return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace

void launch_rowwork(const Job* d_jobs, int njobs, const int64_t* d_job_row_base, int64_t total_rows, int64_t entries,
                    Stats* d_stats, ErrWord* d_err, cudaStream_t stream) {
    if (total_rows <= 0) return;
    auto run = [&](auto t) {
        constexpr int T = decltype(t)::value;
        rowwork_kernel<T><<<grid_for(total_rows, kRowworkThreads / T, 152 * 8), kRowworkThreads, 0, stream>>>(
            d_jobs, njobs, d_job_row_base, total_rows, d_stats, d_err);
    };
    if (rowwork_lanes(entries, total_rows) == 4) run(std::integral_constant<int, 4>{});
    else run(std::integral_constant<int, 8>{});
}

void launch_bin_scatter(const Job* d_jobs, int njobs, const int64_t* d_job_row_base, int64_t total_rows,
                        const Stats* d_stats, unsigned long long* d_bin_cursor, int64_t* d_items, cudaStream_t stream,
                        const Readback& read) {
    if (total_rows <= 0) return;
    const int grid = grid_for(total_rows, kScatterRows, 152 * 8);
    bin_scatter_kernel<<<grid, 256, 0, stream>>>(d_jobs, njobs, d_job_row_base, total_rows, d_stats, d_bin_cursor,
                                                  d_items, read);
}

size_t scan_partials_count(int64_t n) { return static_cast<size_t>((n + kScanTile - 1) / kScanTile) + 1; }

void launch_scan(int64_t* d_data, int64_t n, int64_t* d_partials, cudaStream_t stream) {
    const int64_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 0) {
        cudaMemsetAsync(d_data, 0, sizeof(int64_t), stream);
        return;
    }
    if (nb > 1) scan_reduce_kernel<<<static_cast<unsigned>(nb), kScanThreads, 0, stream>>>(d_data, n, d_partials);
    if (nb > kScanDirect) scan_partials_kernel<<<1, 1024, 0, stream>>>(d_partials, nb);
    scan_down_kernel<<<static_cast<unsigned>(nb), kScanThreads, 0, stream>>>(d_data, n, d_partials, nb <= kScanDirect);
}

int scan_launches(int64_t n) { return n <= 0 ? 0 : n <= kScanTile ? 1 : n <= kScanDirect * kScanTile ? 2 : 3; }

void launch_compact(const Job* d_job, int rows, int32_t* out_col, double* out_val, cudaStream_t stream) {
    if (rows <= 0) return;
    compact_kernel<<<grid_for(rows, 8, 152 * 16), 256, 0, stream>>>(d_job, rows, out_col, out_val);
}

void launch_compact_holes(const Job* d_jobs, int njobs, const int64_t* d_job_row_base, int64_t total_rows,
                          int64_t slots, const int64_t* items, const int64_t* bin_off, int32_t* out_col,
                          double* out_val, cudaStream_t stream, const Readback& read, const Stats* full,
                          const ErrWord* err) {
    if (total_rows <= 0) {
        if (read.words) launch_readback(read.src, read.dst, static_cast<size_t>(read.words) * 8, stream);
        return;
    }
    const int64_t n_long = bin_off[kNumBins] - bin_off[kLongBin];
    const int long_ctas = static_cast<int>(std::min<int64_t>(n_long, 152 * 8));
    // Rows per warp: about two steps of 256 slots.
    const int64_t mean = slots / total_rows + 1;
    const int group = static_cast<int>(std::min<int64_t>(std::max<int64_t>(512 / mean, 1), 64));
    compact_holes_kernel<<<long_ctas + grid_for(total_rows, 8 * group, 152 * 128), 256, 0, stream>>>(
        d_jobs, njobs, d_job_row_base, total_rows, group, items + bin_off[kLongBin], n_long, long_ctas, out_col,
        out_val, read, full, slots, err);
}

void launch_starts(const int64_t* d_scanned, const int64_t* d_job_row_base, int64_t* dst, int njobs,
                   cudaStream_t stream, const Readback& read) {
    if (njobs <= 0) return;
    starts_kernel<<<grid_for(njobs, 256, 1024), 256, 0, stream>>>(d_scanned, d_job_row_base, dst, njobs, read);
}

void launch_job_products(const Job* d_jobs, int njobs, const int64_t* d_job_row_base, int64_t* d_out,
                         cudaStream_t stream) {
    if (njobs <= 0) return;
    job_products_kernel<<<njobs, 256, 0, stream>>>(d_jobs, d_job_row_base, d_out);
}

namespace {

// Split points of `rows` rows into `parts` contiguous blocks of about equal
// scalar products: first[k] is the first row whose preceding products reach
// floor(k * total / parts) (prefix: exclusive scan of the per-row products,
// prefix[rows] = total); first[0] = 0, first[parts] = rows.  With no products
// at all the rows are split by count, as the reference's partitionRows does.
__global__ void partition_kernel(const int64_t* __restrict__ prefix, int64_t rows, int32_t parts,
                                 int32_t* __restrict__ first) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > parts) return;
    const int64_t total = prefix[rows];
    int64_t r;
    if (k == 0) {
        r = 0;
    } else if (k == parts) {
        r = rows;
    } else if (total == 0) {
        r = rows * k / parts;
    } else {
        const int64_t target = static_cast<int64_t>(static_cast<unsigned __int128>(total) * k / parts);
        int64_t lo = 0, hi = rows;  // smallest i with prefix[i] >= target
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (prefix[mid] >= target) hi = mid;
            else lo = mid + 1;
        }
        r = lo;
    }
    first[k] = static_cast<int32_t>(r);
}

}  // namespace

void launch_partition(const int64_t* d_prefix, int64_t rows, int32_t parts, int32_t* d_first, cudaStream_t stream) {
    partition_kernel<<<(parts + 1 + 127) / 128, 128, 0, stream>>>(d_prefix, rows, parts, d_first);
}

void launch_readback(const void* d_src, void* h_dst, size_t bytes, cudaStream_t stream) {
    if (bytes == 0) return;
    readback_kernel<<<1, 256, 0, stream>>>(static_cast<const unsigned long long*>(d_src),
                                           static_cast<unsigned long long*>(h_dst), static_cast<int64_t>(bytes / 8));
}

void launch_rebase_jobs(const int64_t* d_scanned, int64_t* d_out, const int64_t* d_job_row_base, int njobs,
                        int64_t max_rows, cudaStream_t stream) {
    if (njobs <= 0) return;
    const dim3 grid(grid_for(max_rows + 1, 256, 64), static_cast<unsigned>(njobs));
    rebase_jobs_kernel<<<grid, 256, 0, stream>>>(d_scanned, d_out, d_job_row_base);
}

void launch_add_offset(int64_t* d, int64_t n, int64_t add, cudaStream_t stream) {
    if (n <= 0 || add == 0) return;
    add_offset_kernel<<<grid_for(n, 256, 152 * 8), 256, 0, stream>>>(d, n, add);
}

void launch_rebase(const RebaseItem* d_items, int n, int64_t max_rows, cudaStream_t stream) {
    if (n <= 0) return;
    const dim3 grid(grid_for(max_rows + 1, 256, 64), static_cast<unsigned>(n));
    rebase_kernel<<<grid, 256, 0, stream>>>(d_items);
}

}  // namespace spg
