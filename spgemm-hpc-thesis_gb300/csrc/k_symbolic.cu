// K2 symbolic phase: the number of distinct columns of every output row.
//
// This is the count of `accumulator.emplace` insertions in the reference row
// loop (spgemm_exchange.cpp:288-293), i.e. an upper bound of the row's stored
// entries before exact zeros are dropped.  Rows are counted in open-addressing
// hash tables of at least twice the row's product count:
//   * rows of <= 32 products: one warp, one product per lane, distinct columns
//     found with __match_any_sync (no table);
//   * rows of <= 512 products: one warp per row, table in shared memory;
//   * rows of <= 16384 products: one CTA per row, table in shared memory;
//   * heavier rows: one CTA per row, table in a global-memory slab per CTA.
// Where a bit per column of B takes at most twice the words of the bin's table, the
// table is a bitmap: one atomic per product instead of a hash, a compare-and-swap and
// its retries.  Column c is bit c / words of word c % words, so that neighbouring
// columns lie in neighbouring banks.  A heavier row's bitmap is in shared memory up to
// 2^20 columns.  K2 of power-law squares of 65,536, 131,071 and 262,144 rows: 304 ->
// 187, 541 -> 395 and 1,076 -> 870 us; with the line at the table's size 200, 417 and
// 918, at four times it 187, 444 and 946 (fewer CTAs per SM, more words to clear).
// Every launch reserves the tables of its bin's largest row only (a power of
// two >= twice the bin capacity), so that the bins of short rows keep many
// CTAs per SM.  It also rejects B columns outside [0, B.cols).
#include <algorithm>

#include "spg_enum.cuh"

namespace spg {
namespace {

constexpr int kSymWarpThreads = 256;
constexpr int kSymHeavyThreads = 512;
constexpr int kLastSymSmemBin = 18;  // rows of <= 16384 products: shared-memory tables
// Last bins of the 64- and 128-thread CTAs (rows of <= 1024 and 2048 products).
constexpr int kSymB64 = 10, kSymB128 = 12;

// Table slots reserved per row (warp bins) or per CTA (CTA bins) for bin b:
// the power of two >= twice its capacity, at least 64.
int sym_table_slots(int b) {
    int64_t t = 64;
    while (t < 2 * bin_capacity(b)) t *= 2;
    return static_cast<int>(t);
}

__device__ inline bool col_ok(int32_t c, int32_t cols, ErrWord* err) {
    if (c < 0 || c >= cols) {
        raise_error(err, kErrInvalid, 4, c);
        return false;
    }
    return true;
}

// Inserts col; returns 1 if it was not present.
__device__ inline int hash_insert(int32_t* tab, uint32_t mask, int log2t, int32_t col) {
    uint32_t h = hash_slot(col, log2t);
    while (true) {
        const int32_t old = atomicCAS(&tab[h], -1, col);
        if (old == -1) return 1;
        if (old == col) return 0;
        h = (h + 1) & mask;
    }
}

// Sets column col's bit in a bitmap of 2^log2w words; returns 1 if it was not set.
__device__ inline int bitmap_insert(uint32_t* map, int log2w, int32_t col) {
    const uint32_t bit = 1u << (static_cast<uint32_t>(col) >> log2w);
    return (atomicOr(&map[static_cast<uint32_t>(col) & ((1u << log2w) - 1u)], bit) & bit) == 0u;
}

// log2 of the words reserved per row of a bin: the table's, or a bitmap's of up to
// twice as many.
int reserved_log2(int bin, int64_t max_cols) {
    const int slots = sym_table_slots(bin), map = bitmap_log2(max_cols);
    return map <= kMaxBitmapLog2 && (1 << map) <= 2 * slots ? std::max(map, ceil_log2(slots)) : ceil_log2(slots);
}

template <int NT>
__device__ inline void clear_words(int32_t* tab, uint32_t n, int tid, int32_t value) {
    if (n >= 4 * NT) {
        for (uint32_t s = 4 * tid; s < n; s += 4 * NT) *reinterpret_cast<int4*>(tab + s) = make_int4(value, value, value, value);
    } else {
        for (uint32_t s = tid; s < n; s += NT) tab[s] = value;
    }
}

__global__ void __launch_bounds__(kSymWarpThreads)
sym_warp_kernel(const Job* __restrict__ jobs, const int64_t* __restrict__ items, int64_t count, int tiny,
                int wtab_log2, ErrWord* __restrict__ err) {
    extern __shared__ __align__(16) int32_t s_dyn[];  // kSymWarpThreads / 32 tables of wtab slots
    const int wtab = 1 << wtab_log2;
    __shared__ RowSegs<32, 512> s_seg[kSymWarpThreads / 32];  // rows of at most 512 products
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (kSymWarpThreads / 32);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * (kSymWarpThreads / 32) + w; i < count; i += warps) {
        const int64_t it = items[i];
        const Job& J = jobs[item_job(it)];
        const int row = item_row(it);
        const int64_t ub = J.ub[row];
        int found = 0;
        if (tiny) {
            // <= 32 products: product t goes to lane t; count the first lane of each column group.
            int32_t* stage = s_dyn + w * wtab;
            team_row_products<32, 512, 4, false>(J, row, s_seg[w], nullptr, lane, [&](int32_t seq, int32_t c, double, double) {
                stage[seq] = c;
            });
            __syncwarp();
            const bool valid = lane < ub;
            const int32_t col = valid ? stage[lane] : -1;
            __syncwarp();
            if (valid) col_ok(col, J.B.cols, err);
            const unsigned peers = __match_any_sync(0xffffffffu, valid ? col : -1);
            const bool first = valid && (peers & lanemask_lt()) == 0;
            found = __popc(__ballot_sync(0xffffffffu, first));
        } else {
            const int log2t = max(6, ceil_log2(2 * ub));
            const uint32_t tsize = 1u << log2t, mask = tsize - 1;
            int32_t* tab = s_dyn + w * wtab;
            const int log2w = bitmap_log2(J.B.cols);
            const bool bits = log2w <= wtab_log2;
            clear_words<32>(tab, bits ? 1u << log2w : tsize, lane, bits ? 0 : -1);
            __syncwarp();
            int mine = 0;
            team_row_products<32, 512, 4, false>(J, row, s_seg[w], nullptr, lane, [&](int32_t, int32_t c, double, double) {
                if (!col_ok(c, J.B.cols, err)) return;
                mine += bits ? bitmap_insert(reinterpret_cast<uint32_t*>(tab), log2w, c) : hash_insert(tab, mask, log2t, c);
            });
            found = warp_sum(mine);
            __syncwarp();
        }
        if (lane == 0) J.cnt[row] = found;
    }
}

template <int NT, int CAP>
__global__ void __launch_bounds__(NT)
sym_block_kernel(const Job* __restrict__ jobs, const int64_t* __restrict__ items, int64_t count,
                 int tab_log2, ErrWord* __restrict__ err) {
    extern __shared__ __align__(16) int32_t s_tab[];  // 2^tab_log2 words
    __shared__ RowSegs<NT, CAP> s_seg;
    __shared__ int64_t s_warp[NT / 32 + 1];
    __shared__ int s_found;
    for (int64_t i = blockIdx.x; i < count; i += gridDim.x) {
        const int64_t it = items[i];
        const Job& J = jobs[item_job(it)];
        const int row = item_row(it);
        const int log2t = max(6, ceil_log2(2 * J.ub[row]));
        const uint32_t tsize = 1u << log2t, mask = tsize - 1;
        const int log2w = bitmap_log2(J.B.cols);
        const bool bits = log2w <= tab_log2;
        clear_words<NT>(s_tab, bits ? 1u << log2w : tsize, threadIdx.x, bits ? 0 : -1);
        if (threadIdx.x == 0) s_found = 0;
        __syncthreads();
        int mine = 0;
        team_row_products<NT, CAP, 4, false>(J, row, s_seg, s_warp, threadIdx.x, [&](int32_t, int32_t c, double, double) {
            if (!col_ok(c, J.B.cols, err)) return;
            mine += bits ? bitmap_insert(reinterpret_cast<uint32_t*>(s_tab), log2w, c) : hash_insert(s_tab, mask, log2t, c);
        });
        mine = warp_sum(mine);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_found, mine);
        __syncthreads();
        if (threadIdx.x == 0) J.cnt[row] = s_found;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kSymHeavyThreads)
sym_heavy_kernel(const Job* __restrict__ jobs, const int64_t* __restrict__ items, int64_t count,
                 int32_t* __restrict__ slabs, int64_t slab_slots, int map_log2, ErrWord* __restrict__ err) {
    extern __shared__ __align__(16) int32_t s_map[];  // 2^map_log2 words; none if map_log2 < 0
    __shared__ SegTab<kSymHeavyThreads> s_seg;
    __shared__ int64_t s_warp[kSymHeavyThreads / 32 + 1];
    __shared__ unsigned long long s_found;
    int32_t* tab = slabs + static_cast<int64_t>(blockIdx.x) * slab_slots;
    for (int64_t i = blockIdx.x; i < count; i += gridDim.x) {
        const int64_t it = items[i];
        const Job& J = jobs[item_job(it)];
        const int row = item_row(it);
        const int log2t = ceil_log2(2 * J.ub[row]);
        const uint32_t tsize = 1u << log2t, mask = tsize - 1;
        const int log2w = bitmap_log2(J.B.cols);
        const bool bits = log2w <= map_log2;
        clear_words<kSymHeavyThreads>(bits ? s_map : tab, bits ? 1u << log2w : tsize, threadIdx.x, bits ? 0 : -1);
        if (threadIdx.x == 0) s_found = 0;
        __syncthreads();
        int mine = 0;
        team_products<kSymHeavyThreads, false>(J, row, s_seg, s_warp, threadIdx.x,
                                               [&](int64_t, int32_t c, double, double) {
            if (!col_ok(c, J.B.cols, err)) return;
            mine += bits ? bitmap_insert(reinterpret_cast<uint32_t*>(s_map), log2w, c) : hash_insert(tab, mask, log2t, c);
        });
        mine = warp_sum(mine);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_found, static_cast<unsigned long long>(mine));
        __syncthreads();
        if (threadIdx.x == 0) J.cnt[row] = static_cast<int64_t>(s_found);
        __syncthreads();
    }
}

int capped_grid(int64_t work, int per_block, int cap) {
    const int64_t g = (work + per_block - 1) / per_block;
    return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

int heavy_ctas(int64_t count, int num_sms) { return static_cast<int>(count < num_sms * 2 ? count : num_sms * 2); }

}  // namespace

size_t symbolic_scratch_bytes(const int64_t* bin_count, int64_t max_ub, int num_sms) {
    const int64_t count = bin_count[kBinHeavy];  // the only bin with global-memory tables
    if (count == 0) return 0;
    return static_cast<size_t>(heavy_ctas(count, num_sms)) * (size_t{1} << ceil_log2(2 * max_ub)) * sizeof(int32_t);
}

void launch_symbolic(int bin, const Job* d_jobs, const int64_t* d_items, int64_t count, int64_t max_ub,
                     int64_t max_cols, int64_t map_cols, void* d_scratch, size_t, Stats*, ErrWord* d_err,
                     cudaStream_t stream, int num_sms) {
    if (count <= 0) return;
    if (bin <= kLastWarpBin) {
        const int wtab_log2 = reserved_log2(bin, max_cols);
        const int smem = (kSymWarpThreads / 32) * (4 << wtab_log2);
        allow_smem<sym_warp_kernel>((kSymWarpThreads / 32) * 4 * 2 * sym_table_slots(kLastWarpBin));
        const int grid = capped_grid(count, kSymWarpThreads / 32, num_sms * 32);
        sym_warp_kernel<<<grid, kSymWarpThreads, smem, stream>>>(d_jobs, d_items, count, bin == 1, wtab_log2, d_err);
    } else if (bin <= kLastSymSmemBin) {
        const int tab_log2 = reserved_log2(bin, max_cols);
        const int smem = 4 << tab_log2;
        auto run = [&](auto kernel, int nt) {
            kernel<<<capped_grid(count, 1, num_sms * (2048 / nt)), nt, smem, stream>>>(d_jobs, d_items, count, tab_log2, d_err);
        };
        // CTA size by row size: 6-12 products per thread on the bins below 4096 products
        allow_smem<sym_block_kernel<64, 1024>>(4 << kMaxBitmapLog2);
        allow_smem<sym_block_kernel<128, 2048>>(4 << kMaxBitmapLog2);
        if (bin <= kSymB64) run(sym_block_kernel<64, 1024>, 64);
        else if (bin <= kSymB128) run(sym_block_kernel<128, 2048>, 128);
        else if (bin <= kLastSmemBin) {
            allow_smem<sym_block_kernel<256, 8192>>(4 << kMaxBitmapLog2);
            run(sym_block_kernel<256, 8192>, 256);
        } else {
            allow_smem<sym_block_kernel<512, 16384>>(4 << kMaxBitmapLog2);
            run(sym_block_kernel<512, 16384>, 512);
        }
    } else {
        const int grid = heavy_ctas(count, num_sms);
        const int64_t slots = int64_t{1} << ceil_log2(2 * max_ub);
        // the shared bitmaps of the products that have few enough columns
        const int map_log2 = heavy_map_log2(map_cols);
        const int smem = map_log2 < 0 ? 0 : 4 << map_log2;
        allow_smem<sym_heavy_kernel>(4 << kMaxBitmapLog2);
        sym_heavy_kernel<<<grid, kSymHeavyThreads, smem, stream>>>(d_jobs, d_items, count,
                                                                  static_cast<int32_t*>(d_scratch), slots, map_log2, d_err);
    }
}

}  // namespace spg
