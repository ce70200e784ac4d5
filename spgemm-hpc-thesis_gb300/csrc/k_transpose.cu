// CSR transpose on the GPU: A^T keeps, in every row, the entries of A's
// column in A's row-major order (a stable counting sort by column), which is
// what a transposition by stable sort of the entries produces on the host.
//
// A device-wide stable LSD radix sort of the entries by column, digits of at
// most 8 bits over the bits of (cols - 1).  Each pass: per-tile digit histograms,
// one scan of the digit-major (digit, tile) table, and a scatter.  The entries
// themselves move (column, row, value: 16 bytes), so that every pass reads in
// order; a tile (4096 entries) is first ordered by digit in shared memory --
// ranks from the warp ballot groups and per-warp digit counters of the numeric
// kernels -- and then written from there, neighbouring threads to neighbouring
// addresses of a digit's run (32 entries on average with 7-bit digits).  The first pass reads A
// and finds the rows of its entries from A's offsets, the last writes rows and
// values of A^T and no column.  Bound by DRAM and by these runs: 12.4 M entries of
// a 524,287^2 power-law matrix in 0.49 ms, the scatters (0.10 ms each, 3.9 TB/s)
// leading; 1.25 ms when the passes moved 8-byte indices and gathered columns and
// values through them.
#include <algorithm>

#include "k_numeric_row.cuh"

namespace spg {
namespace {

constexpr int kTW = 16;
constexpr int kTItems = 8;
constexpr int kTThreads = kTW * 32;
constexpr int kTTile = kTThreads * kTItems;

// Entries of a pass's input or output; col is A's (the sort's key).
struct Entries {
    int32_t* col = nullptr;
    int32_t* row = nullptr;
    double* val = nullptr;
};

struct PassSmem {
    double val[kTTile];
    int32_t col[kTTile];
    int32_t row[kTTile];
    alignas(16) uint32_t hist[kHistWords<kTW>];
    int64_t warp_tmp[kTW + 1];
    int64_t base[256];   // first output position of the tile's entries of a digit, less their first place in the tile
    int32_t red[kTW];
    int64_t edge_row[2];  // rows of the tile's first and last entry
};

// A tile's rows are walked up to this many, and above it found by search: a walk
// takes a dependent load per kTThreads rows, a search one per bit of the rows for
// all entries of the tile at once.  A tile alone, walked / searched (whole call):
// 33,000 rows 80 / 69 us, 66,000 97 / 71, 1 M 601 / 77, 20 M 17.6 / 0.12 ms; 244
// tiles at once: 5 rows an entry 143 / 157 us, 8 169 / 173, 16 219 / 218.
constexpr int64_t kWalkRows = 8 * kTTile;

// counts[d * tiles + tile] of digit d in each tile
__global__ void __launch_bounds__(kTThreads)
tile_hist_kernel(const int32_t* __restrict__ col, int64_t n, int shift, uint32_t mask, int64_t tiles,
                 int64_t* __restrict__ counts) {
    __shared__ uint32_t h[256];
    const int64_t tile = blockIdx.x;
    if (threadIdx.x < 256) h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t t0 = tile * kTTile;
    int32_t c[kTItems];
#pragma unroll
    for (int i = 0; i < kTItems; ++i) {
        const int64_t p = t0 + i * kTThreads + threadIdx.x;
        c[i] = p < n ? col[p] : -1;
    }
#pragma unroll
    for (int i = 0; i < kTItems; ++i)
        if (c[i] >= 0) atomicAdd(&h[(static_cast<uint32_t>(c[i]) >> shift) & mask], 1u);
    __syncthreads();
    if (threadIdx.x < 256) counts[static_cast<int64_t>(threadIdx.x) * tiles + tile] = h[threadIdx.x];
}

// Last row whose first entry is at or before p (rp[0] = 0 <= p < rp[rows]), by a
// whole warp: 32-fold narrower per step.
__device__ inline int64_t row_of_entry(const int64_t* __restrict__ rp, int64_t rows, int64_t p, int lane) {
    int64_t lo = 0;
    for (int64_t range = rows; range > 1;) {
        const int64_t stride = (range + 31) / 32;
        const int64_t r = lo + lane * stride;
        const unsigned below = __ballot_sync(0xffffffffu, r < rows && rp[r] <= p);
        lo += (__popc(below) - 1) * stride;
        range = stride;
    }
    return lo;
}

// Rows of the tile's entries into sm.row, in the tile's order: every row's number
// at its first entry, then a running maximum; a tile with a long stretch of empty
// rows searches A's offsets for every entry instead.
__device__ inline void tile_rows(PassSmem& sm, const int64_t* __restrict__ rp, int64_t rows, int64_t t0, int n, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kTTile; i += kTThreads) sm.row[i] = 0;
    if (warp < 2) {
        const int64_t r = row_of_entry(rp, rows, warp ? t0 + n - 1 : t0, lane);
        if (lane == 0) sm.edge_row[warp] = r;
    }
    __syncthreads();
    const int64_t r0 = sm.edge_row[0], r1 = sm.edge_row[1];
    if (r1 - r0 > kWalkRows) {
        int64_t r[kTItems];
#pragma unroll
        for (int i = 0; i < kTItems; ++i) r[i] = r0;
        for (int64_t range = r1 - r0 + 1; range > 1;) {
            const int64_t half = range / 2;
#pragma unroll
            for (int i = 0; i < kTItems; ++i) {
                const int p = i * kTThreads + tid;
                if (p < n && rp[r[i] + half] <= t0 + p) r[i] += half;
            }
            range -= half;
        }
#pragma unroll
        for (int i = 0; i < kTItems; ++i) sm.row[i * kTThreads + tid] = static_cast<int32_t>(r[i]);
        __syncthreads();
        return;
    }
    for (int64_t r = r0 + 1 + tid; r <= r1; r += kTThreads) {
        const int64_t s = rp[r] - t0;
        if (s > 0) atomicMax(&sm.row[s], static_cast<int32_t>(r - r0));  // empty rows: the last one wins
    }
    __syncthreads();
    int32_t m[kTItems];
    int32_t most = 0;
#pragma unroll
    for (int i = 0; i < kTItems; ++i) {
        most = max(most, sm.row[tid * kTItems + i]);
        m[i] = most;
    }
    int32_t incl = most;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl = max(incl, t);
    }
    if (lane == 31) sm.red[warp] = incl;
    int32_t before = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) before = 0;
    __syncthreads();
    for (int w = 0; w < warp; ++w) before = max(before, sm.red[w]);
#pragma unroll
    for (int i = 0; i < kTItems; ++i) sm.row[tid * kTItems + i] = static_cast<int32_t>(r0) + max(before, m[i]);
    __syncthreads();
}

// One pass: entries of the tile to offs[digit * tiles + tile] + their rank among
// the tile's entries of the digit.  FIRST: rows from rp.  LAST: no columns out.
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(kTThreads, 2)
tile_scatter_kernel(Entries in, Entries out, const int64_t* __restrict__ rp, int64_t rows, int64_t n, int shift,
                    uint32_t mask, int64_t tiles, const int64_t* __restrict__ offs) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PassSmem& sm = *reinterpret_cast<PassSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t tile = blockIdx.x, t0 = tile * kTTile;
    const int nt = static_cast<int>(min(static_cast<int64_t>(kTTile), n - t0));
    for (int d = tid; d < kHistWords<kTW>; d += kTThreads) sm.hist[d] = 0;
    // item i of a thread: entry (warp * kTItems + i) * 32 + lane, so that ranks in
    // (warp, item, lane) order are the entries' order
    int32_t c[kTItems], r[kTItems];
    double v[kTItems];
    uint32_t rk[kTItems];
#pragma unroll
    for (int i = 0; i < kTItems; ++i) {
        const int p = (warp * kTItems + i) * 32 + lane;
        c[i] = -1;
        if (p < nt) {
            c[i] = in.col[t0 + p];
            v[i] = in.val[t0 + p];
            if constexpr (!FIRST) r[i] = in.row[t0 + p];
        }
    }
    if constexpr (FIRST) {
        tile_rows(sm, rp, rows, t0, nt, tid);
#pragma unroll
        for (int i = 0; i < kTItems; ++i) r[i] = sm.row[(warp * kTItems + i) * 32 + lane];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kTItems; ++i) {
        const uint32_t d = c[i] >= 0 ? (static_cast<uint32_t>(c[i]) >> shift) & mask : 255u;  // padding ranks last
        rk[i] = rank_item(d, &sm.hist[hidx<kTW>(static_cast<int>(d), warp)], lane);
    }
    __syncthreads();
    scan_counters<kTW>(sm.hist, sm.warp_tmp);
    __syncthreads();
    if (tid <= static_cast<int>(mask))
        sm.base[tid] = offs[static_cast<int64_t>(tid) * tiles + tile] - sm.hist[hidx<kTW>(tid, 0)];
#pragma unroll
    for (int i = 0; i < kTItems; ++i) {
        if (c[i] < 0) continue;
        const uint32_t d = (static_cast<uint32_t>(c[i]) >> shift) & mask;
        const uint32_t at = sm.hist[hidx<kTW>(static_cast<int>(d), warp)] + rk[i];
        sm.col[at] = c[i];
        sm.row[at] = r[i];
        sm.val[at] = v[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kTItems; ++i) {
        const int p = i * kTThreads + tid;
        if (p >= nt) break;
        const int32_t col = sm.col[p];
        const int64_t at = sm.base[(static_cast<uint32_t>(col) >> shift) & mask] + p;
        if constexpr (!LAST) out.col[at] = col;
        out.row[at] = sm.row[p];
        out.val[at] = sm.val[p];
    }
}

__global__ void __launch_bounds__(256)
col_count_kernel(const int32_t* __restrict__ col, int64_t n, int64_t* __restrict__ cnt) {
    constexpr int U = 4;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x * U;
    for (int64_t p0 = static_cast<int64_t>(blockIdx.x) * blockDim.x * U + threadIdx.x; p0 < n; p0 += stride) {
        int32_t c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) c[u] = p0 + u * blockDim.x < n ? col[p0 + u * blockDim.x] : -1;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c[u] >= 0) atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[c[u]]), 1ull);
    }
}

int grid_of(int64_t work, int per_block, int cap) {
    const int64_t g = (work + per_block - 1) / per_block;
    return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

int column_bits(int32_t cols) {
    int bits = 0;
    while (bits < 31 && (int64_t{1} << bits) < cols) ++bits;
    return bits;
}
int pass_count(int32_t cols) { return std::max(1, (column_bits(cols) + 7) / 8); }

size_t up256(size_t x) { return (x + 255) & ~size_t{255}; }

// Scratch: counts (256 tiles + 1), scan partials of the counts and of the
// columns, then the entries between passes: values, columns and rows of one set,
// and with more than two passes the columns of a second one, whose rows and values
// lie in the result's arrays (20 bytes an entry).
struct TransposeLayout {
    size_t counts = 0, partials = 0, col_partials = 0, val = 0, col = 0, row = 0, col2 = 0, bytes = 0;
};
TransposeLayout transpose_layout(int64_t nnz, int32_t cols) {
    TransposeLayout L;
    const int64_t tiles = (nnz + kTTile - 1) / kTTile;
    L.partials = up256(static_cast<size_t>(256 * tiles + 1) * 8);
    L.col_partials = L.partials + up256(scan_partials_count(256 * tiles + 1) * 8);
    const int between = std::min(pass_count(cols) - 1, 2);
    const size_t n = static_cast<size_t>(nnz);
    L.val = L.col_partials + up256(scan_partials_count(static_cast<int64_t>(cols) + 1) * 8);
    L.col = L.val + (between > 0 ? up256(n * 8) : 0);
    L.row = L.col + (between > 0 ? up256(n * 4) : 0);
    L.col2 = L.row + (between > 0 ? up256(n * 4) : 0);
    L.bytes = L.col2 + (between > 1 ? up256(n * 4) : 0);
    return L;
}

}  // namespace

size_t transpose_scratch_bytes(int64_t nnz, int32_t cols) { return transpose_layout(nnz, cols).bytes; }

void launch_transpose(const int64_t* rp, const int32_t* col, const double* val, int32_t rows, int32_t cols, int64_t nnz,
                      int64_t* out_rp, int32_t* out_col, double* out_val, void* scratch, cudaStream_t st,
                      cudaStream_t counts_st) {
    const int64_t tiles = (nnz + kTTile - 1) / kTTile;
    const TransposeLayout L = transpose_layout(nnz, cols);
    unsigned char* s = static_cast<unsigned char*>(scratch);
    int64_t* counts = reinterpret_cast<int64_t*>(s + L.counts);
    int64_t* partials = reinterpret_cast<int64_t*>(s + L.partials);

    // row pointer of A^T: column counts, scanned (beside the passes: bound by
    // atomics in L2, they by DRAM)
    cudaMemsetAsync(out_rp, 0, sizeof(int64_t) * (static_cast<size_t>(cols) + 1), counts_st);
    if (nnz > 0) col_count_kernel<<<grid_of(nnz, 1024, 152 * 8), 256, 0, counts_st>>>(col, nnz, out_rp);
    launch_scan(out_rp, cols, reinterpret_cast<int64_t*>(s + L.col_partials), counts_st);
    if (nnz == 0) return;
    const int bits = column_bits(cols), passes = pass_count(cols);
    const int smem = static_cast<int>(sizeof(PassSmem));
    // the last pass reads the scratch's set, the one before it the other, and so on
    const Entries own{reinterpret_cast<int32_t*>(s + L.col), reinterpret_cast<int32_t*>(s + L.row),
                      reinterpret_cast<double*>(s + L.val)};
    const Entries shared{reinterpret_cast<int32_t*>(s + L.col2), out_col, out_val};
    Entries in;
    in.col = const_cast<int32_t*>(col);
    in.val = const_cast<double*>(val);
    for (int p = 0, shift = 0; p < passes; ++p) {
        // digits of about equal width: fewer digits, longer runs
        const int width = (bits - shift + passes - p - 1) / (passes - p);
        const uint32_t mask = (1u << width) - 1u;
        const bool first = p == 0, last = p == passes - 1;
        Entries out = last ? Entries{nullptr, out_col, out_val} : (passes - p) % 2 == 0 ? own : shared;
        tile_hist_kernel<<<static_cast<unsigned>(tiles), kTThreads, 0, st>>>(in.col, nnz, shift, mask, tiles, counts);
        launch_scan(counts, (static_cast<int64_t>(mask) + 1) * tiles, partials, st);
        auto kern = first ? (last ? tile_scatter_kernel<true, true> : tile_scatter_kernel<true, false>)
                          : (last ? tile_scatter_kernel<false, true> : tile_scatter_kernel<false, false>);
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        kern<<<static_cast<unsigned>(tiles), kTThreads, smem, st>>>(in, out, rp, rows, nnz, shift, mask, tiles, counts);
        in = out;
        shift += width;
    }
}

}  // namespace spg
