// Rules of the dispatch that depend on sizes alone, free of device code.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace spg {

__host__ __device__ inline int ceil_log2(int64_t x) {
    int l = 0;
    while ((int64_t{1} << l) < x) ++l;
    return l;
}

// K2's bitmaps of columns: log2 of the words of one of `cols` columns, and the most
// that shared memory takes (128 KiB).
__host__ __device__ inline int bitmap_log2(int64_t cols) {
    const int l = ceil_log2(cols) - 5;
    return l > 0 ? l : 0;
}
constexpr int kMaxBitmapLog2 = 15;

// The columns of a B that K2's rows above 16,384 products count for the bitmap that
// their launch reserves: none where its bitmap does not fit.
inline int64_t heavy_map_cols(int64_t cols) { return bitmap_log2(cols) <= kMaxBitmapLog2 ? cols : 0; }

// log2 of the words reserved for the widest of those; -1: no bitmap and no shared
// memory for one (128 KiB that no row can use halve the CTAs per SM: 2,000 rows of
// 40,000 products, 2^20 + 1 columns, 4.7 ms with them and 3.4 without).
inline int heavy_map_log2(int64_t map_cols) { return map_cols > 0 ? bitmap_log2(map_cols) : -1; }

// K1's lanes per row, by the entries of A in the rows of a launch.  Measured with 4 / 8
// lanes (2 and 32 were slower everywhere; one warp per row with 64-bit shared atomics
// before): 65,536 rows of 16 entries 13.3 / 15.8 us (21), power-law rows of 24 on
// average 244 / 255 us (323), uneven rows of 34 38 / 35 us (34), R and R*A of the
// 128^3 Galerkin chain (8 and 32 entries) 110 / 86 us (143).
inline int rowwork_lanes(int64_t entries, int64_t rows) { return entries / rows <= 24 ? 4 : 8; }

// K4's rows of bins 1 and 2 (<= 32 and <= 64 products) eight and four to a warp, or one:
// `entries` of A in the `count` rows of the bin.  Several rows to a warp leave fewer
// warps than the GPU holds below 64 rows per SM (accumulated stages with 4-500 such
// rows: 9.5 us a launch against 7).  They also walk their entries one row after the
// other, which entries whose B row is empty make long.  Several / one, in us:
//   bin 1, rows of 14 products: 10,000 rows of 16 entries 17.8 / 18.3, of 32 21.7 / 19.2,
//     of 1,024 265 / 134; 20,000 of 32 24 / 27, of 64 35 / 33, of 1,024 306 / 226; 50,000 of
//     96 77 / 79, of 192 143 / 130; 200,000 of 16 81 / 142, of 512 1,012 / 1,044;
//   bin 2, rows of 44 products: 20,000 rows of 32 32 / 28, of 128 56 / 46, of 1,024 246 /
//     185; 200,000 of 32 157 / 151, of 64 202 / 202, of 128 328 / 306, of 512 936 / 817;
//     rows of 56 products without empty B rows: 50,000 of 8 40 / 48, of 36 54 / 66, of 56
//     68 / 79, 200,000 of 8 122 / 162, of 28 174 / 184, of 56 226 / 276.
inline bool several_rows_per_warp(int bin, int64_t count, int64_t entries, int num_sms) {
    if (count < static_cast<int64_t>(num_sms) * 64) return false;
    if (bin == 1) return 8 * (entries / count) <= 3 * (count / num_sms);
    return bin == 2 && entries / count <= 64;
}

// The row blocks of a product that is copied to the host while it is computed.
struct RowBlock {
    int32_t first, end;  // rows
    int64_t entries;     // of A in them
};

// Operands with at least this many entries in A are multiplied in row blocks.
constexpr int64_t kBlockedEntries = int64_t{1} << 22;

// Row blocks by A's entries: 1/32, 1/32, 1/16, then 1/8 each, so that the first
// copy starts after a small block and the later blocks keep the copy engine
// busy while the next one computes.  Small operands run as one block.  The
// cuts come from A's row offsets on the host, or from equal row counts
// when A lives on the device (row_ptr is nullptr).
inline std::vector<RowBlock> row_blocks(int32_t rows, int64_t nnz, const int64_t* row_ptr) {
    std::vector<int32_t> cut{0};
    if (nnz >= kBlockedEntries && rows > 1) {
        const double fr[] = {1.0 / 32, 1.0 / 32, 1.0 / 16, 1.0 / 8, 1.0 / 8, 1.0 / 8, 1.0 / 8, 1.0 / 8, 1.0 / 8, 1.0 / 8};
        double acc = 0.0;
        for (double f : fr) {
            acc += f;
            int32_t r;
            if (acc >= 1.0 - 1e-12) {
                r = rows;
            } else if (row_ptr) {
                const int64_t target = static_cast<int64_t>(acc * static_cast<double>(nnz));
                r = static_cast<int32_t>(std::lower_bound(row_ptr, row_ptr + rows + 1, target) - row_ptr);
            } else {
                r = static_cast<int32_t>(acc * rows);
            }
            r = std::min(std::max(r, cut.back()), rows);
            if (r > cut.back()) cut.push_back(r);
        }
    }
    if (cut.back() != rows) cut.push_back(rows);
    std::vector<RowBlock> blocks;
    for (size_t k = 0; k + 1 < cut.size(); ++k) {
        const int32_t r0 = cut[k], r1 = cut[k + 1];
        blocks.push_back({r0, r1, row_ptr ? row_ptr[r1] - row_ptr[r0]
                                          : static_cast<int64_t>(static_cast<double>(nnz) * (r1 - r0) / rows)});
    }
    return blocks;
}

}  // namespace spg
