// Rules of the dispatch that depend on sizes alone, free of device code.
#pragma once

#include <cstdint>

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

}  // namespace spg
