// The dispatch's rules on sizes (csrc/dispatch.h), on the host.
#include <algorithm>
#include <cstdio>
#include <initializer_list>
#include <vector>

#include "dispatch.h"

static int failures = 0;
#define CHECK(x) \
    do { \
        if (!(x)) { \
            std::printf("line %d: %s\n", __LINE__, #x); \
            ++failures; \
        } \
    } while (0)

static int map_log2(std::initializer_list<int64_t> cols) {
    int64_t most = 0;
    for (int64_t c : cols) most = std::max(most, spg::heavy_map_cols(c));
    return spg::heavy_map_log2(most);
}

int main() {
    // K2, heavy rows: a bitmap holds every column, is reserved for the widest product
    // that has one, and not at all where none has
    for (int64_t c : {1, 32, 33, 64, 65, 1 << 17, (1 << 20) - 1, 1 << 20}) {
        CHECK((int64_t{32} << spg::bitmap_log2(c)) >= c);
        CHECK(map_log2({c}) == spg::bitmap_log2(c));
    }
    CHECK(map_log2({1 << 20}) == spg::kMaxBitmapLog2);
    CHECK(map_log2({(1 << 20) + 1}) == -1);
    CHECK(map_log2({1 << 30}) == -1);
    CHECK(map_log2({0}) == -1);
    CHECK(map_log2({1 << 21, 5000, 40}) == spg::bitmap_log2(5000));

    // Row blocks cover the rows in order, and each knows its own entries: K1's lanes
    // follow the mean of the block, not the matrix's entries over the block's rows
    for (int32_t rows : {2, 33, 262144, 1 << 20})
        for (int64_t mean : {8, 24, 25, 40, 1 << 22}) {
            std::vector<int64_t> rp(static_cast<size_t>(rows) + 1, 0);
            for (int32_t r = 0; r < rows; ++r) rp[r + 1] = rp[r] + mean + (r % 3 - 1) * (r + 1 < rows - rows % 3);
            const int64_t nnz = rp[rows];
            for (const int64_t* row_ptr : {static_cast<const int64_t*>(rp.data()), static_cast<const int64_t*>(nullptr)}) {
                const std::vector<spg::RowBlock> blocks = spg::row_blocks(rows, nnz, row_ptr);
                CHECK((blocks.size() > 1) == (nnz >= spg::kBlockedEntries));
                int32_t at = 0;
                int64_t entries = 0;
                for (const spg::RowBlock& b : blocks) {
                    CHECK(b.first == at && b.end > at);
                    at = b.end;
                    entries += b.entries;
                    const int64_t own = rp[b.end] - rp[b.first];
                    CHECK(b.entries == own || (!row_ptr && b.entries >= own - 2 && b.entries <= own + 2));
                    if (mean != 24 && mean != 25)
                        CHECK(spg::rowwork_lanes(b.entries, b.end - b.first) == spg::rowwork_lanes(nnz, rows));
                }
                CHECK(at == rows);
                CHECK(entries <= nnz && entries >= nnz - 10);
            }
        }
    CHECK(spg::row_blocks(0, 0, nullptr).empty());

    // Short rows several to a warp: many rows of few entries, not rows whose entries
    // mostly meet empty rows of B (measured on both sides, see the rule)
    constexpr int kSms = 152;
    auto several = [](int bin, int64_t rows, int64_t each) {
        return spg::several_rows_per_warp(bin, rows, rows * each, kSms);
    };
    CHECK(several(1, 10000, 16) && several(1, 20000, 32) && several(1, 50000, 96) && several(1, 262144, 32));
    CHECK(!several(1, 10000, 64) && !several(1, 20000, 128) && !several(1, 50000, 192) && !several(1, 20000, 2000));
    CHECK(several(2, 262144, 8) && several(2, 50000, 56) && !several(2, 20000, 128) && !several(2, 200000, 512));
    for (int bin : {1, 2}) CHECK(!several(bin, 64 * kSms - 1, 2) && several(bin, 64 * kSms, 2));
    CHECK(!several(3, 262144, 8));
    CHECK(spg::rowwork_lanes(24 * 1000 + 999, 1000) == 4 && spg::rowwork_lanes(25 * 1000, 1000) == 8);
    return failures ? 1 : 0;
}
