// The dispatch's rules on sizes (csrc/dispatch.h), on the host.
#include <algorithm>
#include <cstdio>
#include <initializer_list>

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
    return failures ? 1 : 0;
}
