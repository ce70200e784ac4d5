// Register sort of a warp's 32 * ITEMS keys.
//
// Every lane holds ITEMS keys; afterwards lane l holds the l-th run of ITEMS
// keys of the ascending order.  Each lane sorts its own keys (Batcher's merge
// exchange), then runs of 1, 2, 4, 8 and 16 lanes are merged pairwise: the
// first step of a merge compares with the mirrored element of the other run,
// the next ones are half-cleaners between lanes, and a bitonic merge inside
// the lane ends it.  Fifteen shuffles per key whatever ITEMS is, the rest
// minima and maxima between registers; no shared memory, no branch, and ITEMS
// independent chains to hide each step's latency.
#pragma once

#include <cstdint>
#include <utility>

namespace spg {

struct CePair {
    int a, b;
};

// Batcher's merge exchange for n keys (Knuth, TAOCP 3, 5.2.2 Algorithm M).
template <int N>
struct MergeExchange {
    static constexpr int count() {
        int c = 0;
        for (int p = 1; p < N; p *= 2)
            for (int k = p; k >= 1; k /= 2)
                for (int j = k % p; j <= N - 1 - k; j += 2 * k)
                    for (int i = 0; i < k && i + j + k < N; ++i)
                        if ((i + j) / (2 * p) == (i + j + k) / (2 * p)) ++c;
        return c;
    }
    CePair pair[N > 1 ? 256 : 1] = {};
    constexpr MergeExchange() {
        int c = 0;
        for (int p = 1; p < N; p *= 2)
            for (int k = p; k >= 1; k /= 2)
                for (int j = k % p; j <= N - 1 - k; j += 2 * k)
                    for (int i = 0; i < k && i + j + k < N; ++i)
                        if ((i + j) / (2 * p) == (i + j + k) / (2 * p)) pair[c++] = CePair{i + j, i + j + k};
    }
};

// Sorts a bitonic sequence of n keys: half-cleaners while n is even, then the
// remaining odd run (1 or 3 keys) in full.
template <int N>
struct BitonicMerge {
    static constexpr int count() {
        int c = 0, n = N;
        for (; n > 1 && n % 2 == 0; n /= 2) c += N / 2;
        if (n == 3) c += N;
        return c;
    }
    CePair pair[N > 1 ? 256 : 1] = {};
    constexpr BitonicMerge() {
        int c = 0, n = N;
        for (; n > 1 && n % 2 == 0; n /= 2)
            for (int s = 0; s < N; s += n)
                for (int i = 0; i < n / 2; ++i) pair[c++] = CePair{s + i, s + i + n / 2};
        if (n == 3)
            for (int s = 0; s < N; s += 3) {
                pair[c++] = CePair{s, s + 1};
                pair[c++] = CePair{s + 1, s + 2};
                pair[c++] = CePair{s, s + 1};
            }
    }
};

template <typename K, int N>
__device__ __forceinline__ void compare_exchange(K (&k)[N], int a, int b) {
    const K lo = min(k[a], k[b]);
    k[b] = max(k[a], k[b]);
    k[a] = lo;
}

template <typename Net, typename K, int N, int... I>
__device__ __forceinline__ void run_network(K (&k)[N], std::integer_sequence<int, I...>) {
    constexpr Net net{};
    (compare_exchange(k, std::integral_constant<int, net.pair[I].a>::value, std::integral_constant<int, net.pair[I].b>::value),
     ...);
}

template <typename K, int ITEMS>
__device__ __forceinline__ void warp_sort(K (&k)[ITEMS], int lane) {
    if constexpr (ITEMS > 1)
        run_network<MergeExchange<ITEMS>>(k, std::make_integer_sequence<int, MergeExchange<ITEMS>::count()>{});
#pragma unroll
    for (int m = 1; m < 32; m *= 2) {  // runs of m lanes into runs of 2m
        {
            const bool low = (lane & m) == 0;
            K t[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) t[i] = __shfl_xor_sync(0xffffffffu, k[ITEMS - 1 - i], 2 * m - 1);
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) k[i] = low ? min(k[i], t[i]) : max(k[i], t[i]);
        }
#pragma unroll
        for (int d = m / 2; d >= 1; d /= 2) {
            const bool low = (lane & d) == 0;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const K t = __shfl_xor_sync(0xffffffffu, k[i], d);
                k[i] = low ? min(k[i], t) : max(k[i], t);
            }
        }
        if constexpr (ITEMS > 1)
            run_network<BitonicMerge<ITEMS>>(k, std::make_integer_sequence<int, BitonicMerge<ITEMS>::count()>{});
    }
}

}  // namespace spg
