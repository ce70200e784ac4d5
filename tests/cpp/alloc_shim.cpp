// Stands in front of the CUDA runtime's device allocations in a test process:
// counts them and the bytes they hold, and lets chosen ones fail as if the device
// memory had run out.  Loaded (RTLD_GLOBAL) before the engine, so that the engine's
// calls bind here.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <atomic>
#include <chrono>
#include <mutex>
#include <thread>
#include <unordered_map>

namespace {

std::mutex lock;
std::unordered_map<void*, size_t> live;
std::atomic<long long> slow_bytes{-1}, slow_ms{0};  // allocations of at least that many bytes take that long
long long limit = -1;  // most bytes held at once
long long calls, bytes, peak, failed, fail_from, fail_count, total;

template <typename F>
F next(const char* name) {
    return reinterpret_cast<F>(dlsym(RTLD_NEXT, name));
}

template <typename Alloc>
cudaError_t counted(void** p, size_t n, Alloc&& alloc) {
    {
        std::lock_guard<std::mutex> g(lock);
        const long long i = calls++;
        if ((fail_count && i >= fail_from && i - fail_from < fail_count) ||
            (limit >= 0 && bytes + static_cast<long long>(n) > limit)) {
            ++failed;
            return cudaErrorMemoryAllocation;
        }
    }
    const long long slow = slow_bytes;
    if (slow >= 0 && static_cast<long long>(n) >= slow) std::this_thread::sleep_for(std::chrono::milliseconds(slow_ms));
    const cudaError_t e = alloc();
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> g(lock);
        live[*p] = n;
        total += static_cast<long long>(n);
        bytes += static_cast<long long>(n);
        if (bytes > peak) peak = bytes;
    }
    return e;
}

void forget(void* p) {
    std::lock_guard<std::mutex> g(lock);
    const auto it = live.find(p);
    if (it == live.end()) return;
    bytes -= static_cast<long long>(it->second);
    live.erase(it);
}

}  // namespace

extern "C" {

cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t st) {
    static const auto real = next<cudaError_t (*)(void**, size_t, cudaStream_t)>("cudaMallocAsync");
    return counted(p, n, [&] { return real(p, n, st); });
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t st) {
    static const auto real = next<cudaError_t (*)(void**, size_t, cudaMemPool_t, cudaStream_t)>("cudaMallocFromPoolAsync");
    return counted(p, n, [&] { return real(p, n, pool, st); });
}
cudaError_t cudaMalloc(void** p, size_t n) {
    static const auto real = next<cudaError_t (*)(void**, size_t)>("cudaMalloc");
    return counted(p, n, [&] { return real(p, n); });
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t st) {
    static const auto real = next<cudaError_t (*)(void*, cudaStream_t)>("cudaFreeAsync");
    forget(p);
    return real(p, st);
}
cudaError_t cudaFree(void* p) {
    static const auto real = next<cudaError_t (*)(void*)>("cudaFree");
    forget(p);
    return real(p);
}

// Allocations from now on are numbered from 0; `count` of them from number `from` on
// fail.  The peak starts again from what is held now.
void shim_start(long long from, long long count) {
    std::lock_guard<std::mutex> g(lock);
    calls = failed = total = 0;
    peak = bytes;
    fail_from = from;
    fail_count = count;
}
// A device of that many bytes more than are held now (< 0: without a limit).
void shim_limit(long long more) {
    std::lock_guard<std::mutex> g(lock);
    limit = more < 0 ? -1 : bytes + more;
}
void shim_slow(long long from_bytes, long long ms) {
    slow_ms = ms;
    slow_bytes = from_bytes;
}
// calls, failed ones, bytes held now, their peak, all bytes ever asked for
void shim_stats(long long* out) {
    std::lock_guard<std::mutex> g(lock);
    out[0] = calls;
    out[1] = failed;
    out[2] = bytes;
    out[3] = peak;
    out[4] = total;
}
// bytes asked for at p (-1: not a live allocation)
long long shim_size(void* p) {
    std::lock_guard<std::mutex> g(lock);
    const auto it = live.find(p);
    return it == live.end() ? -1 : static_cast<long long>(it->second);
}

}  // extern "C"
