// BlockCache: device blocks kept by a handle between its calls (blocks.h).
#include "blocks.h"

#include <algorithm>
#include <mutex>
#include <unordered_map>

namespace spg {
namespace {

struct Owned {
    size_t bytes;
    uint64_t cache;  // id of the cache that allocated it
};

// Every block handed out by a cache and not yet freed, and the caches.
struct Registry {
    std::mutex lock;
    std::unordered_map<void*, Owned> blocks;
    std::vector<BlockCache*> caches;
    uint64_t next_id = 1;
};

Registry& registry() {
    static Registry* r = new Registry;  // outlives handles destroyed at exit
    return *r;
}

uint64_t new_id() {
    Registry& r = registry();
    std::lock_guard<std::mutex> g(r.lock);
    return r.next_id++;
}

// Sizes that blocks come in, so that calls of about the same size share them:
// powers of two below 1 MiB, steps of an eighth to 32 MiB, then of 2 MiB.
size_t block_size(size_t bytes) {
    size_t p = 512;
    while (p < bytes && p < (size_t{1} << 20)) p *= 2;
    if (bytes <= p) return p;
    size_t step = size_t{2} << 20;
    if (bytes < (size_t{32} << 20)) {
        while (p * 2 <= bytes) p *= 2;
        step = p / 8;
    }
    return (bytes + step - 1) / step * step;
}

}  // namespace

// Every handle's kept blocks go back to the pool; called with the lock held.
void give_back_all() {
    for (BlockCache* c : registry().caches) {
        if (c->kept_.empty() || c->capturing_) continue;
        c->give_back_locked(0);
        cudaStreamSynchronize(c->stream_);
    }
}

BlockCache::BlockCache(int device, cudaStream_t stream) : id_(new_id()), device_(device), stream_(stream) {
    size_t total = 0, free_now = 0;  // of the current device, the handle's
    if (cudaMemGetInfo(&free_now, &total) == cudaSuccess) limit_ = total / 16;
    else cudaGetLastError();
    Registry& r = registry();
    std::lock_guard<std::mutex> g(r.lock);
    r.caches.push_back(this);
}

BlockCache::~BlockCache() {
    Registry& r = registry();
    std::lock_guard<std::mutex> g(r.lock);
    give_back_locked(0);
    r.caches.erase(std::remove(r.caches.begin(), r.caches.end(), this), r.caches.end());
}

void BlockCache::give_back_locked(size_t most) {
    size_t n = 0;
    for (; n < kept_.size() && kept_bytes_ > most; ++n) {
        cudaFreeAsync(kept_[n].p, stream_);
        kept_bytes_ -= kept_[n].bytes;
    }
    kept_.erase(kept_.begin(), kept_.begin() + static_cast<std::ptrdiff_t>(n));
}

cudaError_t BlockCache::alloc(void** p, size_t bytes) {
    const size_t want = block_size(bytes);
    Registry& r = registry();
    std::lock_guard<std::mutex> g(r.lock);
    // the smallest kept block that is not more than a quarter too large
    size_t best = kept_.size();
    for (size_t i = 0; i < kept_.size(); ++i)
        if (kept_[i].bytes >= want && kept_[i].bytes <= want + want / 4 &&
            (best == kept_.size() || kept_[i].bytes < kept_[best].bytes))
            best = i;
    if (best < kept_.size()) {
        const Kept k = kept_[best];
        kept_.erase(kept_.begin() + static_cast<std::ptrdiff_t>(best));
        kept_bytes_ -= k.bytes;
        r.blocks[k.p] = Owned{k.bytes, id_};
        *p = k.p;
        return cudaSuccess;
    }
    cudaError_t e = cudaMallocAsync(p, want, stream_);
    size_t got = want;
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        give_back_all();
        got = std::max<size_t>(bytes, 16);
        e = cudaMallocAsync(p, got, stream_);
    }
    if (e == cudaSuccess) r.blocks[*p] = Owned{got, id_};
    return e;
}

void BlockCache::free(void* p) {
    if (!p) return;
    Registry& r = registry();
    std::lock_guard<std::mutex> g(r.lock);
    const auto it = r.blocks.find(p);
    const bool own = it != r.blocks.end() && it->second.cache == id_;
    const size_t bytes = own ? it->second.bytes : 0;
    if (it != r.blocks.end()) r.blocks.erase(it);
    if (!own || bytes > limit_) {
        cudaFreeAsync(p, stream_);
        return;
    }
    kept_.push_back(Kept{p, bytes});
    kept_bytes_ += bytes;
    size_t others = 0;
    for (const BlockCache* c : r.caches)
        if (c != this && c->device_ == device_) others += c->kept_bytes_;
    const size_t most = limit_ - std::min(limit_, others);
    if (kept_bytes_ > most) give_back_locked(most);
    if (kept_.size() > 256) give_back_locked(kept_bytes_ - 1);
}

void BlockCache::set_capturing(bool on) {
    std::lock_guard<std::mutex> g(registry().lock);
    capturing_ = on;
}

void block_release(void* p) {
    if (!p) return;
    Registry& r = registry();
    {
        std::lock_guard<std::mutex> g(r.lock);
        r.blocks.erase(p);
    }
    cudaFree(p);
}

cudaError_t device_malloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    {
        std::lock_guard<std::mutex> g(registry().lock);
        give_back_all();
    }
    int device = 0;
    cudaMemPool_t pool;
    if (cudaGetDevice(&device) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess)
        cudaMemPoolTrimTo(pool, 0);
    return cudaMalloc(p, bytes);
}

}  // namespace spg
